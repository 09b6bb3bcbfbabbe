// Host-once plan of the sparse cluster factorisation (see gp_cluster_plan.h).
#include "gp_cluster_plan.h"

#include <algorithm>
#include <cmath>
#include <map>
#include <set>
#include <stdexcept>
#include <string>

namespace gp {
namespace {

struct PatSink {
    int ws;
    std::set<int> *ent, *var;   // every entry; those that depend on the state
    void put(int r, int c, double) {
        ent->insert((r - ws) * 32 + (c - ws));
        var->insert((r - ws) * 32 + (c - ws));
    }
    void putc(int r, int c, double) { ent->insert((r - ws) * 32 + (c - ws)); }
    void putv(int r, int k, double) { ent->insert((r - ws) * 32 + 29 + k); }
    void putf(int r, double) { ent->insert((r - ws) * 32 + 31); }
};

struct DenseSink {
    int ws;
    double *a;   // [32*32]
    void put(int r, int c, double v) { a[(r - ws) * 32 + (c - ws)] = v; }
    void putc(int r, int c, double v) { put(r, c, v); }
    void putv(int r, int k, double v) { a[(r - ws) * 32 + 29 + k] = v; }
    void putf(int r, double v) { a[(r - ws) * 32 + 31] = v; }
};

// Entries to their slots with the backward-Euler scaling: the constant ones
// (image) or the state-dependent ones, as the device's two sinks.
struct SlotSink {
    int ws;
    const short *slot_of;
    double *v;
    unsigned diff;
    double dt;
    bool image;
    const double *z, *zold;
    void store(int r, int c, double x) {
        const bool d = diff >> (r - ws) & 1;
        if (d) x *= -dt;
        if (d && r == c) x += 1.0;
        v[slot_of[(r - ws) * 32 + (c - ws)]] = x;
    }
    void put(int r, int c, double x) {
        if (!image) store(r, c, x);
    }
    void putc(int r, int c, double x) {
        if (image) store(r, c, x);
    }
    void putv(int r, int k, double x) {
        if (image) return;
        v[slot_of[(r - ws) * 32 + 29 + k]] = diff >> (r - ws) & 1 ? -dt * x : x;
    }
    void putf(int r, double x) {
        if (image) return;
        v[slot_of[(r - ws) * 32 + 31]] = diff >> (r - ws) & 1 ? z[r] - zold[r] - dt * x : x;
    }
};

// One operation on slots, for the scheduler.
struct SlotOp {
    int code, d, a, b;   // REC_*; b unused but for FMS
};

// Schedules `ops` (in program order) for kCluWarps warps: list scheduling by
// the longest path to the end.  Within a stage no operation reads or writes
// a slot that another one writes, so the warps need only meet between
// stages.  The unit of length is one FP64 instruction's time on its pipe; a
// reciprocal takes about five, and a stage without one takes up to two
// operations a warp.
void schedule(const std::vector<SlotOp> &ops, int n_slots, std::vector<CluRec> *out) {
    const int n = (int)ops.size();
    std::vector<std::vector<int>> succ(n);
    std::vector<int> npred(n, 0), last_write(n_slots, -1);
    std::vector<std::vector<int>> readers(n_slots);
    auto dep = [&](int from, int to) {
        if (from >= 0 && from != to) {
            succ[from].push_back(to);
            npred[to]++;
        }
    };
    for (int i = 0; i < n; i++) {
        const SlotOp &o = ops[i];
        std::vector<int> rd = {o.a};
        if (o.code == REC_FMS) rd.push_back(o.b);
        for (int s : rd) dep(last_write[s], i);
        dep(last_write[o.d], i);
        for (int r : readers[o.d]) dep(r, i);
        readers[o.d].clear();
        for (int s : rd) readers[s].push_back(i);
        last_write[o.d] = i;
    }
    auto len = [&](int i) { return ops[i].code == REC_RCP ? 5 : 1; };
    std::vector<int> prio(n, 0);
    for (int i = n - 1; i >= 0; i--) {
        for (int j : succ[i]) prio[i] = std::max(prio[i], prio[j]);
        prio[i] += len(i) + 1;
    }
    std::vector<int> ready;
    for (int i = 0; i < n; i++)
        if (npred[i] == 0) ready.push_back(i);
    while (!ready.empty()) {
        std::stable_sort(ready.begin(), ready.end(), [&](int a, int b) { return prio[a] > prio[b]; });
        const bool rcp = ops[ready[0]].code == REC_RCP;
        const int cap = rcp ? 5 : 2;
        std::vector<int> take[kCluWarps], rest;
        int load[kCluWarps] = {};
        for (int i : ready) {
            int w = 0;
            for (int v = 1; v < kCluWarps; v++)
                if (load[v] < load[w]) w = v;
            if (load[w] + len(i) > cap) {
                rest.push_back(i);
                continue;
            }
            load[w] += len(i);
            take[w].push_back(i);
        }
        for (int w = 0; w < kCluWarps; w++) {
            std::vector<CluRec> &q = out[w];
            for (size_t k = 0; k < take[w].size(); k++) {
                const SlotOp &o = ops[take[w][k]];
                CluRec r{o.d * 32, o.a * 32, o.b * 32, o.code};
                CluRec t{0, 0, 0, 0};
                if (o.code != REC_RCP && k + 1 < take[w].size() && ops[take[w][k + 1]].code == o.code) {
                    const SlotOp &u = ops[take[w][++k]];
                    t = CluRec{u.d * 32, u.a * 32, u.b * 32, 0};
                    r.w |= u.code << 4;
                }
                q.push_back(r);
                q.push_back(t);
            }
            if (take[w].empty()) {
                q.push_back(CluRec{0, 0, 0, 0});
                q.push_back(CluRec{0, 0, 0, 0});
            }
            q[q.size() - 2].w |= REC_SYNC;
        }
        for (int w = 0; w < kCluWarps; w++)
            for (int i : take[w])
                for (int j : succ[i])
                    if (--npred[j] == 0) rest.push_back(j);
        ready.swap(rest);
    }
}

DevRef ref(const gp_device_table &T, int k) {
    DevRef d;
    d.dp = T.diff_ptr ? T.diff_ptr[k] : -1;
    d.ap = T.alg_ptr ? T.alg_ptr[k] : -1;
    d.cp = T.ctrl_ptr ? T.ctrl_ptr[k] : -1;
    d.pp = T.par_ptr[k];
    d.bus = T.bus[k];
    d.link0 = T.link0 ? T.link0[k] : -1;
    d.link1 = T.link1 ? T.link1[k] : -1;
    return d;
}

template <class Sink>
void eval_cluster(const gp_problem *pr, int c, const double *z, const double *u0, const double *p, Sink &s,
                  double *C, double *I) {
    const int net = pr->n_diff + pr->n_alg;
    genrou_eval(ref(pr->dev[GP_GENROU], pr->cl_gen[c]), net, z, u0, p, s, C, I);
    const int gt = pr->cl_gov_type[c];
    if (gt == GP_IEESGO) ieesgo_eval(ref(pr->dev[GP_IEESGO], pr->cl_gov[c]), z, p, s);
    else if (gt == GP_TGOV1) tgov1_eval(ref(pr->dev[GP_TGOV1], pr->cl_gov[c]), z, p, s);
    const int et = pr->cl_exc_type[c];
    if (et == GP_SEXS) sexs_eval(ref(pr->dev[GP_SEXS], pr->cl_exc[c]), net, z, p, s);
    else if (et == GP_ESDC1A) esdc1a_eval(ref(pr->dev[GP_ESDC1A], pr->cl_exc[c]), net, z, p, s);
    if (pr->cl_pss[c] >= 0) ieeest_eval(ref(pr->dev[GP_IEEEST], pr->cl_pss[c]), z, p, s);
}

// Minimum-cost perfect assignment (Hungarian method, O(n^3)).
std::vector<int> assign(const std::vector<std::vector<double>> &cost) {
    const int n = (int)cost.size();
    const double INF = 1e300;
    std::vector<double> u(n + 1, 0.0), v(n + 1, 0.0);
    std::vector<int> pm(n + 1, 0), way(n + 1, 0);
    for (int i = 1; i <= n; i++) {
        pm[0] = i;
        int j0 = 0;
        std::vector<double> minv(n + 1, INF);
        std::vector<char> used(n + 1, 0);
        do {
            used[j0] = 1;
            const int i0 = pm[j0];
            double delta = INF;
            int j1 = 0;
            for (int j = 1; j <= n; j++)
                if (!used[j]) {
                    const double cur = cost[i0 - 1][j - 1] - u[i0] - v[j];
                    if (cur < minv[j]) { minv[j] = cur; way[j] = j0; }
                    if (minv[j] < delta) { delta = minv[j]; j1 = j; }
                }
            for (int j = 0; j <= n; j++) {
                if (used[j]) { u[pm[j]] += delta; v[j] -= delta; }
                else minv[j] -= delta;
            }
            j0 = j1;
        } while (pm[j0] != 0);
        do {
            const int j1 = way[j0];
            pm[j0] = pm[j1];
            j0 = j1;
        } while (j0);
    }
    std::vector<int> row_to_col(n, -1);
    for (int j = 1; j <= n; j++) row_to_col[pm[j] - 1] = j - 1;
    return row_to_col;
}

}  // namespace

void make_cluster_plan(const gp_problem *pr, const double *z0, const double *u0, const double *p,
                       ClusterPlan &pl) {
    const int net = pr->n_diff + pr->n_alg;
    const int n_sys = net + 2 * pr->n_bus;
    std::vector<double> zz(n_sys, 0.0), uu(std::max(1, pr->n_ctrl), 0.0), pz(std::max(1, pr->n_par), 0.0);
    std::map<std::vector<int>, int> key_to_class;
    std::vector<std::set<int>> cls_ent, cls_var;
    std::vector<std::vector<int>> cls_loc3;
    pl.cluster_class.assign(pr->n_clusters, -1);
    std::vector<std::vector<int>> members;
    for (int c = 0; c < pr->n_clusters; c++) {
        if (pr->cl_gen[c] < 0) continue;
        const int W = pr->cl_w_size[c], ws = pr->cl_w_start[c];
        std::set<int> ent, var;
        PatSink ps{ws, &ent, &var};
        double C[6], I[2];
        eval_cluster(pr, c, zz.data(), uu.data(), pz.data(), ps, C, I);
        for (int r = 0; r < W; r++)
            if (pr->is_diff[ws + r]) ent.insert(r * 32 + r);
        for (int e : ent) {
            const int r = e / 32, cc = e % 32;
            if (r >= W || (cc >= W && cc < 29)) throw std::runtime_error("cluster entry outside its block");
        }
        const DevRef g = ref(pr->dev[GP_GENROU], pr->cl_gen[c]);
        std::vector<int> loc3 = {g.dp + 5 - ws, g.ap + 2 - ws, g.ap + 3 - ws};
        std::vector<int> key = {W, pr->cl_gov_type[c], pr->cl_exc_type[c], pr->cl_pss[c] >= 0 ? 1 : 0};
        for (int r = 0; r < W; r++) key.push_back(pr->is_diff[ws + r]);
        key.insert(key.end(), loc3.begin(), loc3.end());
        key.insert(key.end(), ent.begin(), ent.end());
        key.push_back(-1);
        key.insert(key.end(), var.begin(), var.end());
        auto it = key_to_class.find(key);
        int cls;
        if (it == key_to_class.end()) {
            cls = (int)cls_ent.size();
            key_to_class[key] = cls;
            cls_ent.push_back(ent);
            cls_var.push_back(var);
            cls_loc3.push_back(loc3);
            pl.cls_W.push_back(W);
            pl.cls_rep.push_back(c);
            members.emplace_back();
        } else {
            cls = it->second;
        }
        pl.cluster_class[c] = cls;
        members[cls].push_back(c);
    }
    pl.n_class = (int)cls_ent.size();
    pl.slot_of.assign((size_t)pl.n_class * 1024, 0);
    pl.perm_col.assign((size_t)pl.n_class * 32, 0);
    pl.pos3.assign((size_t)pl.n_class * 3, 0);
    pl.prog_ptr.assign(1, 0);
    pl.prog_mid.clear();
    pl.prog_sol.clear();
    pl.rhs_base.clear();
    pl.nslot.clear();
    pl.ops.clear();
    pl.max_slots = 0;
    pl.lu_flops = 0;
    pl.n_img.clear();
    pl.diff_mask.clear();
    pl.const_ptr.assign(1, 0);
    pl.const_ops.clear();
    pl.full_ptr.assign(1, 0);
    pl.sol_ptr.assign(1, 0);
    pl.full.clear();
    pl.sol.clear();
    pl.max_img = pl.max_rb = 1;
    std::vector<std::vector<unsigned char>> cls_base;
    const double dt_rep = 1.0 / 120.0;
    for (int cls = 0; cls < pl.n_class; cls++) {
        const int W = pl.cls_W[cls], rep = pl.cls_rep[cls], ws = pr->cl_w_start[rep];
        const std::set<int> &ent = cls_ent[cls];
        std::vector<std::vector<char>> pat(W, std::vector<char>(W, 0));
        for (int e : ent)
            if (e % 32 < W) pat[e / 32][e % 32] = 1;
        // representative values (scenario 0) with the backward-Euler scaling
        std::vector<double> a(1024, 0.0);
        DenseSink ds{ws, a.data()};
        double C[6], I[2];
        eval_cluster(pr, rep, z0, u0, p, ds, C, I);
        std::vector<char> isd(W);
        for (int r = 0; r < W; r++) {
            isd[r] = pr->is_diff[ws + r] ? 1 : 0;
            if (isd[r]) {
                for (int c = 0; c < W; c++) a[r * 32 + c] *= -dt_rep;
                a[r * 32 + r] += 1.0;
            }
        }
        // pivot pairs: differential rows keep their diagonal, algebraic rows
        // are matched to algebraic columns by maximum product of |a_ij|
        std::vector<int> alg;
        for (int r = 0; r < W; r++)
            if (!isd[r]) alg.push_back(r);
        std::vector<int> row_of_col(W);
        for (int r = 0; r < W; r++)
            if (isd[r]) row_of_col[r] = r;
        if (!alg.empty()) {
            const int na = (int)alg.size();
            std::vector<std::vector<double>> cost(na, std::vector<double>(na, 1e30));
            for (int i = 0; i < na; i++)
                for (int j = 0; j < na; j++)
                    if (pat[alg[i]][alg[j]]) {
                        const double v = std::fabs(a[alg[i] * 32 + alg[j]]);
                        cost[i][j] = v > 0.0 ? -std::log(v) : 700.0;
                    }
            std::vector<int> r2c = assign(cost);
            for (int i = 0; i < na; i++) {
                if (!pat[alg[i]][alg[r2c[i]]])
                    throw std::runtime_error("cluster block has no structurally non-singular pivot choice");
                row_of_col[alg[r2c[i]]] = alg[i];
            }
        }
        // minimum-degree order of the pivot pairs (indexed by column)
        std::vector<std::vector<char>> G(W, std::vector<char>(W, 0));
        for (int i = 0; i < W; i++)
            for (int j = 0; j < W; j++)
                if (i != j && pat[row_of_col[i]][j]) G[i][j] = G[j][i] = 1;
        std::vector<int> ord;
        std::vector<char> alive(W, 1);
        for (int step = 0; step < W; step++) {
            int best = -1, bd = 1 << 30;
            for (int v = 0; v < W; v++)
                if (alive[v]) {
                    int dgr = 0;
                    for (int u = 0; u < W; u++) dgr += alive[u] && G[v][u];
                    if (dgr < bd) { bd = dgr; best = v; }
                }
            ord.push_back(best);
            alive[best] = 0;
            for (int x = 0; x < W; x++)
                if (alive[x] && G[best][x])
                    for (int y = 0; y < W; y++)
                        if (alive[y] && G[best][y] && x != y) G[x][y] = 1;
        }
        std::vector<int> ipcol(W), iprow(W);
        for (int k = 0; k < W; k++) {
            ipcol[ord[k]] = k;
            iprow[row_of_col[ord[k]]] = k;
        }
        // symbolic LU of the permuted block
        std::vector<std::vector<char>> Q(W, std::vector<char>(W, 0));
        for (int r = 0; r < W; r++)
            for (int c = 0; c < W; c++)
                if (pat[r][c]) Q[iprow[r]][ipcol[c]] = 1;
        for (int k = 0; k < W; k++) {
            if (!Q[k][k]) throw std::runtime_error("zero structural pivot in a cluster block");
            for (int i = k + 1; i < W; i++)
                if (Q[i][k])
                    for (int j = k + 1; j < W; j++)
                        if (Q[k][j]) Q[i][j] = 1;
        }
        std::vector<std::vector<int>> slot(W, std::vector<int>(W, -1));
        // the state-dependent entries last, after the pivot reciprocals
        std::vector<std::vector<char>> var(W, std::vector<char>(W, 0));
        for (int e : cls_var[cls]) var[iprow[e / 32]][ipcol[e % 32]] = 1;
        int ns = 0;
        for (int i = 0; i < W; i++)
            for (int j = 0; j < W; j++)
                if (Q[i][j] && !var[i][j]) slot[i][j] = ns++;
        const int inv0 = ns, n_img = inv0 + W;
        ns = n_img;
        for (int i = 0; i < W; i++)
            for (int j = 0; j < W; j++)
                if (Q[i][j] && var[i][j]) slot[i][j] = ns++;
        const int rb = ns;
        const int trash = rb + 3 * W;
        const int nslot = trash + 1;
        short *so = pl.slot_of.data() + (size_t)cls * 1024;
        for (int q = 0; q < 1024; q++) so[q] = (short)trash;
        for (int r = 0; r < W; r++) {
            for (int c = 0; c < W; c++)
                if (slot[iprow[r]][ipcol[c]] >= 0) so[r * 32 + c] = (short)slot[iprow[r]][ipcol[c]];
            so[r * 32 + 29] = (short)(rb + iprow[r]);
            so[r * 32 + 30] = (short)(rb + W + iprow[r]);
            so[r * 32 + 31] = (short)(rb + 2 * W + iprow[r]);
        }
        auto op = [&](unsigned char code, int d, int a_, int b) {
            CluOp o;
            o.code = code;
            o.pad = 0;
            o.d = (short)d;
            o.a = (short)a_;
            o.b = (short)b;
            pl.ops.push_back(o);
        };
        // part 1: backward-Euler scaling of the differential rows
        for (int r = 0; r < W; r++) {
            if (!isd[r]) {
                op(OP_ROW, rb + 2 * W + iprow[r], r, 0);
                continue;
            }
            for (int c = 0; c < W; c++)
                if (ent.count(r * 32 + c)) op(OP_SCL, slot[iprow[r]][ipcol[c]], 0, 0);
            if (ent.count(r * 32 + 29)) op(OP_SCL, rb + iprow[r], 0, 0);
            if (ent.count(r * 32 + 30)) op(OP_SCL, rb + W + iprow[r], 0, 0);
            op(OP_DIAG, slot[iprow[r]][ipcol[r]], 0, 0);
            op(OP_BEF, rb + 2 * W + iprow[r], r, 0);
        }
        pl.prog_mid.push_back((int)pl.ops.size());
        // part 2: LU without pivoting on the permuted block, then the solves
        int64_t fl = 0;
        for (int k = 0; k < W; k++) {
            op(OP_RCP, inv0 + k, slot[k][k], 0);
            for (int i = k + 1; i < W; i++)
                if (Q[i][k]) op(OP_MUL, slot[i][k], inv0 + k, 0);
            for (int i = k + 1; i < W; i++)
                if (Q[i][k])
                    for (int j = k + 1; j < W; j++)
                        if (Q[k][j]) { op(OP_FMS, slot[i][j], slot[i][k], slot[k][j]); fl++; }
        }
        pl.prog_sol.push_back((int)pl.ops.size());
        for (int k = 0; k < W; k++)
            for (int i = k + 1; i < W; i++)
                if (Q[i][k]) { op(OP_FMS3, i, slot[i][k], k); fl += 3; }
        for (int k = W - 1; k >= 0; k--) {
            op(OP_MUL3, k, inv0 + k, 0);
            for (int i = 0; i < k; i++)
                if (Q[i][k]) { op(OP_FMS3, i, slot[i][k], k); fl += 3; }
        }
        // the device's form: operations whose operands depend on the
        // parameters and the time step alone (const_ops, in program order),
        // the others, and the solves of the columns with the structural
        // zeros of the two B columns left out
        {
            std::vector<char> cst(rb, 1);
            for (int k = 0; k < W; k++) cst[inv0 + k] = 0;
            for (int sl = n_img; sl < rb; sl++) cst[sl] = 0;
            std::vector<SlotOp> full, sol;
            for (int q = pl.prog_mid.back(); q < pl.prog_sol.back(); q++) {
                const CluOp &o = pl.ops[q];
                const bool c = cst[o.a] && (o.code == OP_RCP || cst[o.d]) && (o.code != OP_FMS || cst[o.b]);
                cst[o.d] = c;
                if (c) pl.const_ops.push_back(o);
                else
                    full.push_back(SlotOp{o.code == OP_RCP ? REC_RCP : (o.code == OP_MUL ? REC_MUL : REC_FMS), o.d,
                                          o.a, o.b});
            }
            pl.const_ptr.push_back((int)pl.const_ops.size());
            std::vector<char> nz(3 * W, 0);
            for (int r = 0; r < W; r++) {
                nz[iprow[r]] = ent.count(r * 32 + 29) ? 1 : 0;
                nz[W + iprow[r]] = ent.count(r * 32 + 30) ? 1 : 0;
                nz[2 * W + iprow[r]] = 1;
            }
            for (int q = pl.prog_sol.back(); q < (int)pl.ops.size(); q++) {
                const CluOp &o = pl.ops[q];
                const int code = o.code == OP_MUL3 ? REC_MUL : REC_FMS;
                for (int c = 0; c < 3; c++) {
                    if (!nz[c * W + (code == REC_FMS ? o.b : o.d)]) continue;
                    nz[c * W + o.d] = 1;
                    full.push_back(SlotOp{code, rb + c * W + o.d, o.a, code == REC_FMS ? rb + c * W + o.b : 0});
                }
                // (d, b shifted past the LU slots for the dependencies)
                sol.push_back(SlotOp{code, rb + o.d, o.a, code == REC_FMS ? rb + o.b : 0});
            }
            std::vector<CluRec> st[kCluWarps];
            schedule(full, rb + 3 * W, st);
            for (int w = 0; w < kCluWarps; w++) {
                pl.full.insert(pl.full.end(), st[w].begin(), st[w].end());
                pl.full_ptr.push_back((int)pl.full.size() / 2);
                st[w].clear();
            }
            schedule(sol, rb + W, st);
            for (int w = 0; w < kCluWarps; w++) {
                for (CluRec &r : st[w]) {
                    r.d = std::max(0, r.d - rb * 32);
                    r.b = std::max(0, r.b - rb * 32);
                }
                pl.sol.insert(pl.sol.end(), st[w].begin(), st[w].end());
                pl.sol_ptr.push_back((int)pl.sol.size() / 2);
            }
            std::vector<unsigned char> base(rb, 0);
            unsigned dm = 0;
            for (int r = 0; r < W; r++)
                if (isd[r]) {
                    dm |= 1u << r;
                    base[slot[iprow[r]][ipcol[r]]] |= 1;
                }
            for (int k = 0; k < W; k++) base[slot[k][k]] |= 2;
            cls_base.push_back(base);
            pl.diff_mask.push_back(dm);
            pl.n_img.push_back(n_img);
            pl.max_img = std::max(pl.max_img, n_img);
            pl.max_rb = std::max(pl.max_rb, rb);
        }
        pl.prog_ptr.push_back((int)pl.ops.size());
        pl.rhs_base.push_back(rb);
        pl.nslot.push_back(nslot);
        pl.max_slots = std::max(pl.max_slots, nslot);
        for (int j = 0; j < W; j++) pl.perm_col[(size_t)cls * 32 + j] = ord[j];
        for (int t = 0; t < 3; t++) pl.pos3[(size_t)cls * 3 + t] = ipcol[cls_loc3[cls][t]];
        pl.lu_flops += fl * (int64_t)members[cls].size();
    }
    pl.base_stride = pl.max_rb;
    pl.base.assign((size_t)std::max(1, pl.n_class) * pl.base_stride, 0);
    for (int cls = 0; cls < pl.n_class; cls++)
        std::copy(cls_base[cls].begin(), cls_base[cls].end(), pl.base.begin() + (size_t)cls * pl.base_stride);
    // warp tasks: 32 clusters of one class, the classes with the most slots
    // (the longest programs) first, so that the warps that start last are
    // the short ones
    pl.order.clear();
    pl.task_class.clear();
    pl.task_first.clear();
    pl.task_count.clear();
    std::vector<int> by_len(pl.n_class);
    for (int cls = 0; cls < pl.n_class; cls++) by_len[cls] = cls;
    std::stable_sort(by_len.begin(), by_len.end(), [&](int a, int b) { return pl.nslot[a] > pl.nslot[b]; });
    for (int cls : by_len) {
        const int first = (int)pl.order.size();
        pl.order.insert(pl.order.end(), members[cls].begin(), members[cls].end());
        for (size_t s = 0; s < members[cls].size(); s += 32) {
            pl.task_class.push_back(cls);
            pl.task_first.push_back(first + (int)s);
            pl.task_count.push_back((int)std::min<size_t>(32, members[cls].size() - s));
        }
    }
}

double host_cluster_run(const gp_problem *pr, const ClusterPlan &pl, int c, const double *z, const double *zold,
                        const double *u0, const double *p, double dt, double *yx, double *out8, double *f_out) {
    const int cls = pl.cluster_class[c];
    if (cls < 0) throw std::runtime_error("trivial cluster has no program");
    const int W = pl.cls_W[cls], ws = pr->cl_w_start[c];
    std::vector<double> v(pl.nslot[cls], 0.0);
    const int rb = pl.rhs_base[cls];
    double *R0 = v.data() + rb, *R1 = R0 + W, *R2 = R1 + W;
    // the constant entries and their part of the factorisation, taken at
    // another state (as on the device, whose image is of an earlier one): an
    // entry wrongly marked constant shows
    std::vector<double> z_img(z, z + pr->n_diff + pr->n_alg + 2 * pr->n_bus);
    for (double &x : z_img) x = 0.37 - 0.6 * x;
    const unsigned char *base = pl.base.data() + (size_t)cls * pl.base_stride;
    for (int s = 0; s < rb; s++)
        if (base[s] & 1) v[s] = 1.0;
    double C[6], I[2];
    SlotSink si{ws, pl.slot_of.data() + (size_t)cls * 1024, v.data(), pl.diff_mask[cls], dt, true, z, zold};
    eval_cluster(pr, c, z_img.data(), u0, p, si, C, I);
    for (int q = pl.const_ptr[cls]; q < pl.const_ptr[cls + 1]; q++) {
        const CluOp &o = pl.const_ops[q];
        if (o.code == OP_RCP) v[o.d] = 1.0 / v[o.a];
        else if (o.code == OP_MUL) v[o.d] *= v[o.a];
        else v[o.d] -= v[o.a] * v[o.b];
    }
    // the state-dependent entries and the residual
    si.image = false;
    eval_cluster(pr, c, z, u0, p, si, C, I);
    double fmax = 0.0;
    for (int j = 0; j < W; j++) fmax = std::max(fmax, std::fabs(R2[j]));
    if (f_out)
        for (int r = 0; r < W; r++) f_out[r] = v[pl.slot_of[(size_t)cls * 1024 + r * 32 + 31]];
    // the staged operations, stage by stage, the last warp's share first
    int pos[kCluWarps];
    for (int w = 0; w < kCluWarps; w++) pos[w] = pl.full_ptr[(size_t)cls * kCluWarps + w];
    while (pos[0] < pl.full_ptr[(size_t)cls * kCluWarps + 1])
        for (int w = kCluWarps - 1; w >= 0; w--)
            for (bool more = true; more;) {
                const CluRec *r = pl.full.data() + 2 * (size_t)pos[w]++;
                for (int h = 0; h < 2; h++) {
                    const int code = h ? r[0].w >> 4 & 15 : r[0].w & 15;
                    double &d = v[r[h].d / 32];
                    if (code == REC_FMS) d -= v[r[h].a / 32] * v[r[h].b / 32];
                    else if (code == REC_MUL) d *= v[r[h].a / 32];
                    else if (code == REC_RCP) d = 1.0 / v[r[h].a / 32];
                }
                more = !(r[0].w & REC_SYNC);
            }
    for (int j = 0; j < W; j++) {
        const int st = pl.perm_col[(size_t)cls * 32 + j];
        yx[st] = R2[j];
        yx[W + st] = R0[j];
        yx[2 * W + st] = R1[j];
    }
    const int *p3 = pl.pos3.data() + (size_t)cls * 3;
    double X1[3], X2[3], Y[3];
    for (int t = 0; t < 3; t++) {
        X1[t] = R0[p3[t]];
        X2[t] = R1[p3[t]];
        Y[t] = R2[p3[t]];
    }
    out8[0] = C[0] * X1[0] + C[1] * X1[1] + C[2] * X1[2];
    out8[1] = C[0] * X2[0] + C[1] * X2[1] + C[2] * X2[2];
    out8[2] = C[3] * X1[0] + C[4] * X1[1] + C[5] * X1[2];
    out8[3] = C[3] * X2[0] + C[4] * X2[1] + C[5] * X2[2];
    out8[4] = C[0] * Y[0] + C[1] * Y[1] + C[2] * Y[2];
    out8[5] = C[3] * Y[0] + C[4] * Y[1] + C[5] * Y[2];
    out8[6] = I[0];
    out8[7] = I[1];
    return fmax;
}

}  // namespace gp
