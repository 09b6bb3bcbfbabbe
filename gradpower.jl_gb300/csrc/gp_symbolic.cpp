// Host-once symbolic analysis: nested dissection on the bus graph, the
// elimination tree, fundamental supernodes, multifrontal front layout and
// the level schedule.  See gp_symbolic.h.
#include "gp_symbolic.h"

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <future>
#include <queue>
#include <stdexcept>
#include <system_error>
#include <thread>

namespace gp {
namespace {

struct Graph {
    int n = 0;
    std::vector<int> ptr, adj;
};

// Minimum-degree order of a small induced subgraph (|V| <= 64) using an
// explicit elimination graph held in 64-bit masks.
void leaf_min_degree(const Graph &G, const std::vector<int> &V, std::vector<int> &order) {
    const int k = (int)V.size();
    std::vector<std::pair<int, int>> at(k);   // node -> place in V
    for (int a = 0; a < k; a++) at[a] = {V[a], a};
    std::sort(at.begin(), at.end());
    uint64_t m[64] = {};
    for (int a = 0; a < k; a++) {
        int v = V[a];
        for (int q = G.ptr[v]; q < G.ptr[v + 1]; q++) {
            auto it = std::lower_bound(at.begin(), at.end(), std::make_pair(G.adj[q], 0));
            if (it != at.end() && it->first == G.adj[q] && it->second != a) m[a] |= (uint64_t)1 << it->second;
        }
    }
    uint64_t alive = (k == 64) ? ~(uint64_t)0 : (((uint64_t)1 << k) - 1);
    for (int step = 0; step < k; step++) {
        int best = -1, bd = 1 << 30;
        for (int a = 0; a < k; a++)
            if (alive >> a & 1) {
                int d = __builtin_popcountll(m[a] & alive);
                if (d < bd) { bd = d; best = a; }
            }
        uint64_t nb = m[best] & alive & ~((uint64_t)1 << best);
        for (int a = 0; a < k; a++)
            if (nb >> a & 1) m[a] |= nb & ~((uint64_t)1 << a);
        alive &= ~((uint64_t)1 << best);
        order.push_back(V[best]);
    }
}

// Nested dissection.  The two halves of a large set are ordered by two
// threads: a call touches its own set's entries of the arrays below and, of
// set_id, reads its neighbours' (atomics: another call may be writing them;
// no value but a node's own set's equals its id).  The order does not depend
// on the threads.
struct ND {
    const Graph &G;
    std::vector<std::atomic<int>> set_id;
    std::vector<int> lev;
    std::atomic<int> next_id{1};
    // sets of at least PAR nodes give one half to another thread (analysis of
    // 70,000 buses on eight cores 630 -> 295 ms, of 2,000 20 -> 10)
    static constexpr int PAR = 200;
    // threads that may be started beside the caller's: a core each, and as
    // many again for those that wait for their half; the rest runs inline,
    // as where a thread cannot be had
    std::atomic<int> spare{2 * (int)std::max(1u, std::thread::hardware_concurrency())};
    int set_of(int v) const { return set_id[v].load(std::memory_order_relaxed); }
    void assign(const std::vector<int> &V, int id) {
        for (int v : V) set_id[v].store(id, std::memory_order_relaxed);
    }
    // sets of at most LEAF nodes are ordered by minimum degree as a whole;
    // separators and sets that do not split, in chunks of CHUNK.  LEAF 6
    // against 48: the tree of the 39-bus ring has 4 levels instead of 6, the
    // one of 70,000 buses 23,565 supernodes instead of 26,477 and 13 levels
    // instead of 16; FP64 runs of 70,000 buses x 8 57.0 -> 50.6 ms, 2,000 x
    // 64 39.2 -> 34.6.  (8: 4 and 23,775; 4 and 3 have fewer flops but more
    // supernodes.)
    static constexpr int LEAF = 6, CHUNK = 48;

    explicit ND(const Graph &g)
        : G(g), set_id(g.n), lev(g.n, -1), part(g.n, 0), stamp(g.n, 0) {
        for (auto &s : set_id) s.store(0, std::memory_order_relaxed);
    }

    // BFS inside the set `sid` from r; fills lev for visited nodes and
    // returns the visited nodes in BFS order.
    void bfs(int r, int sid, std::vector<int> &visit) {
        visit.clear();
        visit.push_back(r);
        lev[r] = 0;
        for (size_t h = 0; h < visit.size(); h++) {
            int u = visit[h];
            for (int q = G.ptr[u]; q < G.ptr[u + 1]; q++) {
                int v = G.adj[q];
                if (set_of(v) == sid && lev[v] < 0) {
                    lev[v] = lev[u] + 1;
                    visit.push_back(v);
                }
            }
        }
    }

    void clear_lev(const std::vector<int> &V) {
        for (int v : V) lev[v] = -1;
    }

    // Splits the connected set V into A, B and a separator S: the smallest
    // of the breadth-first level sets near the middle, seen from r and from
    // the far end, each then refined (part: 0 A, 1 B, 2 S).  Against the
    // median level alone, unrefined (and leaves of 48), on the 70,000-bus
    // grid: largest front 132 -> 40 rows, factorisation flops 33.7 -> 19.4 M
    // a scenario, levels 30 -> 16; FP64 run of 8 scenarios x 18 steps 104 -> 58 ms (its
    // factorisations 78 -> 36 ms), mixed (36 steps) 70 -> 56 ms.
    std::vector<signed char> part;
    void split(const std::vector<int> &V, int r, int sid, int &pass_id, std::vector<int> &A, std::vector<int> &B,
               std::vector<int> &S) {
        std::vector<int> visit, best;
        std::vector<signed char> best_part;
        double best_cost = 1e300;
        for (int side = 0; side < 2; side++) {
            clear_lev(V);
            bfs(r, sid, visit);
            const int nlev = lev[visit.back()] + 1, n = (int)V.size(), far = visit.back();
            std::vector<int> cnt(nlev, 0);
            for (int v : V) cnt[lev[v]]++;
            // the smallest levels with at least a third of the nodes on
            // either side, and the median one
            std::vector<std::pair<int, int>> cand;
            int acc = 0, median = -1;
            for (int l = 0; l < nlev; l++) {
                if (l > 0 && l < nlev - 1 && acc >= n / 3 && n - acc - cnt[l] >= n / 3) cand.push_back({cnt[l], l});
                acc += cnt[l];
                if (median < 0 && 2 * acc >= n) median = std::max(0, std::min(l, nlev - 2));
            }
            std::sort(cand.begin(), cand.end());
            if (cand.size() > 3) cand.resize(3);
            cand.push_back({0, median});
            for (auto &c : cand) {
                const int l = c.second;
                for (int v : V) {
                    if (lev[v] != l) {
                        part[v] = lev[v] < l ? 0 : 1;
                        continue;
                    }
                    bool touches = false;
                    for (int q = G.ptr[v]; q < G.ptr[v + 1] && !touches; q++) {
                        const int u = G.adj[q];
                        touches = set_of(u) == sid && lev[u] == l + 1;
                    }
                    part[v] = touches ? 2 : 0;
                }
                const double cost = refine(V, sid, pass_id);
                if (cost < best_cost) {
                    best_cost = cost;
                    best_part.resize(V.size());
                    for (size_t i = 0; i < V.size(); i++) best_part[i] = part[V[i]];
                }
            }
            r = far;
        }
        clear_lev(V);
        for (size_t i = 0; i < V.size(); i++)
            (best_part[i] == 0 ? A : (best_part[i] == 1 ? B : S)).push_back(V[i]);
    }

    // Vertex-separator refinement (C. Fiduccia, R. Mattheyses, "A linear-time
    // heuristic for improving network partitions", DAC 1982, in its form for
    // vertex separators): a separator node moves to one side and pulls its
    // neighbours on the other side into the separator; the moves of a pass
    // are taken back to its best point.  Returns the separator's cost.
    std::vector<int> stamp;
    double refine(const std::vector<int> &V, int sid, int &pass_id) {
        const int n = (int)V.size();
        int w[3] = {0, 0, 0};
        for (int v : V) w[(int)part[v]]++;
        const int lo = std::max(1, (int)(0.3 * n));
        auto cost = [&] {
            const double bal = std::max(w[0], w[1]) / (double)std::max(1, std::min(w[0], w[1]));
            return w[2] * (1.0 + 0.1 * std::max(0.0, bal - 1.2)) + (w[0] == 0 || w[1] == 0 ? 1e9 : 0.0);
        };
        auto pulls = [&](int v, int to) {
            int k = 0;
            for (int q = G.ptr[v]; q < G.ptr[v + 1]; q++) k += set_of(G.adj[q]) == sid && part[G.adj[q]] == 1 - to;
            return k;
        };
        double best = cost();
        for (int pass = 0; pass < 6; pass++) {
            using Item = std::pair<int, std::pair<int, int>>;   // gain, node, side
            std::priority_queue<Item> heap;
            auto push = [&](int v) {
                for (int to = 0; to < 2; to++) heap.push({1 - pulls(v, to), {v, to}});
            };
            pass_id++;
            for (int v : V)
                if (part[v] == 2) push(v);
            std::vector<std::pair<int, signed char>> undo;
            size_t keep = 0;
            const double start = best;
            int since = 0;
            while (!heap.empty() && since < 20) {
                const Item it = heap.top();
                heap.pop();
                const int v = it.second.first, to = it.second.second;
                if (part[v] != 2 || stamp[v] == pass_id) continue;
                const int k = pulls(v, to);
                if (1 - k != it.first) {
                    heap.push({1 - k, {v, to}});
                    continue;
                }
                if (w[1 - to] - k < lo) continue;
                stamp[v] = pass_id;   // (a node leaves the separator once a pass)
                undo.push_back({v, 2});
                part[v] = (signed char)to;
                w[2]--;
                w[to]++;
                for (int q = G.ptr[v]; q < G.ptr[v + 1]; q++) {
                    const int u = G.adj[q];
                    if (set_of(u) != sid || part[u] != 1 - to) continue;
                    undo.push_back({u, (signed char)(1 - to)});
                    part[u] = 2;
                    w[1 - to]--;
                    w[2]++;
                    push(u);
                }
                // separator nodes beside v gained or lost a neighbour
                for (int q = G.ptr[v]; q < G.ptr[v + 1]; q++) {
                    const int u = G.adj[q];
                    if (set_of(u) == sid && part[u] == 2 && stamp[u] != pass_id) push(u);
                }
                const double c = cost();
                since++;
                if (c < best) {
                    best = c;
                    keep = undo.size();
                    since = 0;
                }
            }
            while (undo.size() > keep) {
                const auto u = undo.back();
                undo.pop_back();
                w[(int)part[u.first]]--;
                part[u.first] = u.second;
                w[(int)u.second]++;
            }
            if (best >= start) break;
        }
        return best;
    }
    // pass_id: refinement passes on the path to this set (a node's stamps
    // are of earlier ones)
    void run(std::vector<int> V, int sid, int pass_id, std::vector<int> &order) {
        if ((int)V.size() <= LEAF) {
            leaf_min_degree(G, V, order);
            return;
        }
        // connected components
        std::vector<int> visit;
        bfs(V[0], sid, visit);
        if (visit.size() < V.size()) {
            std::vector<std::vector<int>> comps;
            comps.push_back(visit);
            for (int v : V)
                if (lev[v] < 0) {
                    std::vector<int> c;
                    bfs(v, sid, c);
                    comps.push_back(c);
                }
            clear_lev(V);
            for (auto &c : comps) {
                int id = next_id++;
                assign(c, id);
                run(c, id, pass_id, order);
            }
            return;
        }
        // pseudo-peripheral start: repeat BFS from a farthest, lowest-degree node
        int r = V[0];
        int depth = -1;
        for (int t = 0; t < 4; t++) {
            clear_lev(V);
            bfs(r, sid, visit);
            int d = lev[visit.back()];
            if (d <= depth) break;
            depth = d;
            int best = visit.back(), bd = 1 << 30;
            for (int i = (int)visit.size() - 1; i >= 0 && lev[visit[i]] == d; i--) {
                int v = visit[i];
                int dg = 0;
                for (int q = G.ptr[v]; q < G.ptr[v + 1]; q++) dg += set_of(G.adj[q]) == sid;
                if (dg < bd) { bd = dg; best = v; }
            }
            r = best;
        }
        std::vector<int> A, B, S;
        split(V, r, sid, pass_id, A, B, S);
        if (A.empty() || B.empty()) {
            // no useful split: order the whole set by minimum degree on its
            // own adjacency (ties in BFS order)
            std::vector<int> tmp = V;
            while (!tmp.empty()) {
                size_t take = std::min<size_t>(CHUNK, tmp.size());
                std::vector<int> chunk(tmp.begin(), tmp.begin() + take);
                leaf_min_degree(G, chunk, order);
                tmp.erase(tmp.begin(), tmp.begin() + take);
            }
            return;
        }
        int ida = next_id++, idb = next_id++, ids = next_id++;
        assign(A, ida);
        assign(B, idb);
        assign(S, ids);
        std::vector<int> ob;
        std::future<void> half;
        if ((int)V.size() >= PAR) {
            if (spare.fetch_sub(1) > 0) {
                try {
                    half = std::async(std::launch::async, [&] { run(B, idb, pass_id, ob); });
                } catch (const std::system_error &) {   // (the process may start no more threads)
                }
            }
            if (!half.valid()) spare.fetch_add(1);
        }
        run(A, ida, pass_id, order);
        if (half.valid()) {
            half.get();
            spare.fetch_add(1);
            order.insert(order.end(), ob.begin(), ob.end());
        } else {
            run(B, idb, pass_id, order);
        }
        // separator nodes: order them by minimum degree in chunks
        for (size_t a = 0; a < S.size(); a += CHUNK) {
            std::vector<int> chunk(S.begin() + a, S.begin() + std::min(S.size(), a + CHUNK));
            leaf_min_degree(G, chunk, order);
        }
    }
};

void merge_into(std::vector<int> &dst, const std::vector<int> &src, int skip_le) {
    // dst := dst ∪ {x in src : x > skip_le}, both sorted
    std::vector<int> out;
    out.reserve(dst.size() + src.size());
    size_t i = 0, j = 0;
    while (j < src.size() && src[j] <= skip_le) j++;
    while (i < dst.size() || j < src.size()) {
        int x;
        if (j >= src.size() || (i < dst.size() && dst[i] < src[j])) x = dst[i++];
        else if (i >= dst.size() || src[j] < dst[i]) x = src[j++];
        else { x = dst[i++]; j++; }
        out.push_back(x);
    }
    dst.swap(out);
}

}  // namespace

void analyse(int n, const std::vector<int> &rowptr, const std::vector<int> &colidx,
             const std::vector<int> &group, int n_nodes, Symbolic &S) {
    // ---- node graph ----
    Graph G;
    G.n = n_nodes;
    {
        std::vector<std::vector<int>> nb(n_nodes);
        for (int i = 0; i < n; i++)
            for (int q = rowptr[i]; q < rowptr[i + 1]; q++) {
                int a = group[i], b = group[colidx[q]];
                if (a != b) { nb[a].push_back(b); nb[b].push_back(a); }
            }
        G.ptr.assign(n_nodes + 1, 0);
        for (int a = 0; a < n_nodes; a++) {
            std::sort(nb[a].begin(), nb[a].end());
            nb[a].erase(std::unique(nb[a].begin(), nb[a].end()), nb[a].end());
            G.ptr[a + 1] = G.ptr[a] + (int)nb[a].size();
        }
        G.adj.reserve(G.ptr[n_nodes]);
        for (int a = 0; a < n_nodes; a++) G.adj.insert(G.adj.end(), nb[a].begin(), nb[a].end());
    }
    // ---- nested dissection on nodes ----
    ND nd(G);
    std::vector<int> node_order;
    {
        std::vector<int> all(n_nodes);
        for (int a = 0; a < n_nodes; a++) all[a] = a;
        nd.run(all, 0, 0, node_order);
    }
    if ((int)node_order.size() != n_nodes) throw std::runtime_error("nested dissection lost nodes");
    // ---- expand to scalar unknowns ----
    std::vector<std::vector<int>> members(n_nodes);
    for (int i = 0; i < n; i++) members[group[i]].push_back(i);
    S.n = n;
    S.perm.clear();
    S.perm.reserve(n);
    for (int a : node_order)
        for (int i : members[a]) S.perm.push_back(i);
    if ((int)S.perm.size() != n) throw std::runtime_error("unknowns without a node");
    // ---- elimination tree of the dissection's order, then of its postorder
    // with the column structures ----
    std::vector<int> par, nchild;
    std::vector<std::vector<int>> cs;
    for (int round = 0; round < 2; round++) {
        S.iperm.assign(n, 0);
        for (int k = 0; k < n; k++) S.iperm[S.perm[k]] = k;
        // lower part per column (sorted), and by row for the tree
        std::vector<int> up_ptr(n + 1, 0);
        for (int i = 0; i < n; i++)
            for (int q = rowptr[i]; q < rowptr[i + 1]; q++) {
                const int a = S.iperm[i], b = S.iperm[colidx[q]];
                if (a != b) up_ptr[std::max(a, b) + 1]++;
            }
        for (int j = 0; j < n; j++) up_ptr[j + 1] += up_ptr[j];
        std::vector<int> upp(up_ptr[n]), at(up_ptr.begin(), up_ptr.end() - 1);
        for (int i = 0; i < n; i++)
            for (int q = rowptr[i]; q < rowptr[i + 1]; q++) {
                const int a = S.iperm[i], b = S.iperm[colidx[q]];
                if (a != b) upp[at[std::max(a, b)]++] = std::min(a, b);
            }
        // elimination tree (Liu, path compression)
        par.assign(n, -1);
        std::vector<int> anc(n, -1);
        for (int j = 0; j < n; j++)
            for (int q = up_ptr[j]; q < up_ptr[j + 1]; q++) {
                int r = upp[q];
                while (anc[r] != -1 && anc[r] != j) {
                    int nx = anc[r];
                    anc[r] = j;
                    r = nx;
                }
                if (anc[r] == -1) { anc[r] = j; par[r] = j; }
            }
        nchild.assign(n, 0);
        std::vector<std::vector<int>> kids(n);
        for (int j = 0; j < n; j++)
            if (par[j] >= 0) {
                nchild[par[j]]++;
                kids[par[j]].push_back(j);
            }
        if (round == 1) {
            // column structures: the rows below a column's diagonal and
            // those its children pass on (the rows come in increasing order)
            cs.assign(n, {});
            for (int i = 0; i < n; i++)
                for (int q = up_ptr[i]; q < up_ptr[i + 1]; q++)
                    if (cs[upp[q]].empty() || cs[upp[q]].back() != i) cs[upp[q]].push_back(i);
            for (int j = 0; j < n; j++)
                for (int c : kids[j]) merge_into(cs[j], cs[c], j);
            break;
        }
        // postorder, each column's child with the tallest subtree last: the
        // supernode that a merge can join to its parent's columns (they
        // must follow it directly) is then the one on the longest path.
        // (The unknowns of a node stay adjacent: each has the one before it
        // as its only child, since whatever reaches a node reaches its
        // first unknown.)
        std::vector<int> height(n, 0), post;
        for (int j = 0; j < n; j++)
            if (par[j] >= 0) height[par[j]] = std::max(height[par[j]], height[j] + 1);
        post.reserve(n);
        std::vector<std::pair<int, size_t>> walk;
        for (int j = 0; j < n; j++) {
            std::stable_sort(kids[j].begin(), kids[j].end(), [&](int a, int b) {
                return height[a] < height[b];
            });
        }
        for (int root = 0; root < n; root++) {
            if (par[root] >= 0) continue;
            walk.push_back({root, 0});
            while (!walk.empty()) {
                auto &w = walk.back();
                if (w.second < kids[w.first].size()) {
                    const int c = kids[w.first][w.second++];
                    walk.push_back({c, 0});
                } else {
                    post.push_back(w.first);
                    walk.pop_back();
                }
            }
        }
        std::vector<int> perm(n);
        for (int k = 0; k < n; k++) perm[k] = S.perm[post[k]];
        S.perm.swap(perm);
    }
    // ---- fundamental supernodes ----
    std::vector<int> fstart;
    for (int j = 0; j < n; j++) {
        bool join = j > 0 && par[j - 1] == j && nchild[j] == 1 && cs[j - 1].size() == cs[j].size() + 1;
        if (!join) fstart.push_back(j);
    }
    int nf = (int)fstart.size();
    fstart.push_back(n);
    // ---- amalgamation: merge a supernode into its parent when the parent's
    // columns follow it directly and the merge adds no explicit zero, or when
    // the merged supernode has at most 24 columns and less than a fifth of
    // its entries are zeros.  Every level costs the factorisation and the
    // solves a hand-off (3 to 10 us), every zero FP64 work: this rule against
    // at most two zeros a column (widths to 48), and against a share of 0.35
    // (widths to 12) or 0.2 (to 32), FP64 runs: 70,000 buses x 8 (18 steps)
    // 58.0, 59.1, 59.6 ms, 9,001 x 3 29.2, 28.0, 30.7, 39 x 64 53.0, 61, 54.6
    // ----
    {
        std::vector<int> fsup_of(n);
        for (int f = 0; f < nf; f++)
            for (int j = fstart[f]; j < fstart[f + 1]; j++) fsup_of[j] = f;
        std::vector<int> st(fstart.begin(), fstart.end() - 1), ncol(nf), fpar(nf, -1);
        std::vector<char> gone(nf, 0);
        std::vector<int64_t> zeros(nf, 0);   // explicit zeros of the merged supernode, one triangle
        for (int f = 0; f < nf; f++) {
            ncol[f] = fstart[f + 1] - fstart[f];
            int last = fstart[f + 1] - 1;
            if (par[last] >= 0) fpar[f] = fsup_of[par[last]];
        }
        for (int f = 0; f < nf; f++) {
            int p = fpar[f];
            if (p < 0 || fstart[f + 1] != st[p]) continue;
            int64_t rs = (int64_t)cs[fstart[f + 1] - 1].size();
            int64_t rp = (int64_t)cs[fstart[p + 1] - 1].size();
            int64_t extra = (int64_t)ncol[f] * (ncol[p] + rp - rs);
            int64_t width = ncol[f] + ncol[p];
            zeros[p] += zeros[f] + extra;
            const double share = (double)zeros[p] / (double)(width * (width + 2 * rp));
            const bool ok = extra == 0 || (width <= 24 && share < 0.2);
            if (!ok) {
                zeros[p] -= zeros[f] + extra;
                continue;
            }
            st[p] = st[f];
            ncol[p] += ncol[f];
            gone[f] = 1;
        }
        S.sup_start.clear();
        for (int f = 0; f < nf; f++)
            if (!gone[f]) S.sup_start.push_back(st[f]);
        std::sort(S.sup_start.begin(), S.sup_start.end());
    }
    S.nsup = (int)S.sup_start.size();
    S.sup_start.push_back(n);
    S.sup_of.assign(n, 0);
    for (int s = 0; s < S.nsup; s++)
        for (int j = S.sup_start[s]; j < S.sup_start[s + 1]; j++) S.sup_of[j] = s;
    S.row_ptr.assign(S.nsup + 1, 0);
    S.rows.clear();
    for (int s = 0; s < S.nsup; s++) {
        int last = S.sup_start[s + 1] - 1;
        S.rows.insert(S.rows.end(), cs[last].begin(), cs[last].end());
        S.row_ptr[s + 1] = (int)S.rows.size();
    }
    S.parent.assign(S.nsup, -1);
    for (int s = 0; s < S.nsup; s++) {
        int last = S.sup_start[s + 1] - 1;
        if (par[last] >= 0) S.parent[s] = S.sup_of[par[last]];
    }
    // children
    std::vector<int> ccount(S.nsup + 1, 0);
    for (int s = 0; s < S.nsup; s++)
        if (S.parent[s] >= 0) ccount[S.parent[s] + 1]++;
    S.child_ptr.assign(S.nsup + 1, 0);
    for (int s = 0; s < S.nsup; s++) S.child_ptr[s + 1] = S.child_ptr[s] + ccount[s + 1];
    S.children.assign(S.child_ptr[S.nsup], 0);
    {
        std::vector<int> fill(S.child_ptr.begin(), S.child_ptr.end() - 1);
        for (int s = 0; s < S.nsup; s++)
            if (S.parent[s] >= 0) S.children[fill[S.parent[s]]++] = s;
    }
    // levels (children have smaller indices than parents)
    S.level.assign(S.nsup, 0);
    S.nlevels = 0;
    for (int s = 0; s < S.nsup; s++) {
        int lv = 0;
        for (int q = S.child_ptr[s]; q < S.child_ptr[s + 1]; q++) lv = std::max(lv, S.level[S.children[q]] + 1);
        S.level[s] = lv;
        S.nlevels = std::max(S.nlevels, lv + 1);
    }
    S.level_ptr.assign(S.nlevels + 1, 0);
    for (int s = 0; s < S.nsup; s++) S.level_ptr[S.level[s] + 1]++;
    for (int l = 0; l < S.nlevels; l++) S.level_ptr[l + 1] += S.level_ptr[l];
    S.level_sups.assign(S.nsup, 0);
    {
        std::vector<int> fill(S.level_ptr.begin(), S.level_ptr.end() - 1);
        for (int s = 0; s < S.nsup; s++) S.level_sups[fill[S.level[s]]++] = s;
    }
    // fronts, update vectors, relative maps, costs
    S.front_off.assign(S.nsup + 1, 0);
    S.uvec_off.assign(S.nsup + 1, 0);
    S.relmap_ptr.assign(S.nsup + 1, 0);
    S.nnz_lu = 0;
    S.flops = 0.0;
    S.max_front = 0;
    for (int s = 0; s < S.nsup; s++) {
        int m = S.front_m(s), ns = S.front_n(s), r = S.front_r(s);
        S.front_off[s + 1] = S.front_off[s] + (int64_t)m * m;
        S.uvec_off[s + 1] = S.uvec_off[s] + r;
        S.relmap_ptr[s + 1] = S.relmap_ptr[s] + r;
        S.nnz_lu += (int64_t)ns * ns + 2LL * ns * r;
        for (int k = 0; k < ns; k++) {
            double t = m - k - 1;
            S.flops += t + 2.0 * t * t;
        }
        S.max_front = std::max(S.max_front, m);
    }
    S.relmap.assign(S.relmap_ptr[S.nsup], 0);
    for (int c = 0; c < S.nsup; c++) {
        int s = S.parent[c];
        int base = S.relmap_ptr[c];
        for (int a = 0; a < S.front_r(c); a++) {
            int i = S.rows[S.row_ptr[c] + a];
            if (s < 0) throw std::runtime_error("root supernode with a non-empty row structure");
            int pos;
            if (i < S.sup_start[s + 1]) {
                pos = i - S.sup_start[s];
                if (pos < 0) throw std::runtime_error("relative index below parent");
            } else {
                auto b = S.rows.begin() + S.row_ptr[s], e = S.rows.begin() + S.row_ptr[s + 1];
                auto it = std::lower_bound(b, e, i);
                if (it == e || *it != i) throw std::runtime_error("child row missing from parent structure");
                pos = S.front_n(s) + (int)(it - b);
            }
            S.relmap[base + a] = pos;
        }
    }
}

}  // namespace gp
