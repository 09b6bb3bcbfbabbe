// Small systems: the whole FP64 Newton iteration of a scenario in one CTA,
// and as many backward-Euler steps as lie between two events in one launch.
//
// For a system of a few dozen buses the batch kernels (gp_kernels.cu,
// gp_dag.cu, gp_solve.cu) spend their time between the arithmetic: eight
// launches an iteration, claims, flags and round trips to L2 for fronts of a
// few hundred entries.  Here a scenario's state, cluster results, reduced
// matrix (its fronts) and right-hand side stay in the shared memory of one
// SM, scenarios never wait for one another, and the phases of an iteration
// meet at CTA barriers:
//  - the cluster tasks, kCluWarps warps each (gp_cluster.cuh);
//  - the network rows, a thread a bus (gp_network.cuh), and the residual norm;
//  - the factorisation, a warp a front, the levels of the assembly tree one
//    after the other, the right-hand side as an extra column;
//  - the backward solve, levels in reverse, and the update.
// What bounds it: the FP64 pipe's 64 cycles per warp instruction along the
// elimination's columns and the cluster programs' stages (latency, not
// throughput: 39 buses leave most of the SM idle).
// Every value receives the operations of the batch kernels, in their order.
// Measured, ms a call, batch kernels -> this: 2 buses x 1, 60 steps 8.4 -> 3.1;
// 39 buses x 64, 120 steps 46 -> 19.0 (an iteration there: clusters 14 us,
// network 5, assembly 1, factorisation 28, backward solve 7).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "gp_cluster.cuh"
#include "gp_front.cuh"
#include "gp_internal.h"
#include "gp_network.cuh"
#include "gp_warp.cuh"

namespace gp {

namespace {

constexpr unsigned FULL = kFullMask;
constexpr int kSmallWarps = 8;
constexpr int kSmallThreads = 32 * kSmallWarps;
constexpr int kSmallGroups = kSmallWarps / kCluWarps;   // cluster tasks at a time

// Barrier of one group of kCluThreads threads.
struct GroupSync {
    int id;
    __device__ __forceinline__ void operator()() const {
        asm volatile("bar.sync %0, %1;" ::"r"(id + 1), "n"(kCluThreads) : "memory");
    }
};

struct SmallLayout {   // offsets in doubles
    int z, zold, yx, clout, svar, x, front, v, vals, total;
};

__host__ __device__ inline SmallLayout small_layout(const DevProblem &P, const DevClu &C, const DevSmall &D) {
    const int net = P.n_diff + P.n_alg;
    auto even = [](int n) { return (n + 1) & ~1; };
    SmallLayout o;
    o.z = 0;
    o.zold = o.z + even(P.n_sys);
    o.yx = o.zold + even(net);
    o.clout = o.yx + even(3 * net);
    o.svar = o.clout + 8 * P.n_cl;
    o.x = o.svar + even(P.n_var);
    o.front = o.x + even(P.n_red);
    o.v = o.front + even(D.front_total);
    o.vals = o.v + kSmallWarps * 2 * kSmallMaxFront;
    o.total = o.vals + (C.n_tasks > 0 ? kSmallGroups * C.max_slots * 32 : 0);
    return o;
}

// The fronts' own entries (constants of S, right-hand sides, then the
// scenario's entries and line trips), by the whole CTA.
__device__ void small_assemble(const DevProblem &P, const DevSmall &D, int m, double *fronts, const double *svar,
                               const double *x) {
    for (int i = threadIdx.x; i < D.front_total; i += kSmallThreads) fronts[i] = D.front_const[i];
    __syncthreads();
    for (int i = threadIdx.x; i < P.n_red; i += kSmallThreads) fronts[D.rhs_pos[i]] = x[i];
    for (int e = threadIdx.x; e < D.n_var_ent; e += kSmallThreads) fronts[D.var_pos[e]] += svar[D.var_idx[e]];
    __syncthreads();
}

// The children's update matrices and vectors of supernode s into its front,
// child by child, then the front's elimination with the right-hand side as
// column mm; one warp, lane i on row i.  A column's chain: the pivot search
// in three integer reductions (25 cycles each) beside the reciprocal of
// every candidate (270), the multiplier, the next column's update (64 each);
// the other columns' updates follow at 64 cycles each.  Rows stay in place,
// pos is the place a row has in the eliminated order (exchanged as the batch
// kernels exchange rows); the rows are put in order at the end.
__device__ void small_factor(const DevSym &S, const DevSmall &D, int s, double *fronts, double *x, int *status) {
    const int lane = threadIdx.x & 31;
    const int4 d = D.desc[s];   // start, pivots, rows, front offset
    const int start = d.x, ns = d.y, mm = d.z, nc = mm + 1;
    double *F = fronts + d.w;
    for (int q = S.child_ptr[s]; q < S.child_ptr[s + 1]; q++) {
        const int c = S.children[q];
        for (int t = D.ea_ptr[c] + lane; t < D.ea_ptr[c + 1]; t += 32) {
            const int2 e = D.ea[t];
            fronts[e.x] += fronts[e.y];
        }
        __syncwarp();
    }
    const bool row = lane < mm;
    int pos = lane;
    double v = row ? F[lane] : 0.0;
    for (int k = 0; k < ns; k++) {
        const bool cand = pos >= k && pos < ns;
        const double own = cand ? v : 1.0;
        const bool special = recip_special(own);
        const double rown = recip_normal(special ? 1.0 : own);
        const unsigned kh = cand ? (unsigned)__double2hiint(v) & 0x7fffffffu : 0u;
        const unsigned mh = __reduce_max_sync(FULL, kh);
        const unsigned kl = cand && kh == mh ? (unsigned)__double2loint(v) : 0u;
        const unsigned ml = __reduce_max_sync(FULL, kl);
        // (the smallest place on ties)
        const unsigned pk = __reduce_min_sync(FULL, cand && kh == mh && kl == ml ? (unsigned)(pos * 32 + lane) : ~0u);
        const int pv = (int)(pk >> 5), pl = (int)(pk & 31u);
        if (lane == 0 && (mh | ml) == 0u) *status |= 4;
        double inv = __shfl_sync(FULL, rown, pl);
        if (__shfl_sync(FULL, (int)special, pl)) inv = 1.0 / __shfl_sync(FULL, own, pl);
        if (lane == pl) pos = k;
        else if (pos == k) pos = pv;
        const bool upd = row && pos > k;
        const double l = v * inv;
        if (upd || lane == pl) F[lane + k * mm] = upd ? l : inv;
        // the next column first, into a register
        {
            const double u = F[pl + (k + 1) * mm];
            v = row ? F[lane + (k + 1) * mm] : 0.0;
            if (upd) {
                v -= l * u;
                F[lane + (k + 1) * mm] = v;
            }
        }
#pragma unroll 4
        for (int j = k + 2; j < nc; j++) {
            const double u = F[pl + j * mm];
            if (upd) F[lane + j * mm] -= l * u;
        }
        __syncwarp();
    }
    if (__any_sync(FULL, pos != lane)) {
        for (int j0 = 0; j0 < nc; j0 += 4) {
            double t[4];
#pragma unroll
            for (int u = 0; u < 4; u++) t[u] = row && j0 + u < nc ? F[lane + (j0 + u) * mm] : 0.0;
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (row && j0 + u < nc) F[pos + (j0 + u) * mm] = t[u];
        }
        __syncwarp();
    }
    if (lane < ns) x[start + lane] = F[mm * mm + lane];
}

__global__ void __launch_bounds__(kSmallThreads) small_newton_kernel(DevProblem P, DevWork W, DevSym S, DevClu Cl,
                                                                     DevSmall D, SmallRun R) {
    extern __shared__ __align__(16) double sm[];
    __shared__ unsigned long long s_nb[kSmallWarps];
    __shared__ int s_status;
    const int m = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (R.masked && !W.active[m]) return;
    const SmallLayout o = small_layout(P, Cl, D);
    const int net = P.n_diff + P.n_alg;
    double *z = sm + o.z, *zold = sm + o.zold, *yx = sm + o.yx, *clout = sm + o.clout, *svar = sm + o.svar,
           *x = sm + o.x, *fronts = sm + o.front, *v = sm + o.v + warp * 2 * kSmallMaxFront;
    const int grp = warp / kCluWarps, gtid = tid % kCluThreads;
    double *vals = sm + o.vals + (size_t)grp * Cl.max_slots * 32;
    const double *u0 = W.u0 + (size_t)m * P.n_ctrl, *p = W.p + (size_t)m * P.n_par;
    double *zg = W.z + (size_t)m * P.n_sys;
    for (int i = tid; i < P.n_sys; i += kSmallThreads) z[i] = zg[i];
    if (tid == 0) s_status = W.status[m];
    if (grp < Cl.n_tasks) load_image(P, Cl, grp, m, R.dt, vals, gtid);
    __syncthreads();
    for (int k = R.k0; k < R.k1; k++) {
        for (int i = tid; i < net; i += kSmallThreads) zold[i] = z[i];
        __syncthreads();
        int it = 0;
        for (;;) {
            // ---- clusters (the first task's image is already on its way) ----
            unsigned long long nb = 0ull;
            const GroupSync sync{grp};
            for (int t = grp; t < Cl.n_tasks; t += kSmallGroups) {
                if (t != grp) load_image(P, Cl, t, m, R.dt, vals, gtid);
                const int cls = Cl.task_class[t];
                double Cc[6] = {0, 0, 0, 0, 0, 0}, Ic[2] = {0, 0};
                cluster_fill(P, Cl, t, m, z, zold, u0, p, R.dt, vals, gtid, s_nb + grp * kCluWarps, Cc, Ic, sync);
                const unsigned long long wn = s_nb[warp];
                nb = wn > nb ? wn : nb;
                cluster_solve<double>(Cl, cls, vals, gtid, sync);
                if (lane < Cl.task_count[t]) {
                    const int c = Cl.order[Cl.task_first[t] + lane];
                    cluster_out<double>(P, Cl, cls, c, vals, gtid, Cc, Ic, yx, clout + (size_t)c * 8);
                }
                sync();
            }
            if (grp < Cl.n_tasks) load_image(P, Cl, grp, m, R.dt, vals, gtid);   // for the next evaluation
            __syncthreads();
            // ---- network rows ----
            for (int i = tid; i < P.n_bus; i += kSmallThreads) {
                const unsigned long long t =
                    network_bus(P, m, P.bus_order[i], z, p, clout, svar, x, nullptr, true);
                nb = t > nb ? t : nb;
            }
            nb = warp_max(nb);
            if (lane == 0) s_nb[warp] = nb;
            __syncthreads();
            nb = s_nb[0];
#pragma unroll
            for (int w = 1; w < kSmallWarps; w++) nb = s_nb[w] > nb ? s_nb[w] : nb;
            const double nrm = __longlong_as_double((long long)nb);
            if (nrm < R.tol) break;
            if (nb >= 0x7ff0000000000000ull || it >= R.itermax) {
                if (tid == 0) s_status |= nb >= 0x7ff0000000000000ull ? 2 : 1;
                break;
            }
            it++;
            // ---- factorisation with the forward solve, backward solve ----
            small_assemble(P, D, m, fronts, svar, x);
            if (S.asmt_ptr) {
                // tripped lines' off-diagonal entries
                for (int s = warp; s < S.nsup; s += kSmallWarps)
                    for (int e = S.asmt_ptr[s] + lane; e < S.asmt_ptr[s + 1]; e += 32)
                        add_trips(P, S, m, e, fronts + D.desc[s].w + S.asmt_pos[e]);
                __syncthreads();
            }
            for (int l = 0; l < D.n_levels; l++) {
                for (int q = D.lev_ptr[l] + warp; q < D.lev_ptr[l + 1]; q += kSmallWarps)
                    small_factor(S, D, D.lev_sup[q], fronts, x, &s_status);
                __syncthreads();
            }
            for (int l = D.n_levels - 1; l >= 0; l--) {
                for (int q = D.lev_ptr[l] + warp; q < D.lev_ptr[l + 1]; q += kSmallWarps) {
                    const int s = D.lev_sup[q];
                    const int4 d = D.desc[s];
                    const int start = d.x, ns = d.y, mm = d.z;
                    const int *rows = S.rows + S.row_ptr[s];
                    if (lane < mm) v[lane] = lane < ns ? x[start + lane] : x[rows[lane - ns]];
                    __syncwarp();
                    const double *F = fronts + d.w;
                    bwd_u12<double>(F, mm, 0, ns, mm, ns, v);
                    bwd_cols_j<double, 1>(F, mm, 0, 0, ns, ns, v);
                    if (lane < ns) x[start + lane] = v[lane];
                    __syncwarp();
                }
                __syncthreads();
            }
            // ---- update ----
            for (int i = tid; i < P.n_sys; i += kSmallThreads) {
                if (i >= net) {
                    z[i] += x[P.iperm[i - net]];
                } else {
                    const int b = D.state_bus[i];
                    if (b >= 0) {
                        const double dvr = x[P.iperm[2 * b]], dvi = x[P.iperm[2 * b + 1]];
                        z[i] -= yx[i] + yx[net + i] * dvr + yx[2 * net + i] * dvi;
                    } else {
                        z[i] += x[P.iperm[D.red_of[i]]];
                    }
                }
            }
            __syncthreads();
        }
        if (tid == 0 && R.iters) R.iters[(size_t)(2 * k + R.slot) * P.M + m] = it;
        if (R.traj) {
            double *t = R.traj + (size_t)m * R.traj_stride + (size_t)(k + 1) * P.n_sys;
            for (int i = tid; i < P.n_sys; i += kSmallThreads) t[i] = z[i];
        }
        __syncthreads();
    }
    cp_async_wait();
    for (int i = tid; i < P.n_sys; i += kSmallThreads) zg[i] = z[i];
    if (tid == 0) W.status[m] = s_status;
}

}  // namespace

int small_shared_bytes(const DevProblem &P, const DevClu &C, const DevSmall &D) {
    return small_layout(P, C, D).total * (int)sizeof(double);
}

int small_configure(int bytes) { return raise_shared_limit(small_newton_kernel, bytes) ? 0 : -1; }

void launch_small(const DevProblem &P, const DevWork &W, const DevSym &S, const DevClu &C, const DevSmall &D,
                  const SmallRun &R, cudaStream_t st) {
    small_newton_kernel<<<P.M, kSmallThreads, D.bytes, st>>>(P, W, S, C, D, R);
}

}  // namespace gp
