// Device code of the cluster evaluation and of the staged cluster programs,
// shared by the batch kernels (gp_kernels.cu) and the small-system kernel
// (gp_small.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "gp_devices.cuh"
#include "gp_internal.h"
#include "gp_warp.cuh"

namespace gp {

__device__ __forceinline__ unsigned long long norm_bits(double v) {
    // the bit pattern of |v| (non-negative doubles order like their bit
    // patterns); NaN counts as +inf.  Integer operations only: the FP64
    // pipe is the scarce one on this GPU.
    const unsigned long long a = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    return a > 0x7ff0000000000000ull ? 0x7ff0000000000000ull : a;
}

__device__ __forceinline__ DevRef devref(const DTab &T, int k) {
    DevRef d;
    d.dp = T.diff_ptr[k];
    d.ap = T.alg_ptr[k];
    d.cp = T.ctrl_ptr[k];
    d.pp = T.par_ptr[k];
    d.bus = T.bus[k];
    d.link0 = T.link0[k];
    d.link1 = T.link1[k];
    return d;
}

// The warps' shares of a cluster's evaluation: 0 the machine's flux rows, 1
// its network-frame rows (C, I) and the exciter, 2 the governor, 3 the
// stabiliser.  `off` receives the entries of an offline exciter.
template <class Sink, class Off, class KP>
__device__ __forceinline__ void eval_share(const DevProblem &P, int c, int share, const double *z, const double *u0,
                                           const double *p, Sink &sink, Off &off, double Cc[6], double Ic[2],
                                           const KP &kc, bool exc_on) {
    if (share == 0) {
        genrou_flux(devref(P.dev[0], P.cl_gen[c]), z, u0, p, sink, kc);
    } else if (share == 1) {
        const int et = P.cl_exc_type[c], iex = P.cl_exc[c];
        const DevRef dg = devref(P.dev[0], P.cl_gen[c]);
        DevRef dex{};
        if (et == 3 || et == 4) dex = devref(P.dev[et], iex);
        genrou_stator(dg, P.net, z, sink, Cc, Ic);
        if (exc_on) {
            if (et == 3) sexs_eval(dex, P.net, z, p, sink, kc);
            else if (et == 4) esdc1a_eval(dex, P.net, z, p, sink, kc);
        } else {
            if (et == 3) sexs_eval(dex, P.net, z, p, off, kc);
            else if (et == 4) esdc1a_eval(dex, P.net, z, p, off, kc);
        }
    } else if (share == 2) {
        const int gt = P.cl_gov_type[c], igv = P.cl_gov[c];
        if (gt == 1) ieesgo_eval(devref(P.dev[1], igv), z, p, sink, kc);
        else if (gt == 2) tgov1_eval(devref(P.dev[2], igv), z, p, sink, kc);
    } else {
        const int ip = P.cl_pss[c];
        if (ip >= 0) ieeest_eval(devref(P.dev[5], ip), z, p, sink, kc);
    }
}

__device__ __forceinline__ bool exciter_on(const DevProblem &P, int m, int c) {
    return !P.exc_off || !P.exc_off[(size_t)m * P.n_cl + c];
}

// State-dependent entries, the B columns and the backward-Euler residual
// (its norm in nb).  Same scaling as ImageSink.
template <bool ON>
struct LaneSink {
    double *v;
    const short *slot_of;
    const double *z, *zold;
    int ws, lane;
    unsigned diff;
    double dt;
    unsigned long long *nb;
    __device__ __forceinline__ void put(int r, int c, double x) {
        const int lr = r - ws;
        const bool d = diff >> lr & 1;
        double y = ON ? x : 0.0;
        if (d) y = __dmul_rn(y, -dt);
        if (d && r == c) y = __dadd_rn(y, 1.0);
        v[(int)__ldg(slot_of + lr * 32 + (c - ws)) * 32 + lane] = y;
    }
    __device__ __forceinline__ void putc(int, int, double) {}
    __device__ __forceinline__ void putv(int r, int k, double x) {
        const int lr = r - ws;
        double y = ON ? x : 0.0;
        if (diff >> lr & 1) y = __dmul_rn(y, -dt);
        v[(int)__ldg(slot_of + lr * 32 + 29 + k) * 32 + lane] = y;
    }
    __device__ __forceinline__ void putf(int r, double x) {
        const int lr = r - ws;
        double y = ON ? x : 0.0;
        if (diff >> lr & 1) y = z[r] - zold[r] - dt * y;
        v[(int)__ldg(slot_of + lr * 32 + 31) * 32 + lane] = y;
        const unsigned long long t = norm_bits(y);
        *nb = t > *nb ? t : *nb;
    }
};

// A staged stream of record pairs (CluRec) by one of the task's warps: v0 +
// offsets for d and b, va + offsets for a.  The next pair is read ahead;
// sync() is the barrier of the task's warps.
template <class T, class Sync>
__device__ __forceinline__ void run_stages(const int4 *q, int n, T *v0, const T *va, int lane, Sync sync) {
    v0 += lane;
    va += lane;
    int4 r0 = __ldg(q), r1 = __ldg(q + 1);
    for (int i = 0; i < n; i++) {
        const int4 c0 = r0, c1 = r1;
        if (i + 1 < n) {
            r0 = __ldg(q + 2 * i + 2);
            r1 = __ldg(q + 2 * i + 3);
        }
        const int code = c0.w & 255;
        if (code == (REC_FMS | REC_FMS << 4)) {
            const T a0 = va[c0.y], b0 = v0[c0.z], a1 = va[c1.y], b1 = v0[c1.z];
            T d0 = v0[c0.x], d1 = v0[c1.x];
            d0 -= a0 * b0;
            d1 -= a1 * b1;
            v0[c0.x] = d0;
            v0[c1.x] = d1;
        } else if (code == REC_FMS) {
            v0[c0.x] -= va[c0.y] * v0[c0.z];
        } else if (code == REC_MUL) {
            v0[c0.x] *= va[c0.y];
        } else if (code == (REC_MUL | REC_MUL << 4)) {
            const T a0 = va[c0.y], a1 = va[c1.y];
            const T d0 = v0[c0.x], d1 = v0[c1.x];
            v0[c0.x] = d0 * a0;
            v0[c1.x] = d1 * a1;
        } else if (code == REC_RCP) {
            v0[c0.x] = recip(va[c0.y]);
        }
        if (c0.w & REC_SYNC) sync();
    }
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Warp maximum of ordered norm bits.
__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
    const unsigned hi = (unsigned)(v >> 32), lo = (unsigned)v;
    const unsigned mh = __reduce_max_sync(kFullMask, hi);
    const unsigned ml = __reduce_max_sync(kFullMask, hi == mh ? lo : 0u);
    return (unsigned long long)mh << 32 | ml;
}


constexpr int kCluThreads = 32 * kCluWarps;

// The constant slots of a task's image into vals (asynchronous copies).
__device__ __forceinline__ void load_image(const DevProblem &P, const DevClu &Cl, int task, int m, double dt,
                                           double *vals, int tid) {
    const double *img = Cl.img + ((((size_t)(dt == 0.0) * P.M + m) * Cl.n_tasks + task) * Cl.max_img) * 32;
    for (int e = tid; e < Cl.n_img[Cl.task_class[task]] * 16; e += kCluThreads) cp_async16(vals + 2 * e, img + 2 * e);
}

// One warp task of scenario m up to the factorisation, by the kCluThreads
// threads tid of a group (sync: its barrier): the state-dependent slots, the
// B columns and the residual into vals (whose constant slots load_image
// fetched; waited for here), the residual's norm into s_nb[warp].  Cc and Ic
// are warp 1's.  z, zold, u0, p: the scenario's.
template <class Sync>
__device__ __forceinline__ void cluster_fill(const DevProblem &P, const DevClu &Cl, int task, int m, const double *z,
                                             const double *zold, const double *u0, const double *p, double dt,
                                             double *vals, int tid, unsigned long long *s_nb, double Cc[6],
                                             double Ic[2], Sync sync) {
    const int lane = tid & 31, warp = tid >> 5;
    const int cls = Cl.task_class[task];
    const bool act = lane < Cl.task_count[task];
    const int c = Cl.order[Cl.task_first[task] + (act ? lane : 0)];
    const int ws = P.cl_w_start[c], Wn = P.cl_w_size[c];
    const int rb = Cl.rhs_base[cls], n_img = Cl.n_img[cls];
    double *R0 = vals + (size_t)rb * 32, *R2 = R0 + (size_t)2 * Wn * 32;
    for (int e = tid; e < 2 * Wn * 32; e += kCluThreads) R0[e] = 0.0;
    if (!act) {
        // idle lanes factor an identity so that none divides by zero
        const unsigned char *base = Cl.base + (size_t)cls * Cl.base_stride;
        for (int s = n_img + warp; s < rb; s += kCluWarps) vals[s * 32 + lane] = base[s] & 2 ? 1.0 : 0.0;
        for (int j = warp; j < Wn; j += kCluWarps) R2[j * 32 + lane] = 0.0;
    }
    sync();
    unsigned long long nb = 0ull;
    if (act) {
        const short *so = Cl.slot_of + (size_t)cls * 1024;
        const unsigned diff = Cl.diff_mask[cls];
        LaneSink<true> on{vals, so, z, zold, ws, lane, diff, dt, &nb};
        LaneSink<false> off{vals, so, z, zold, ws, lane, diff, dt, &nb};
        const LoadK lk{Cl.kc + (((size_t)m * Cl.n_tasks + task) * kConstSlots) * 32 + lane, 32};
        eval_share(P, c, warp, z, u0, p, on, off, Cc, Ic, lk, exciter_on(P, m, c));
    }
    nb = warp_max(nb);
    if (lane == 0) s_nb[warp] = nb;
    cp_async_wait();
    sync();
}

// The task's scheduled operations on vals (FP64 or FP32 slots).
template <class T, class Sync>
__device__ __forceinline__ void cluster_solve(const DevClu &Cl, int cls, T *vals, int tid, Sync sync) {
    const int w = cls * kCluWarps + (tid >> 5);
    run_stages<T>(reinterpret_cast<const int4 *>(Cl.full) + 2 * (size_t)Cl.full_ptr[w],
                  Cl.full_ptr[w + 1] - Cl.full_ptr[w], vals, vals, tid & 31, sync);
    sync();
}

// The task's results: A^-1 f and A^-1 B into yx ([3][n_da], the lane's
// cluster), and by warp 1 the couplings' products and the injection (o[8]).
template <class T>
__device__ __forceinline__ void cluster_out(const DevProblem &P, const DevClu &Cl, int cls, int c, const T *vals,
                                            int tid, const double Cc[6], const double Ic[2], double *yx_m,
                                            double *o) {
    const int lane = tid & 31, warp = tid >> 5;
    const int ws = P.cl_w_start[c], Wn = P.cl_w_size[c], n_da = P.n_diff + P.n_alg;
    const T *R0 = vals + (size_t)Cl.rhs_base[cls] * 32, *R1 = R0 + (size_t)Wn * 32, *R2 = R1 + (size_t)Wn * 32;
    const int *pc = Cl.perm_col + cls * 32, *p3 = Cl.pos3 + cls * 3;
    double *yx = yx_m + ws;
    for (int j = warp; j < Wn; j += kCluWarps) {
        const int st = pc[j];
        yx[st] = (double)R2[j * 32 + lane];
        yx[n_da + st] = (double)R0[j * 32 + lane];
        yx[2 * n_da + st] = (double)R1[j * 32 + lane];
    }
    if (warp != 1) return;
    double X0[3], X1[3], X2[3];
#pragma unroll
    for (int t = 0; t < 3; t++) {
        X0[t] = (double)R2[p3[t] * 32 + lane];
        X1[t] = (double)R0[p3[t] * 32 + lane];
        X2[t] = (double)R1[p3[t] * 32 + lane];
    }
    o[0] = Cc[0] * X1[0] + Cc[1] * X1[1] + Cc[2] * X1[2];
    o[1] = Cc[0] * X2[0] + Cc[1] * X2[1] + Cc[2] * X2[2];
    o[2] = Cc[3] * X1[0] + Cc[4] * X1[1] + Cc[5] * X1[2];
    o[3] = Cc[3] * X2[0] + Cc[4] * X2[1] + Cc[5] * X2[2];
    o[4] = Cc[0] * X0[0] + Cc[1] * X0[1] + Cc[2] * X0[2];
    o[5] = Cc[3] * X0[0] + Cc[4] * X0[1] + Cc[5] * X0[2];
    o[6] = Ic[0];
    o[7] = Ic[1];
}

}  // namespace gp
