// Device kernels of the batched backward-Euler Newton step.
//
//  cluster_kernel  one lane per (generator cluster, scenario): evaluates
//                  the cluster's residual rows and Jacobian block
//                  [A_k | B_k] (src/kernels/{genrou,ieesgo,tgov1,sexs,
//                  esdc1a,ieeest}.jl), applies the backward-Euler scaling
//                  (src/dynamics.jl:366-391, 481-500), factors A_k by its
//                  class's static-pivot sparse program and returns A_k^-1 f_k, A_k^-1 B_k and the Schur terms
//                  C_k A_k^-1 B_k, C_k A_k^-1 f_k (src/schur.jl:195-247,
//                  324-346) — the reference's gather + cuBLAS getrf/getrs
//                  sequence (ext/GradPowerCUDAExt/GradPowerCUDAExt.jl:1825-1887,
//                  2750-2779) fused into one pass.
//  network_kernel  one thread per (bus, scenario): complex Ybus row times
//                  V fused with machine injections, ZIP loads
//                  (src/kernels/zipload.jl), static generators
//                  (src/kernels/static_gen.jl) and fault shunts
//                  (src/dynamics.jl:314-327); writes the bus's 2x2 diagonal
//                  block of the reduced matrix S and its right-hand side.
//  update_kernel   z += dz: network and static-generator unknowns from the
//                  solve, cluster states by back-substitution
//                  dw_k = -(A_k^-1 f_k + A_k^-1 B_k dv) (src/schur.jl:383-409).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "gp_cluster.cuh"
#include "gp_devices.cuh"
#include "gp_internal.h"
#include "gp_network.cuh"
#include "gp_warp.cuh"

namespace gp {

#define FULL_MASK 0xffffffffu

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------

// ---------------------------------------------------------------------------
// cluster kernels: one lane per (cluster, scenario), 32 clusters of one
// pattern class per warp task, a task run by the kCluWarps warps of a CTA.
//
// What bounds them.  GB300's FP64 pipe takes 64 cycles of an SM
// sub-partition per warp instruction (19 per SM with all four busy, both
// whatever the active lanes), so a task on one warp is a serial chain of its
// FP64 instructions at 64 cycles each plus the shared-memory round trips
// between them, and the FP64 instruction count is what the throughput limit
// is made of.  Hence
//  - the entries of a cluster block that depend on the parameters and the
//    time step alone, and the part of the factorisation that only touches
//    them, are computed once per integration (cluster_image_kernel; the
//    reciprocals of parameters likewise, DevClu::kc);
//  - the devices of a cluster are evaluated by different warps, and the
//    rest of the factorisation and the three solves is scheduled on the host
//    over the four warps in stages (gp_cluster_plan.cpp), so that a task
//    uses all four sub-partitions;
//  - structurally zero operations on the two B columns are left out.
// Every slot receives the operations it always did, in the same order.
// Measured, one FP64 evaluation, one warp a task and the whole program each
// time -> this: one cluster (2 buses) 60 -> 23 us, 25,600 clusters (2,000
// buses x 64) 180 -> 73 us, 40,000 (70,000 buses x 8) 203 -> 88 us; the
// mixed solver's (mostly kept factors) 70,000 x 8 85 -> 58 us.
// ---------------------------------------------------------------------------

// Image of the constant entries: the slot keeps the entry with the
// backward-Euler scaling (rows of the class's differential mask) and the
// diagonal's one.  ON false: an offline exciter, whose rows hold (the
// entries are zero, the diagonal one).
template <bool ON>
struct ImageSink {
    double *v;             // vals[slot * 32 + lane]
    const short *slot_of;  // class map, local (r, c) -> slot
    int ws, lane;
    unsigned diff;
    double dt;
    __device__ __forceinline__ void put(int, int, double) {}
    __device__ __forceinline__ void putc(int r, int c, double x) {
        const int lr = r - ws;
        const bool d = diff >> lr & 1;
        double y = ON ? x : 0.0;
        if (d) y = __dmul_rn(y, -dt);
        if (d && r == c) y = __dadd_rn(y, 1.0);
        v[(int)slot_of[lr * 32 + (c - ws)] * 32 + lane] = y;
    }
    __device__ __forceinline__ void putv(int, int, double) {}
    __device__ __forceinline__ void putf(int, double) {}
};

// Once per integration, one warp per (task, scenario): the parameter
// constants (DevClu::kc) and, for the call's time step (which = 0) and the
// dt = 0 re-solves (which = 1), the constant slots with their part of the
// factorisation done.  Rerun after a disconnection.
__global__ void __launch_bounds__(32) cluster_image_kernel(DevProblem P, DevWork W, DevClu Cl, double dt, int which) {
    extern __shared__ double vals[];
    const int task = blockIdx.x, m = blockIdx.y, lane = threadIdx.x;
    const int cls = Cl.task_class[task];
    const bool act = lane < Cl.task_count[task];
    const int c = Cl.order[Cl.task_first[task] + (act ? lane : 0)];
    const int rb = Cl.rhs_base[cls], n_img = Cl.n_img[cls];
    const unsigned char *base = Cl.base + (size_t)cls * Cl.base_stride;
    // (idle lanes factor an identity, so that none divides by zero)
    for (int s = 0; s < rb; s++) vals[s * 32 + lane] = base[s] & (act ? 1 : 2) ? 1.0 : 0.0;
    if (act) {
        const short *so = Cl.slot_of + (size_t)cls * 1024;
        const int ws = P.cl_w_start[c];
        const unsigned diff = Cl.diff_mask[cls];
        ImageSink<true> on{vals, so, ws, lane, diff, dt};
        ImageSink<false> off{vals, so, ws, lane, diff, dt};
        const double *z = W.z + (size_t)m * P.n_sys, *u0 = W.u0 + (size_t)m * P.n_ctrl,
                     *p = W.p + (size_t)m * P.n_par;
        double Cc[6], Ic[2];
        const bool exc = exciter_on(P, m, c);
        const RecordK rk{Cl.kc + (((size_t)m * Cl.n_tasks + task) * kConstSlots) * 32 + lane, 32};
        for (int s = 0; s < kCluWarps; s++) eval_share(P, c, s, z, u0, p, on, off, Cc, Ic, rk, exc);
    }
    for (int q = Cl.const_ptr[cls]; q < Cl.const_ptr[cls + 1]; q++) {
        const CluOp o = Cl.const_ops[q];
        double *d = vals + o.d * 32 + lane;
        if (o.code == OP_RCP) *d = recip(vals[o.a * 32 + lane]);
        else if (o.code == OP_MUL) *d *= vals[o.a * 32 + lane];
        else *d -= vals[o.a * 32 + lane] * vals[o.b * 32 + lane];
    }
    double *img = Cl.img + ((((size_t)which * P.M + m) * Cl.n_tasks + task) * Cl.max_img) * 32 + lane;
    for (int s = 0; s < n_img; s++) img[(size_t)s * 32] = vals[s * 32 + lane];
}

// Modes per scenario: 0 exact Newton (Jacobian block, FP64 LU, three solves;
// also the mixed solver's MX_EXACT); 1 the same, and the LU values and
// coupling rows are kept in FP32 for the following iterations (MX_FP32).
// The mixed solver's MX_KEEP scenarios (residual only, solved with the kept
// FP32 LU) run cluster_keep_kernel instead.
struct CtaSync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};

__global__ void __launch_bounds__(kCluThreads, 4) cluster_kernel(DevProblem P, DevWork W, DevClu Cl, DevMixed Mx) {
    extern __shared__ __align__(16) double vals[];
    __shared__ unsigned long long s_nb[kCluWarps];
    const int task = blockIdx.x, m = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (!W.active[m]) return;
    const int r = Mx.on ? Mx.refac[m] : MX_EXACT;
    if (r == MX_KEEP) return;
    const int mode = r == MX_FP32 ? 1 : 0;
    const int cls = Cl.task_class[task];
    const bool act = lane < Cl.task_count[task];
    const int c = Cl.order[Cl.task_first[task] + (act ? lane : 0)];
    const int rb = Cl.rhs_base[cls];
    const double dt = *W.dt;
    // the constant slots arrive while the devices are evaluated
    load_image(P, Cl, task, m, dt, vals, tid);
    double Cc[6] = {0, 0, 0, 0, 0, 0}, Ic[2] = {0, 0};   // warp 1
    cluster_fill(P, Cl, task, m, W.z + (size_t)m * P.n_sys, W.zold + (size_t)m * P.n_sys,
                 W.u0 + (size_t)m * P.n_ctrl, W.p + (size_t)m * P.n_par, dt, vals, tid, s_nb, Cc, Ic, CtaSync());
    if (tid == 0) {
        unsigned long long nb = s_nb[0];
#pragma unroll
        for (int w = 1; w < kCluWarps; w++) nb = s_nb[w] > nb ? s_nb[w] : nb;
        atomicMax(W.norm + m, nb);
    }
    double *yx = W.yx + (size_t)m * 3 * (P.n_diff + P.n_alg), *o = W.clout + ((size_t)m * P.n_cl + c) * 8;
    if (mode == 1) {
        // MX_FP32: the factors are kept in FP32, so the factorisation and
        // the three solves run in FP32 too.  The slots are converted in
        // place, eight a warp at a time: float slot s lies in the first half
        // of double slot s / 2, which an earlier round or this one has read
        float *fv = reinterpret_cast<float *>(vals);
        const int nslot = rb + 3 * P.cl_w_size[c];
        for (int s0 = 0; s0 < nslot; s0 += 8 * kCluWarps) {
            float x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int s = s0 + u * kCluWarps + warp;
                x[u] = s < nslot ? (float)vals[s * 32 + lane] : 0.0f;
            }
            __syncthreads();
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int s = s0 + u * kCluWarps + warp;
                if (s < nslot) fv[s * 32 + lane] = x[u];
            }
            __syncthreads();
        }
        cluster_solve<float>(Cl, cls, fv, tid, CtaSync());
        float *keep = Mx.lu + (((size_t)m * Cl.n_tasks + task) * Mx.n_lu) * 32 + lane;
        for (int s = warp; s < rb; s += kCluWarps) keep[(size_t)s * 32] = fv[s * 32 + lane];
        if (!act) return;
        cluster_out<float>(P, Cl, cls, c, fv, tid, Cc, Ic, yx, o);
    } else {
        // factorisation and solves in FP64
        cluster_solve<double>(Cl, cls, vals, tid, CtaSync());
        if (Cl.save_lu) {
            double *sv = Cl.save_lu + (((size_t)m * Cl.n_tasks + task) * Cl.n_save) * 32 + lane;
            for (int s = warp; s < rb; s += kCluWarps) sv[(size_t)s * 32] = vals[s * 32 + lane];
        }
        if (!act) return;
        cluster_out<double>(P, Cl, cls, c, vals, tid, Cc, Ic, yx, o);
    }
    if (warp != 1) return;
    if (mode == 1) {
        float *cc = Mx.cc + ((size_t)m * P.n_cl + c) * 6;
        for (int t = 0; t < 6; t++) cc[t] = (float)Cc[t];
    }
    if (Cl.save_cc) {
        double *cc = Cl.save_cc + ((size_t)m * P.n_cl + c) * 6;
        for (int t = 0; t < 6; t++) cc[t] = Cc[t];
    }
}

// Residual-only evaluations: Jacobian entries are dropped (the compiler
// removes their arithmetic); the backward-Euler residual goes to its
// position in the solve's column (FP32), its norm to nb, and to f if set.
template <bool ON>
struct KeepSink {
    float *v;              // null: no column
    const short *slot_of;
    const double *z, *zold;
    double *f;
    int ws, lane, base;
    unsigned diff;
    double dt;
    unsigned long long *nb;
    __device__ __forceinline__ void put(int, int, double) {}
    __device__ __forceinline__ void putc(int, int, double) {}
    __device__ __forceinline__ void putv(int, int, double) {}
    __device__ __forceinline__ void putf(int r, double x) {
        const int lr = r - ws;
        double y = ON ? x : 0.0;
        if (diff >> lr & 1) y = z[r] - zold[r] - dt * y;
        if (v) v[((int)__ldg(slot_of + lr * 32 + 31) - base) * 32 + lane] = (float)y;
        if (f) f[r] = y;
        const unsigned long long t = norm_bits(y);
        *nb = t > *nb ? t : *nb;
    }
};

// MX_KEEP scenarios of the mixed solver: the FP64 residual and its solve
// with the kept FP32 LU, nothing else: the kept LU values are copied to
// shared memory while the devices are evaluated, and the staged solve of one
// column follows.  The solve runs in FP32, like the kept LU it applies: FP64
// arithmetic and FP32<->FP64 conversions are scarce on this GPU, and the
// correction of an iteration on kept factors is inexact at the FP32 level
// anyway (the residual that drives it stays FP64).
__global__ void __launch_bounds__(kCluThreads, 6) cluster_keep_kernel(DevProblem P, DevWork W, DevClu Cl,
                                                                      DevMixed Mx) {
    extern __shared__ __align__(16) double vals[];   // kept LU [rhs_base][32] FP32, then the column [W][32] FP32
    __shared__ unsigned long long s_nb[kCluWarps];
    const int task = blockIdx.x, m = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (!W.active[m] || Mx.refac[m] != MX_KEEP) return;
    const int cls = Cl.task_class[task];
    const int cnt = Cl.task_count[task];
    const bool act = lane < cnt;
    const int c = Cl.order[Cl.task_first[task] + (act ? lane : 0)];
    const int ws = P.cl_w_start[c], Wn = P.cl_w_size[c];
    const int rb = Cl.rhs_base[cls], base = rb + 2 * Wn;
    float *lu = reinterpret_cast<float *>(vals), *Rf = lu + (size_t)rb * 32;
    {
        const float *kl = Mx.lu + (((size_t)m * Cl.n_tasks + task) * Mx.n_lu) * 32;
        for (int e = tid; e < rb * 8; e += kCluThreads) cp_async16(lu + 4 * e, kl + 4 * e);
    }
    const double dt = *W.dt;
    double Cc[6], Ic[2] = {0, 0};
    unsigned long long nb = 0ull;
    if (act) {
        const double *z = W.z + (size_t)m * P.n_sys, *zold = W.zold + (size_t)m * P.n_sys;
        const short *so = Cl.slot_of + (size_t)cls * 1024;
        const unsigned diff = Cl.diff_mask[cls];
        KeepSink<true> on{Rf, so, z, zold, nullptr, ws, lane, base, diff, dt, &nb};
        KeepSink<false> off{Rf, so, z, zold, nullptr, ws, lane, base, diff, dt, &nb};
        const LoadK lk{Cl.kc + (((size_t)m * Cl.n_tasks + task) * kConstSlots) * 32 + lane, 32};
        eval_share(P, c, warp, z, W.u0 + (size_t)m * P.n_ctrl, W.p + (size_t)m * P.n_par, on, off, Cc, Ic, lk,
                   exciter_on(P, m, c));
    } else {
        for (int j = warp; j < Wn; j += kCluWarps) Rf[j * 32 + lane] = 0.0f;
    }
    nb = warp_max(nb);
    if (lane == 0) s_nb[warp] = nb;
    cp_async_wait();
    __syncthreads();
    if (tid == 0) {
#pragma unroll
        for (int w = 1; w < kCluWarps; w++) nb = s_nb[w] > nb ? s_nb[w] : nb;
        atomicMax(W.norm + m, nb);
    }
    run_stages<float>(reinterpret_cast<const int4 *>(Cl.sol) + 2 * (size_t)Cl.sol_ptr[cls * kCluWarps + warp],
                      Cl.sol_ptr[cls * kCluWarps + warp + 1] - Cl.sol_ptr[cls * kCluWarps + warp], Rf, lu, lane, CtaSync());
    __syncthreads();
    if (!act) return;
    const int n_da = P.n_diff + P.n_alg;
    double *yx = W.yx + (size_t)m * 3 * n_da + ws;
    const int *pc = Cl.perm_col + cls * 32, *p3 = Cl.pos3 + cls * 3;
    for (int j = warp; j < Wn; j += kCluWarps) yx[pc[j]] = (double)Rf[j * 32 + lane];
    if (warp != 1) return;
    const float Y0 = Rf[p3[0] * 32 + lane], Y1 = Rf[p3[1] * 32 + lane], Y2 = Rf[p3[2] * 32 + lane];
    const float *cc = Mx.cc + ((size_t)m * P.n_cl + c) * 6;
    double *o = W.clout + ((size_t)m * P.n_cl + c) * 8;
    o[4] = (double)fmaf(cc[2], Y2, fmaf(cc[1], Y1, cc[0] * Y0));
    o[5] = (double)fmaf(cc[5], Y2, fmaf(cc[4], Y1, cc[3] * Y0));
    o[6] = Ic[0];
    o[7] = Ic[1];
}

// Parity probes: the residual rows of the clusters (W.f), their norm and the
// injections, nothing else (no parameter constants or images needed).
__global__ void __launch_bounds__(kCluThreads) cluster_residual_kernel(DevProblem P, DevWork W, DevClu Cl) {
    const int task = blockIdx.x, m = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (!W.active[m]) return;
    const bool act = lane < Cl.task_count[task];
    unsigned long long nb = 0ull;
    if (act) {
        const int cls = Cl.task_class[task], c = Cl.order[Cl.task_first[task] + lane];
        const double *z = W.z + (size_t)m * P.n_sys, *zold = W.zold + (size_t)m * P.n_sys;
        double *f = W.f + (size_t)m * P.n_sys;
        double Cc[6], Ic[2];
        KeepSink<true> on{nullptr, nullptr, z, zold, f, P.cl_w_start[c], lane, 0, Cl.diff_mask[cls], *W.dt, &nb};
        KeepSink<false> off{nullptr, nullptr, z, zold, f, P.cl_w_start[c], lane, 0, Cl.diff_mask[cls], *W.dt, &nb};
        eval_share(P, c, warp, z, W.u0 + (size_t)m * P.n_ctrl, W.p + (size_t)m * P.n_par, on, off, Cc, Ic, ComputeK(),
                   exciter_on(P, m, c));
        if (warp == 1) {
            double *o = W.clout + ((size_t)m * P.n_cl + c) * 8;
            for (int t = 0; t < 6; t++) o[t] = 0.0;
            o[6] = Ic[0];
            o[7] = Ic[1];
        }
    }
    nb = warp_max(nb);
    if (lane == 0) atomicMax(W.norm + m, nb);
}

int launch_cluster(const DevProblem &P, const DevWork &W, const DevClu &C, const DevMixed &Mx, cudaStream_t st) {
    if (C.n_tasks == 0) return 0;
    dim3 grid(C.n_tasks, P.M);
    cluster_kernel<<<grid, kCluThreads, (size_t)C.max_slots * 32 * sizeof(double), st>>>(P, W, C, Mx);
    if (!Mx.on) return 1;
    cluster_keep_kernel<<<grid, kCluThreads, (size_t)(C.max_rb + C.max_w) * 32 * sizeof(float), st>>>(P, W, C, Mx);
    return 2;
}

void launch_cluster_residual(const DevProblem &P, const DevWork &W, const DevClu &C, cudaStream_t st) {
    if (C.n_tasks > 0) cluster_residual_kernel<<<dim3(C.n_tasks, P.M), kCluThreads, 0, st>>>(P, W, C);
}

void launch_cluster_image(const DevProblem &P, const DevWork &W, const DevClu &C, double dt, cudaStream_t st) {
    if (C.n_tasks > 0)
        cluster_image_kernel<<<dim3(C.n_tasks, P.M), 32, (size_t)C.max_rb * 32 * sizeof(double), st>>>(
            P, W, C, dt, dt == 0.0 ? 1 : 0);
}

// Parameter products of every ZIP load per scenario for network_kernel:
// (1 - al) P, (1 - al) Q, al g0, al b0.
__global__ void zip_const_kernel(DevProblem P, DevWork W, double *out) {
    const DTab &ZL = P.dev[6];
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)P.M * ZL.n) return;
    const int m = (int)(t / ZL.n), k = (int)(t % ZL.n);
    const double *p = W.p + (size_t)m * P.n_par + ZL.par_ptr[k];
    const double al = p[2];
    double *o = out + (size_t)t * 4;
    o[0] = (1.0 - al) * p[0];
    o[1] = (1.0 - al) * p[1];
    o[2] = al * p[7];
    o[3] = al * p[8];
}

void launch_zip_const(const DevProblem &P, const DevWork &W, double *out, cudaStream_t st) {
    const long long n = (long long)P.M * P.dev[6].n;
    if (n > 0) zip_const_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(P, W, out);
}

int cluster_smem_optin(int bytes) {
    return raise_shared_limit(cluster_kernel, bytes) && raise_shared_limit(cluster_image_kernel, bytes) &&
                   raise_shared_limit(cluster_keep_kernel, bytes)
               ? bytes
               : -1;
}

// ---------------------------------------------------------------------------
// network kernel
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(64) network_kernel(DevProblem P, DevWork W, DevMixed Mx, int want_f,
                                                      int skip_s) {
    const long long task = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = task < (long long)P.M * P.n_bus;
    const int m = valid ? (int)(task / P.n_bus) : P.M;
    // buses in the order of their work (devices, then Ybus row length), so
    // that the lanes of a warp run the same loop trip counts
    const int b = valid ? P.bus_order[(int)(task % P.n_bus)] : 0;
    const bool act = valid && W.active[m];
    unsigned long long nb = 0ull;
    if (act)
        nb = network_bus(P, m, b, W.z + (size_t)m * P.n_sys, W.p + (size_t)m * P.n_par,
                         W.clout + (size_t)m * P.n_cl * 8, W.svar + (size_t)m * P.n_var,
                         W.xperm + (size_t)m * P.n_red, want_f ? W.f + (size_t)m * P.n_sys : nullptr,
                         !skip_s && !(Mx.on && Mx.refac[m] == MX_KEEP));
    // segmented max over lanes of the same scenario, one atomic per segment
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        unsigned long long o = __shfl_down_sync(FULL_MASK, nb, off);
        int om = __shfl_down_sync(FULL_MASK, m, off);
        if (lane + off < 32 && om == m) nb = o > nb ? o : nb;
    }
    const int mprev = __shfl_up_sync(FULL_MASK, m, 1);
    if (act && (lane == 0 || mprev != m)) atomicMax(W.norm + m, nb);
}

void launch_network(const DevProblem &P, const DevWork &W, const DevMixed &Mx, int want_f, cudaStream_t st,
                    int skip_s) {
    // 64-thread blocks: the buses' work differs (devices, row lengths), and
    // small blocks retire and refill the SMs evenly (network phase 9.45 ->
    // 9.0 ms over 0.3 s of the 70k-bus workload against 256-thread blocks;
    // 128: 9.17, 32: 8.97)
    long long tasks = (long long)P.M * P.n_bus;
    int blocks = (int)((tasks + 63) / 64);
    network_kernel<<<blocks, 64, 0, st>>>(P, W, Mx, want_f, skip_s);
}

// ---------------------------------------------------------------------------
// shared-factor Woodbury path
// ---------------------------------------------------------------------------
// The reduced matrix P (scenario 0 at the call's initial state, no fault) is
// factored once per call and shared by every scenario and iteration.  A
// scenario's fault (bus b, admittance yf) subtracts yf from the two
// diagonal entries of its bus: S_m = P - yf U U^T with U = [e_vr e_vi], and
// by the Woodbury identity S_m^-1 r = x - W H^-1 U^T x, x = P^-1 r,
// W = P^-1 U, H = U^T W - I / yf (integrate_gpu_shared_multi!,
// ext/GradPowerCUDAExt/GradPowerCUDAExt.jl:2441-2489, 2560-2574; every
// scenario of the table has one fault bus and admittance, checked by the
// host).

// The scenario's fault: its first table entry (-1: none); *on when one of
// its windows is on.
__device__ __forceinline__ int wb_fault(const DevProblem &P, int m, bool *on) {
    const int e0 = P.fl_ptr[m], e1 = P.fl_ptr[m + 1];
    bool any = false;
    for (int e = e0; e < e1; e++) any = any || P.fl_on[e];
    *on = any;
    return e0 < e1 ? e0 : -1;
}

__global__ void wb_unit_kernel(DevProblem P, DevWork W, int col) {
    const long long task = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (task >= (long long)P.M * P.n_red) return;
    const int m = (int)(task / P.n_red), i = (int)(task % P.n_red);
    bool on;
    const int e = wb_fault(P, m, &on);
    W.xperm[task] = e >= 0 && i == P.iperm[2 * P.fl_bus[e] + col] ? 1.0 : 0.0;
}

__global__ void wb_setup_kernel(DevProblem P, const double *W1, const double *W2, double *Hinv) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= P.M) return;
    bool on;
    const int e = wb_fault(P, m, &on);
    double *h = Hinv + 4 * (size_t)m;
    if (e < 0) {
        h[0] = h[1] = h[2] = h[3] = 0.0;
        return;
    }
    const size_t o = (size_t)m * P.n_red;
    const int r0 = P.iperm[2 * P.fl_bus[e]], r1 = P.iperm[2 * P.fl_bus[e] + 1];
    const double rf = 1.0 / P.fl_yf[e];
    const double a = W1[o + r0] - rf, b = W2[o + r0], c = W1[o + r1], d = W2[o + r1] - rf;
    const double det = a * d - b * c;
    h[0] = d / det;
    h[1] = -b / det;
    h[2] = -c / det;
    h[3] = a / det;
}

__global__ void wb_dots_kernel(DevProblem P, DevWork W, const double *Hinv, double *sv) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= P.M) return;
    bool on;
    const int e = wb_fault(P, m, &on);
    double s0 = 0.0, s1 = 0.0;
    if (e >= 0 && on && W.active[m]) {
        const double *x = W.xperm + (size_t)m * P.n_red;
        const double t0 = x[P.iperm[2 * P.fl_bus[e]]], t1 = x[P.iperm[2 * P.fl_bus[e] + 1]];
        const double *h = Hinv + 4 * (size_t)m;
        s0 = h[0] * t0 + h[1] * t1;
        s1 = h[2] * t0 + h[3] * t1;
    }
    sv[2 * m] = s0;
    sv[2 * m + 1] = s1;
}

__global__ void wb_apply_kernel(DevProblem P, DevWork W, const double *W1, const double *W2, const double *sv) {
    const long long task = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (task >= (long long)P.M * P.n_red) return;
    const int m = (int)(task / P.n_red);
    const double s0 = sv[2 * m], s1 = sv[2 * m + 1];
    if (s0 != 0.0 || s1 != 0.0) W.xperm[task] -= W1[task] * s0 + W2[task] * s1;
}

void launch_wb_unit(const DevProblem &P, const DevWork &W, int col, cudaStream_t st) {
    const long long tasks = (long long)P.M * P.n_red;
    wb_unit_kernel<<<(unsigned)((tasks + 255) / 256), 256, 0, st>>>(P, W, col);
}

void launch_wb_setup(const DevProblem &P, const double *W1, const double *W2, double *Hinv, cudaStream_t st) {
    wb_setup_kernel<<<(P.M + 127) / 128, 128, 0, st>>>(P, W1, W2, Hinv);
}

void launch_wb_correct(const DevProblem &P, const DevWork &W, const double *W1, const double *W2,
                       const double *Hinv, double *s, cudaStream_t st) {
    wb_dots_kernel<<<(P.M + 127) / 128, 128, 0, st>>>(P, W, Hinv, s);
    const long long tasks = (long long)P.M * P.n_red;
    wb_apply_kernel<<<(unsigned)((tasks + 255) / 256), 256, 0, st>>>(P, W, W1, W2, s);
}

// ---------------------------------------------------------------------------
// convergence bookkeeping
// ---------------------------------------------------------------------------

// Start of a Newton iteration: clears the residual norms and the counters;
// the mixed solver takes the modes decided at the previous check.
__global__ void reset_norm_kernel(DevWork W, DevMixed Mx, int M) {
    int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < M) {
        W.norm[m] = 0ull;
        if (Mx.on) {
            const uint8_t r = Mx.refac_next[m];
            Mx.refac[m] = r;
            Mx.refac_next[m] = MX_KEEP;
            if (r == MX_FP32) Mx.age[m] = 0;
        }
    }
    if (m == 0) {
        W.flag[0] = 0;
        W.flag[1] = 0;
        W.flag[2] = 0;
    }
}

void launch_reset_norm(const DevProblem &P, const DevWork &W, const DevMixed &Mx, cudaStream_t st) {
    reset_norm_kernel<<<(P.M + 255) / 256, 256, 0, st>>>(W, Mx, P.M);
}

// Start of a Newton solve of the mixed solver: scenarios whose factors have
// served max_age solves, or every scenario when `force` (first solve, event
// re-solves and the solve after them), refresh them at the first iteration;
// a retried solve is exact from its first iteration.  Refreshes are taken
// together: a refresh costs one factorisation launch whatever the number of
// scenarios in it, so when one scenario refreshes, every scenario does.
// One CTA, so that the decision can be shared.
__global__ void __launch_bounds__(1024) mixed_start_kernel(DevWork W, DevMixed Mx, int M, int force) {
    bool any = false;
    for (int m = threadIdx.x; m < M; m += blockDim.x) {
        if (!W.active[m]) continue;
        if (Mx.all_exact[m]) Mx.refac_next[m] = MX_EXACT;
        else if (force || Mx.age[m] >= Mx.max_age) {
            Mx.refac_next[m] = MX_FP32;
            any = true;
        }
        Mx.age[m] += 1;
    }
    if (__syncthreads_or(any))
        for (int m = threadIdx.x; m < M; m += blockDim.x)
            if (W.active[m] && Mx.refac_next[m] == MX_KEEP) Mx.refac_next[m] = MX_FP32;
}

void launch_mixed_start(const DevProblem &P, const DevWork &W, const DevMixed &Mx, int force, cudaStream_t st) {
    mixed_start_kernel<<<1, std::min(1024, (P.M + 31) / 32 * 32), 0, st>>>(W, Mx, P.M, force);
}

// Restart of the solves marked for a retry: the state goes back to the
// step's starting point (zold), the scenario iterates again from zero
// updates, exactly.  The retry marks are cleared by the host afterwards.
__global__ void retry_start_kernel(DevProblem P, DevWork W, DevMixed Mx) {
    const long long task = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (task >= (long long)P.M * P.n_sys) return;
    const int m = (int)(task / P.n_sys), i = (int)(task % P.n_sys);
    if (!Mx.retry[m]) return;
    W.z[(size_t)m * P.n_sys + i] = W.zold[(size_t)m * P.n_sys + i];
    if (i == 0) {
        W.active[m] = 1;
        W.iters[m] = 0;
        Mx.all_exact[m] = 1;
    }
}

__global__ void predict_kernel(double *z, const double *zold, double *zprev, double *zprev2, double *zprev3, size_t n,
                               int order) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a = zold[i], b = zprev[i], c = zprev2[i];
    if (order == 1) z[i] = 2.0 * a - b;
    else if (order == 2) z[i] = 3.0 * (a - b) + c;
    else if (order == 3) z[i] = 4.0 * (a + c) - 6.0 * b - zprev3[i];
    zprev3[i] = c;
    zprev2[i] = b;
    zprev[i] = a;
}

void launch_predict(double *z, const double *zold, double *zprev, double *zprev2, double *zprev3, size_t n,
                    int order, cudaStream_t st) {
    predict_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(z, zold, zprev, zprev2, zprev3, n, order);
}

void launch_retry_start(const DevProblem &P, const DevWork &W, const DevMixed &Mx, cudaStream_t st) {
    const long long tasks = (long long)P.M * P.n_sys;
    retry_start_kernel<<<(int)((tasks + 255) / 256), 256, 0, st>>>(P, W, Mx);
}


// Convergence test (infinity norm of the FP64 residual), the itermax and
// non-finite checks, and for the mixed solver the mode of the next
// iteration, from the contraction of the step just taken (prev_mode: the
// factors it used):
//  - a step with kept factors that reduced the residual by less than the
//    factor rho_max refreshes them;
//  - a step with freshly refreshed FP32 factors that did not halve the
//    residual means FP32 factors are too coarse for this scenario now: it
//    takes exact Newton steps (fresh FP64 factors) until the solve ends;
//  - so does every scenario still iterating after exact_after iterations.
// A scenario that went exact refreshes its kept factors at the next solve.
// When one scenario refreshes, every scenario on kept factors does.
// A mixed solve that ends at itermax or on a non-finite residual with
// inexact steps is not reported: it is marked for a retry from the step's
// starting point with exact Newton steps, whose outcome is reported.
__global__ void __launch_bounds__(1024) check_kernel(DevWork W, DevMixed Mx, int M, double tol, int itermax,
                                                    LoopCtl ctl) {
    bool any = false;
    for (int m = threadIdx.x; m < M; m += blockDim.x) {
        if (!W.active[m]) continue;
        const unsigned long long bits = W.norm[m];
        const double nrm = __longlong_as_double((long long)bits);
        const bool can_retry = Mx.on && !Mx.all_exact[m];
        if (nrm < tol) {
            W.active[m] = 0;
        } else if (bits >= 0x7ff0000000000000ull || W.iters[m] >= itermax) {
            W.active[m] = 0;
            if (can_retry) {
                Mx.retry[m] = 1;
                atomicAdd(W.flag + 3, 1);
            } else {
                W.status[m] |= bits >= 0x7ff0000000000000ull ? 2 : 1;
            }
        } else {
            if (Mx.on) {
                const int cur = Mx.refac[m], used = Mx.prev_mode[m];
                const bool stepped = W.iters[m] > 0;
                int next = MX_KEEP;
                if (cur == MX_EXACT || W.iters[m] + 1 >= Mx.exact_after ||
                    (stepped && used == MX_FP32 && nrm > 0.5 * Mx.prev_norm[m]))
                    next = MX_EXACT;
                else if (stepped && used == MX_KEEP && nrm > Mx.rho_max * Mx.prev_norm[m])
                    next = MX_FP32;
                if (next == MX_EXACT) Mx.age[m] = Mx.max_age;
                if (next == MX_FP32) any = true;
                Mx.refac_next[m] = (uint8_t)next;
                Mx.prev_mode[m] = (uint8_t)cur;
                Mx.prev_norm[m] = nrm;
                if (cur == MX_FP32) atomicAdd(W.flag + 1, 1);
                else if (cur == MX_EXACT) atomicAdd(W.flag + 2, 1);
            }
            W.iters[m] += 1;
            atomicAdd(W.flag, 1);
        }
    }
    // refreshes are taken together (see mixed_start_kernel)
    if (Mx.on && __syncthreads_or(any))
        for (int m = threadIdx.x; m < M; m += blockDim.x)
            if (W.active[m] && Mx.refac_next[m] == MX_KEEP) Mx.refac_next[m] = MX_FP32;
    if (!ctl.on) return;
    // device-driven loop: the next solve, if any, and its factorisations
    __syncthreads();
    if (threadIdx.x == 0) {
        const int act = atomicAdd(W.flag, 0), n32 = atomicAdd(W.flag + 1, 0), n64 = atomicAdd(W.flag + 2, 0);
        const int v = ctl.mixed ? (n32 > 0 ? 1 : 0) | (n64 > 0 ? 2 : 0) : 0;
        cudaGraphSetConditional(ctl.loop, act > 0 ? 1u : 0u);
        if (ctl.mixed) cudaGraphSetConditional(ctl.var, (unsigned)v);
        ctl.cnt[0] += 1;
        if (act > 0) {
            ctl.cnt[1] += 1;
            ctl.cnt[2] += n32;
            ctl.cnt[3] += n64;
            ctl.cnt[4 + v] += 1;
        }
    }
}

void launch_check(const DevProblem &P, const DevWork &W, const DevMixed &Mx, double tol, int itermax,
                  const LoopCtl &ctl, cudaStream_t st) {
    check_kernel<<<1, std::min(1024, (P.M + 31) / 32 * 32), 0, st>>>(W, Mx, P.M, tol, itermax, ctl);
}

// ---------------------------------------------------------------------------
// Newton update
// ---------------------------------------------------------------------------

// state_bus[i]: bus of the non-trivial cluster owning cluster state i, or
// -1 when the state is a reduced unknown (static generator); red_of[i] its
// reduced index in that case.
__global__ void update_kernel(DevProblem P, DevWork W, const int *state_bus, const int *red_of) {
    const long long task = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (task >= (long long)P.M * P.n_sys) return;
    const int m = (int)(task / P.n_sys), i = (int)(task % P.n_sys);
    if (!W.active[m]) return;
    double *z = W.z + (size_t)m * P.n_sys;
    const double *x = W.xperm + (size_t)m * P.n_red;
    const int n_da = P.n_diff + P.n_alg;
    if (i >= P.net) {
        z[i] += x[P.iperm[i - P.net]];
    } else {
        const int b = state_bus[i];
        if (b >= 0) {
            const double *yx = W.yx + (size_t)m * 3 * n_da;
            const double dvr = x[P.iperm[2 * b]], dvi = x[P.iperm[2 * b + 1]];
            z[i] -= yx[i] + yx[n_da + i] * dvr + yx[2 * n_da + i] * dvi;
        } else {
            z[i] += x[P.iperm[red_of[i]]];
        }
    }
}

void launch_update(const DevProblem &P, const DevWork &W, const DevSym &S, const int *perm, cudaStream_t st) {
    (void)S;
    // `perm` carries the two state maps back to back: state_bus then red_of
    const int n_da = P.n_diff + P.n_alg;
    long long tasks = (long long)P.M * P.n_sys;
    update_kernel<<<(int)((tasks + 255) / 256), 256, 0, st>>>(P, W, perm, perm + n_da);
}

// ---------------------------------------------------------------------------
// events
// ---------------------------------------------------------------------------

__global__ void events_kernel(const int *on_step, const int *off_step, const int *scen, uint8_t *fl_on,
                              uint8_t *active, int n_fl, int step) {
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n_fl) return;
    // a fault switched on and off at the same step ends off, as the
    // reference applies the schedule entries in order (src/dynamics.jl:604-629)
    bool hit = false;
    if (on_step[e] == step) { fl_on[e] = 1; hit = true; }
    if (off_step[e] == step) { fl_on[e] = 0; hit = true; }
    if (hit) active[scen[e]] = 1;
}

void launch_events(const DevProblem &P, const DevWork &W, const int *fl_on_step, const int *fl_off_step,
                   const int *fl_scen, uint8_t *fl_on, int n_fl, int step, cudaStream_t st) {
    (void)P;
    if (n_fl == 0) return;
    events_kernel<<<(n_fl + 255) / 256, 256, 0, st>>>(fl_on_step, fl_off_step, fl_scen, fl_on, W.active, n_fl, step);
}

__global__ void disconnect_kernel(const int *on_step, const int *scen, const int *idx, uint8_t *flags,
                                  uint8_t *active, int n, int step) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n || on_step[e] != step) return;
    flags[idx[e]] = 1;
    active[scen[e]] = 1;
}

void launch_disconnects(const int *on_step, const int *scen, const int *idx, uint8_t *flags, uint8_t *active,
                        int n, int step, cudaStream_t st) {
    if (n == 0) return;
    disconnect_kernel<<<(n + 255) / 256, 256, 0, st>>>(on_step, scen, idx, flags, active, n, step);
}

}  // namespace gp
