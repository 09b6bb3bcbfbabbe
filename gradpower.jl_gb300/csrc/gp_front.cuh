// Parts of one front's work that several kernels share: the tripped lines'
// entries (gp_dag.cu, gp_small.cu) and the backward substitution by a warp
// (gp_solve.cu, gp_small.cu).
#pragma once
#include <cuda_runtime.h>

#include "gp_internal.h"
#include "gp_warp.cuh"

namespace gp {

// Line-trip entry e of scenario m's front into its place *a.  Threads take
// entries in any order and at once, so the entries of one scenario at one
// place (parallel circuits) are all added by the thread of the first
// (asmt_len; 0 at the others).
template <class T>
__device__ __forceinline__ void add_trips(const DevProblem &P, const DevSym &S, int m, int e, T *a) {
    for (int q = e; q < e + S.asmt_len[e]; q++) {
        const int t = S.asmt_tr[q];
        if (P.tr_on[t] && t >= P.tr_ptr[m] && t < P.tr_ptr[m + 1]) *a += (T)S.asmt_val[q];
    }
}

template <class T, int J>
__device__ __forceinline__ T pick(const T (&r)[J], int j) {
    T v = r[0];
#pragma unroll
    for (int q = 1; q < J; q++)
        if (j == q) v = r[q];
    return v;
}

template <class T, int J>
__device__ __forceinline__ void place(T (&r)[J], int j, T v) {
#pragma unroll
    for (int q = 0; q < J; q++)
        if (j == q) r[q] = v;
}

// Columns read per chunk of a sweep.
template <int J>
struct Chunk {
    static constexpr int value = J <= 2 ? 8 : (J <= 4 ? 4 : 2);
};

// ---- backward substitution -----------------------------------------------
// U12 columns c in [c0, c1) (front columns, ns <= c < mm):
// v[i] -= U(i, c) v[c] for i < ns, U(i, c) = F[i + (c - cbase) * ld].
template <class T, int LW = 32>
__device__ __forceinline__ void bwd_u12(const T *__restrict__ F, int ld, int cbase, int c0, int c1, int ns, T *v) {
    warp_row_dots<T, LW>(F + (c0 - cbase) * ld, 1, ld, ns, c1 - c0, [&](int a) { return v[c0 + a]; },
                         [&](int i, T acc) { v[i] -= acc; });
    __syncwarp();
}

// U11 columns k from k1 - 1 down to k0: v[k] *= U(k, k) (the stored
// reciprocal pivot), then v[i] -= U(i, k) v[k] for i < k.
template <class T, int J, int CH = Chunk<J>::value, int LW = 32>
__device__ void bwd_cols_j(const T *__restrict__ F, int ld, int kbase, int k0, int k1, int ns, T *v) {
    const int lane = threadIdx.x & (LW - 1);
    T r[J];
#pragma unroll
    for (int j = 0; j < J; j++) {
        const int i = lane + LW * j;
        r[j] = i < ns ? v[i] : T(0);
    }
    for (int kc = k1 - 1; kc >= k0; kc -= CH) {
        T c[CH][J], d[CH];
#pragma unroll
        for (int kk = 0; kk < CH; kk++) {
            const int k = kc - kk;
            d[kk] = k >= k0 ? F[k + (k - kbase) * ld] : T(0);
#pragma unroll
            for (int j = 0; j < J; j++) {
                const int i = lane + LW * j;
                c[kk][j] = (k >= k0 && i < k) ? F[i + (k - kbase) * ld] : T(0);
            }
        }
#pragma unroll
        for (int kk = 0; kk < CH; kk++) {
            const int k = kc - kk;
            if (k >= k0) {
                const T tk = __shfl_sync(kFullMask, pick(r, k / LW), k % LW, LW) * d[kk];
                if (lane == k % LW) place(r, k / LW, tk);
#pragma unroll
                for (int j = 0; j < J; j++) r[j] -= c[kk][j] * tk;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < J; j++) {
        const int i = lane + LW * j;
        if (i < ns) v[i] = r[j];
    }
    __syncwarp();
}

}  // namespace gp
