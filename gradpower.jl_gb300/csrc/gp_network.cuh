// Residual and reduced-system entries of one bus, shared by the batch kernels
// (gp_kernels.cu) and the small-system kernel (gp_small.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "gp_cluster.cuh"
#include "gp_internal.h"

namespace gp {

// Bus b of scenario m: its rows of the residual (norm returned, rows to f if
// set), of the reduced right-hand side xp (permuted) and, with need_s, the
// entries of S it owns (svar).  With the mixed solver, a scenario iterating
// on kept factors needs only the residual and the right-hand side.  z, p,
// clout, svar, xp, f: the scenario's.
__device__ __forceinline__ unsigned long long network_bus(const DevProblem &P, int m, int b, const double *z,
                                                          const double *p, const double *clout, double *svar,
                                                          double *xp, double *f, bool need_s) {
    unsigned long long nb = 0ull;
    const int net = P.net;
    const double vr = z[net + 2 * b], vi = z[net + 2 * b + 1];
    double fr = 0.0, fi = 0.0, d00 = 0.0, d01 = 0.0, d10 = 0.0, d11 = 0.0, rr = 0.0, ri = 0.0;
    for (int q = P.y_rowptr[b]; q < P.y_rowptr[b + 1]; q++) {
        const int j = P.y_colidx[q];
        const double2 y = P.y_val[q];   // one 16-byte load
        const double g = y.x, bb = y.y;
        const double vrj = z[net + 2 * j], vij = z[net + 2 * j + 1];
        // -(g + j bb)(vrj + j vij), two FMAs per part
        fr = fma(-g, vrj, fma(bb, vij, fr));
        fi = fma(-bb, vrj, fma(-g, vij, fi));
        if (need_s && j == b) { d00 -= g; d01 += bb; d10 -= bb; d11 -= g; }
    }
    for (int q = P.bus_cl_ptr[b]; q < P.bus_cl_ptr[b + 1]; q++) {
        const double *o = clout + (size_t)P.bus_cl[q] * 8;
        if (need_s) { d00 -= o[0]; d01 -= o[1]; d10 -= o[2]; d11 -= o[3]; }
        rr += o[4]; ri += o[5];
        fr += o[6]; fi += o[7];
    }
    const DTab &ZL = P.dev[6];
    for (int q = P.bus_zl_ptr[b]; q < P.bus_zl_ptr[b + 1]; q++) {
        const int k = P.bus_zl[q];
        if (P.zl_off && P.zl_off[(size_t)m * ZL.n + k]) continue;
        // the load's parameter products ((1 - al) P, (1 - al) Q, al y0),
        // from the table zip_const_kernel fills once per call
        const double *kz = P.zl_k + ((size_t)m * ZL.n + k) * 4;
        const double A1 = kz[0], A2 = kz[1], B1 = kz[2], B2 = kz[3];
        const double vm2 = vr * vr + vi * vi, vm2_tld = 0.2;
        const bool above = vm2 > vm2_tld;
        // one division per load (FP64 division is dear here)
        const double inv = 1.0 / (above ? vm2 : vm2_tld);
        // the constant-impedance part al*y0 and the constant-power part
        // (1 - al)(P - jQ)/max(|V|^2, 0.2) multiply the same V: one
        // complex admittance a + jc; f -= (a + jc) V in FMA form
        const double a = fma(inv, A1, B1), c = fma(inv, A2, B2);
        fr = fma(vi, c, fma(-vr, a, fr));
        fi = fma(-vi, a, fma(-vr, c, fi));
        if (!need_s) continue;
        double p11, p12, p21, p22;
        if (above) {
            const double iv4 = inv * inv;
            p11 = ((A1 * vr - A2 * vi) * 2.0 * vr - A1 * vm2) * iv4;
            p12 = ((A1 * vr - A2 * vi) * 2.0 * vi + A2 * vm2) * iv4;
            p21 = ((A2 * vr + A1 * vi) * 2.0 * vr - A2 * vm2) * iv4;
            p22 = ((A2 * vr + A1 * vi) * 2.0 * vi - A1 * vm2) * iv4;
        } else {
            p11 = -A1 * inv;
            p12 = A2 * inv;
            p21 = -A2 * inv;
            p22 = -A1 * inv;
        }
        d00 += -B1 + p11;
        d01 += B2 + p12;
        d10 += -B2 + p21;
        d11 += -B1 + p22;
    }
    const DTab &SG = P.dev[7];
    for (int q = P.bus_sg_ptr[b]; q < P.bus_sg_ptr[b + 1]; q++) {
        const int k = P.bus_sg[q];
        if (P.sg_off && P.sg_off[(size_t)m * SG.n + k]) continue;   // constant-power ones only
        const int pp = SG.par_ptr[k], ap = SG.alg_ptr[k], bt = SG.link0[k];
        const double vm2r = vr * vr + vi * vi, vm2 = vm2r > 0.2 ? vm2r : 0.2;
        double Pg, Qg;
        if (bt == 2) { Pg = p[pp]; Qg = z[ap]; }
        else if (bt == 3) { Pg = z[ap]; Qg = z[ap + 1]; }
        else { Pg = p[pp]; Qg = p[pp + 1]; }
        const double irn = Pg * vr + Qg * vi, iin = Pg * vi - Qg * vr;
        const double inv = 1.0 / vm2;
        fr += irn * inv;
        fi += iin * inv;
        if (!need_s) {
            const int r0 = P.sg_red[k];
            if (bt == 2) {
                const double vset = p[pp + 2];
                const double fa = vr * vr + vi * vi - vset * vset;
                xp[P.iperm[r0]] = -fa;
                if (f) f[ap] = fa;
                const unsigned long long t = norm_bits(fa);
                nb = t > nb ? t : nb;
            } else if (bt == 3) {
                const double vset = p[pp + 2], aset = p[pp + 3];
                const double fa0 = vr - vset * cos(aset), fa1 = vi - vset * sin(aset);
                xp[P.iperm[r0]] = -fa0;
                xp[P.iperm[r0 + 1]] = -fa1;
                if (f) {
                    f[ap] = fa0;
                    f[ap + 1] = fa1;
                }
                unsigned long long t = norm_bits(fa0);
                nb = t > nb ? t : nb;
                t = norm_bits(fa1);
                nb = t > nb ? t : nb;
            }
            continue;
        }
        if (vm2r > 0.2) {
            const double iv4 = inv * inv;
            d00 += Pg * inv - 2.0 * vr * irn * iv4;
            d01 += Qg * inv - 2.0 * vi * irn * iv4;
            d10 += -Qg * inv - 2.0 * vr * iin * iv4;
            d11 += Pg * inv - 2.0 * vi * iin * iv4;
        } else {
            d00 += Pg * inv;
            d01 += Qg * inv;
            d10 += -Qg * inv;
            d11 += Pg * inv;
        }
        double *sv = svar + P.sg_var[k];
        const int r0 = P.sg_red[k];
        if (bt == 2) {
            const double vset = p[pp + 2];
            const double fa = vr * vr + vi * vi - vset * vset;
            // (ap,vr) (ap,vi) (vr,ap) (vi,ap)
            sv[0] = 2.0 * vr; sv[1] = 2.0 * vi; sv[2] = vi * inv; sv[3] = -vr * inv;
            xp[P.iperm[r0]] = -fa;
            if (f) f[ap] = fa;
            const unsigned long long t = norm_bits(fa);
            nb = t > nb ? t : nb;
        } else if (bt == 3) {
            const double vset = p[pp + 2], aset = p[pp + 3];
            const double fa0 = vr - vset * cos(aset), fa1 = vi - vset * sin(aset);
            // (ap,vr) (ap+1,vi) (vr,ap) (vi,ap) (vr,ap+1) (vi,ap+1)
            sv[0] = 1.0; sv[1] = 1.0; sv[2] = vr * inv; sv[3] = vi * inv; sv[4] = vi * inv; sv[5] = -vr * inv;
            xp[P.iperm[r0]] = -fa0;
            xp[P.iperm[r0 + 1]] = -fa1;
            if (f) {
                f[ap] = fa0;
                f[ap + 1] = fa1;
            }
            unsigned long long t = norm_bits(fa0);
            nb = t > nb ? t : nb;
            t = norm_bits(fa1);
            nb = t > nb ? t : nb;
        }
    }
    // tripped lines: their Ybus terms removed (f = -Y V gains
    // +y_line V; the S diagonal block gains the realified y_line)
    for (int e = P.tr_ptr[m]; e < P.tr_ptr[m + 1]; e++) {
        if (!P.tr_on[e]) continue;
        const int fb = P.tr_from[e], tb = P.tr_to[e];
        if (fb != b && tb != b) continue;
        const double *y = P.tr_y + 8 * (size_t)e + (fb == b ? 0 : 4);   // (yff, yft) or (ytf, ytt)
        const double ybr = fb == b ? y[0] : y[2], ybi = fb == b ? y[1] : y[3];
        const double yor = fb == b ? y[2] : y[0], yoi = fb == b ? y[3] : y[1];
        const int o = fb == b ? tb : fb;
        const double vro = z[net + 2 * o], vio = z[net + 2 * o + 1];
        fr += ybr * vr - ybi * vi + yor * vro - yoi * vio;
        fi += ybi * vr + ybr * vi + yoi * vro + yor * vio;
        if (need_s) { d00 += ybr; d01 -= ybi; d10 += ybi; d11 += ybr; }
    }
    for (int e = P.fl_ptr[m]; e < P.fl_ptr[m + 1]; e++) {
        if (P.fl_on[e] && P.fl_bus[e] == b) {
            const double yf = P.fl_yf[e];
            fr -= yf * vr;
            fi -= yf * vi;
            d00 -= yf;
            d11 -= yf;
        }
    }
    if (f) {
        f[net + 2 * b] = fr;
        f[net + 2 * b + 1] = fi;
    }
    if (need_s) {
        double *sv = svar + 4 * b;
        sv[0] = d00; sv[1] = d01; sv[2] = d10; sv[3] = d11;
    }
    xp[P.iperm[2 * b]] = -(fr - rr);
    xp[P.iperm[2 * b + 1]] = -(fi - ri);
    unsigned long long t = norm_bits(fr);
    nb = t > nb ? t : nb;
    t = norm_bits(fi);
    nb = t > nb ? t : nb;
    return nb;
}

}  // namespace gp
