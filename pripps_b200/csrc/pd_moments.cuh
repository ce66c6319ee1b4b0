// Moment form of the pair sum (device code shared by the FP32 and FP64 pair
// kernels).
//
// For one pair at distance r <= 2·radius < d, with sin(φ/2) = r/d and z = q·d,
//
//   sinc(q r) = sin(z sin(φ/2)) / (z sin(φ/2)) = Σ_n c_n(z) cos(nφ),
//   c_n(z) = (4 − 2 δ_n0)/z · Σ_{k>=n} J_{2k+1}(z)
//
// (the Jacobi–Anger expansion of sin(z sin θ) divided by sin θ). J_ν(z) falls
// off faster than exponentially beyond ν = z, so n < M ≈ z_max/2 + O(z_max^{1/3})
// terms give the sum on the whole grid, however fine the grid is:
// Σ_pairs sinc(q r) = Σ_n c_n(q d)·m_n, m_n = Σ_pairs cos(nφ). The pair kernels sum
// the M moments of a tile's pairs instead of nq grid points, and
// pd_profiles forms the grid points from them in FP64.
//
// cos(nφ) depends on r² alone (it is a polynomial in it), so a pair costs no
// square root and no sine: with s2 = r²/d² = sin²(φ/2) its short sequences are
// Reinsch differences in α = 4·s2 (full relative accuracy for close pairs).
// Eight moments at a time come from a product: with c = 8j + 3.5 and
// b = t + 0.5, t = 0..3,
//
//   cos((c±b)φ) = cos(cφ)cos(bφ) ∓ sin(cφ)sin(bφ),
//
// the four b of a pair are computed once, and the pair (cos cφ, sin cφ) is turned
// by 8φ from j to j + 1. One packed FFMA2 per (j, t) then accumulates two
// moments: 8 lane operations per 8 moments, plus 4 for the turn, against 3 per
// grid point in the direct form. The sines and cosines are kept divided by
// sin(φ/2) and cos(φ/2) in the long sequence (X, Y) and multiplied by them in
// the short one, which removes both square roots.
#pragma once

#include <cuda_runtime.h>

#include "pd_common.h"

namespace pd {

// Moments that q_max·d = z needs: the tail Σ_{n>=M} |c_n| is below 1e-11 (FP32
// form, whose terms are rounded to 6e-8 each) or 1e-15 (FP64 form).
// ν − z = a·(z/2)^{1/3} is where the Airy tail of J_ν(z) reaches the bound; a and
// the constant were fitted to the exact tails for z from 0.01 to 900.
__device__ __forceinline__ int moments_needed(double z, bool fp64) {
    const double a = fp64 ? 13.0 : 9.7, b = fp64 ? 3.0 : 3.5;
    const double m = 0.5 * (z + a * cbrt(0.5 * z) + b);
    return m < 1e6 ? static_cast<int>(m) + 1 : 1000000;
}

// d = PD_MOM_STRETCH · 2·radius keeps φ away from π (φ <= 152°), where r²
// determines φ poorly, at the price of 3 % more moments.
constexpr double PD_MOM_STRETCH = 1.03;

// A pair's sequences: X = cos(cφ)/cos(φ/2), Y = sin(cφ)/sin(φ/2) at the first c
// of the block; (c8, t1, t2) turn (X, Y) by 8φ: X' = X·c8 − Y·t1,
// Y' = Y·c8 + X·t2; vx[t] = 2cos((t+½)φ)cos(φ/2), vy[t] = −2sin((t+½)φ)sin(φ/2).
// Then X·vx = m_{c+b} + m_{c−b} and Y·vy = m_{c+b} − m_{c−b}.
struct MomPair2 {  // two pairs, one in each half
    float2 X, Y, c8, t1, t2, vx[4], vy[4];
};

__device__ __forceinline__ float2 mom_f2(float a) { return make_float2(a, a); }

// `turns` = 8-fold blocks before this one (moment block × groups per block); a
// later block starts from X, Y turned by 8·turns·φ: the turn by 8φ is doubled
// `dbl` times and applied `rep` times, turns = rep·2^dbl.
__device__ __forceinline__ void mom_seed_x2(float2 r2, float inv_d2, int rep, int dbl,
                                            MomPair2 &P) {
    const float2 one = mom_f2(1.0f), two = mom_f2(2.0f), M1 = mom_f2(-1.0f), M2 = mom_f2(-2.0f);
    const float2 s2 = __fmul2_rn(r2, mom_f2(inv_d2));
    const float2 e = __ffma2_rn(s2, M1, one);   // cos²(φ/2)
    const float2 c1 = __ffma2_rn(s2, M2, one);  // cos φ
    const float2 na = __fmul2_rn(s2, mom_f2(-4.0f));
    const float2 nq = __fmul2_rn(na, e);        // −sin²φ
    // doublings of φ with sin(nφ) = u_n·sin φ
    const float2 c1q = __fmul2_rn(c1, c1);
    const float2 c2 = __fadd2_rn(c1q, nq);
    const float2 c4 = __ffma2_rn(c2, c2, __fmul2_rn(__fmul2_rn(mom_f2(4.0f), nq), c1q));
    const float2 w = __fmul2_rn(c1, c2);        // u_4/4
    const float2 w4 = __fmul2_rn(mom_f2(4.0f), w);
    float2 c8 = __ffma2_rn(c4, c4, __fmul2_rn(__fmul2_rn(nq, w4), w4));
    float2 u8 = __fmul2_rn(__fmul2_rn(two, w4), c4);
    // cos tφ by Reinsch differences d_{t+1} = d_t − α cos tφ
    float2 d = __fmul2_rn(s2, M2);
    const float2 C1 = c1;
    P.vy[0] = d;
    P.vx[0] = __fadd2_rn(one, C1);
    d = __ffma2_rn(na, C1, d);
    const float2 C2 = __fadd2_rn(C1, d);
    P.vy[1] = d;
    P.vx[1] = __fadd2_rn(C1, C2);
    d = __ffma2_rn(na, C2, d);
    const float2 C3 = __fadd2_rn(C2, d);
    P.vy[2] = d;
    P.vx[2] = __fadd2_rn(C2, C3);
    d = __ffma2_rn(na, C3, d);
    const float2 C4 = __fadd2_rn(C3, d);
    P.vy[3] = d;
    P.vx[3] = __fadd2_rn(C3, C4);
    // c = 3.5: cos(3.5φ)/cos(φ/2) and sin(3.5φ)/sin(φ/2)
    const float2 c13 = __fadd2_rn(C1, C3);
    P.X = __ffma2_rn(two, __ffma2_rn(C2, M1, c13), M1);
    P.Y = __ffma2_rn(two, __fadd2_rn(c13, C2), one);
    const float2 ts = __fmul2_rn(two, s2), te = __fmul2_rn(two, e);
    P.c8 = c8;
    P.t1 = __fmul2_rn(ts, u8);
    P.t2 = __fmul2_rn(te, u8);
    if (rep > 0) {
        for (int k = 0; k < dbl; ++k) {
            const float2 uu = __fmul2_rn(u8, u8);
            u8 = __fmul2_rn(__fmul2_rn(two, c8), u8);
            c8 = __ffma2_rn(c8, c8, __fmul2_rn(nq, uu));
        }
        const float2 T1 = __fmul2_rn(ts, u8), T2 = __fmul2_rn(te, u8);
        for (int k = 0; k < rep; ++k) {
            const float2 x = __ffma2_rn(P.X, c8, __fmul2_rn(__fmul2_rn(P.Y, T1), M1));
            P.Y = __ffma2_rn(P.Y, c8, __fmul2_rn(P.X, T2));
            P.X = x;
        }
    }
}

// Moments of the pairs (i, j), j0 <= j < j1, j > i, of one thread's i into
// acc[4·jj + t] = (Σ X·vx, Σ Y·vy), for the first nj groups of eight of the block.
// `at` holds the atoms [jbase, ...) in shared memory.
template <int KM>
__device__ __forceinline__ void moments_range(const float4 *__restrict__ at, int jbase, float4 pi,
                                              int i, bool ivalid, int j0, int j1, float inv_d2,
                                              int nj, int rep, int dbl, float2 (&acc)[KM / 2]) {
    const float2 M1 = mom_f2(-1.0f);
    for (int j = j0; j < j1; j += 2) {
        const bool inb = j + 1 < j1;
        const float4 pa = at[j - jbase], pb = at[(inb ? j + 1 : j) - jbase];
        const float2 dx = __ffma2_rn(make_float2(pa.x, pb.x), M1, mom_f2(pi.x));
        const float2 dy = __ffma2_rn(make_float2(pa.y, pb.y), M1, mom_f2(pi.y));
        const float2 dz = __ffma2_rn(make_float2(pa.z, pb.z), M1, mom_f2(pi.z));
        const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
        MomPair2 P;
        mom_seed_x2(r2, inv_d2, rep, dbl, P);
        const bool va = ivalid && j > i, vb = ivalid && inb && j + 1 > i;
        float2 Ua = make_float2(va ? P.X.x : 0.0f, va ? P.Y.x : 0.0f);
        float2 Ub = make_float2(vb ? P.X.y : 0.0f, vb ? P.Y.y : 0.0f);
        float2 Va[4], Vb[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            Va[t] = make_float2(P.vx[t].x, P.vy[t].x);
            Vb[t] = make_float2(P.vx[t].y, P.vy[t].y);
        }
#pragma unroll
        for (int jj = 0; jj < KM / 8; ++jj) {
            if (jj >= nj) break;
#pragma unroll
            for (int t = 0; t < 4; ++t) acc[4 * jj + t] = __ffma2_rn(Ua, Va[t], acc[4 * jj + t]);
#pragma unroll
            for (int t = 0; t < 4; ++t) acc[4 * jj + t] = __ffma2_rn(Ub, Vb[t], acc[4 * jj + t]);
            if (jj + 1 < KM / 8) {
                const float xa = fmaf(Ua.x, P.c8.x, -(Ua.y * P.t1.x));
                Ua.y = fmaf(Ua.y, P.c8.x, Ua.x * P.t2.x);
                Ua.x = xa;
                const float xb = fmaf(Ub.x, P.c8.y, -(Ub.y * P.t1.y));
                Ub.y = fmaf(Ub.y, P.c8.y, Ub.x * P.t2.y);
                Ub.x = xb;
            }
        }
    }
}

// Weighted mode: the same moments in acc0, and weighted by the j atom's
// hydration weight in acc1 (16 lane operations per eight moments and the turn's 4).
template <int KM>
__device__ __forceinline__ void moments_range_w(const float4 *__restrict__ at, int jbase,
                                                float4 pi, int i, bool ivalid, int j0, int j1,
                                                float inv_d2, int nj, int rep, int dbl,
                                                float2 (&acc0)[KM / 2], float2 (&acc1)[KM / 2]) {
    const float2 M1 = mom_f2(-1.0f);
    for (int j = j0; j < j1; j += 2) {
        const bool inb = j + 1 < j1;
        const float4 pa = at[j - jbase], pb = at[(inb ? j + 1 : j) - jbase];
        const float2 dx = __ffma2_rn(make_float2(pa.x, pb.x), M1, mom_f2(pi.x));
        const float2 dy = __ffma2_rn(make_float2(pa.y, pb.y), M1, mom_f2(pi.y));
        const float2 dz = __ffma2_rn(make_float2(pa.z, pb.z), M1, mom_f2(pi.z));
        const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
        MomPair2 P;
        mom_seed_x2(r2, inv_d2, rep, dbl, P);
        const bool va = ivalid && j > i, vb = ivalid && inb && j + 1 > i;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const bool v = h ? vb : va;
            const float w = h ? pb.w : pa.w;
            float2 U = h ? make_float2(P.X.y, P.Y.y) : make_float2(P.X.x, P.Y.x);
            U = make_float2(v ? U.x : 0.0f, v ? U.y : 0.0f);
            const float c8 = h ? P.c8.y : P.c8.x, t1 = h ? P.t1.y : P.t1.x,
                        t2 = h ? P.t2.y : P.t2.x;
            float2 V[4], WV[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                V[t] = h ? make_float2(P.vx[t].y, P.vy[t].y) : make_float2(P.vx[t].x, P.vy[t].x);
                WV[t] = __fmul2_rn(mom_f2(w), V[t]);
            }
#pragma unroll
            for (int jj = 0; jj < KM / 8; ++jj) {
                if (jj >= nj) break;
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    acc0[4 * jj + t] = __ffma2_rn(U, V[t], acc0[4 * jj + t]);
                    acc1[4 * jj + t] = __ffma2_rn(U, WV[t], acc1[4 * jj + t]);
                }
                const float x = fmaf(U.x, c8, -(U.y * t1));
                U.y = fmaf(U.y, c8, U.x * t2);
                U.x = x;
            }
        }
    }
}

// FP64 form: the same sequences in double, one pair at a time;
// acc[8·jj + 2t + {0, 1}] = Σ X·vx, Σ Y·vy (and weighted by w_j in accw).
template <int KM, bool WEIGHTED>
__device__ __forceinline__ void moments_range_f64(const double4 *__restrict__ at, double4 pi, int i,
                                                  bool ivalid, int j0, int j1, double inv_d2,
                                                  int nj, int rep, int dbl, double (&acc)[KM],
                                                  double (&accw)[WEIGHTED ? KM : 1]) {
    for (int j = j0; j < j1; ++j) {
        const double4 pj = at[j];
        const double dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
        const double s2 = (dx * dx + dy * dy + dz * dz) * inv_d2;
        const double e = 1.0 - s2, na = -4.0 * s2, nq = na * e;
        const double C1 = fma(-2.0, s2, 1.0);
        const double c1q = C1 * C1;
        const double c2 = c1q + nq;
        const double c4 = fma(c2, c2, 4.0 * nq * c1q);
        const double w4 = 4.0 * C1 * c2;
        double c8 = fma(c4, c4, nq * w4 * w4);
        double u8 = 2.0 * w4 * c4;
        double vx[4], vy[4];
        vy[0] = -2.0 * s2;
        vx[0] = 1.0 + C1;
        vy[1] = fma(na, C1, vy[0]);
        const double C2 = C1 + vy[1];
        vx[1] = C1 + C2;
        vy[2] = fma(na, C2, vy[1]);
        const double C3 = C2 + vy[2];
        vx[2] = C2 + C3;
        vy[3] = fma(na, C3, vy[2]);
        vx[3] = C3 + (C3 + vy[3]);
        const bool valid = ivalid && j > i;
        const double c13 = C1 + C3;
        double X = fma(2.0, c13 - C2, -1.0), Y = fma(2.0, c13 + C2, 1.0);
        const double ts = 2.0 * s2, te = 2.0 * e;
        const double t1 = ts * u8, t2 = te * u8, cc = c8;
        if (rep > 0) {
            for (int k = 0; k < dbl; ++k) {
                const double uu = u8 * u8;
                u8 = 2.0 * c8 * u8;
                c8 = fma(c8, c8, nq * uu);
            }
            const double T1 = ts * u8, T2 = te * u8;
            for (int k = 0; k < rep; ++k) {
                const double x = fma(X, c8, -(Y * T1));
                Y = fma(Y, c8, X * T2);
                X = x;
            }
        }
        X = valid ? X : 0.0;
        Y = valid ? Y : 0.0;
#pragma unroll
        for (int jj = 0; jj < KM / 8; ++jj) {
            if (jj >= nj) break;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                if constexpr (WEIGHTED) {
                    const double px = X * vx[t], py = Y * vy[t];
                    acc[8 * jj + 2 * t] += px;
                    acc[8 * jj + 2 * t + 1] += py;
                    accw[8 * jj + 2 * t] = fma(pj.w, px, accw[8 * jj + 2 * t]);
                    accw[8 * jj + 2 * t + 1] = fma(pj.w, py, accw[8 * jj + 2 * t + 1]);
                } else {
                    acc[8 * jj + 2 * t] = fma(X, vx[t], acc[8 * jj + 2 * t]);
                    acc[8 * jj + 2 * t + 1] = fma(Y, vy[t], acc[8 * jj + 2 * t + 1]);
                }
            }
            const double x = fma(X, cc, -(Y * t1));
            Y = fma(Y, cc, X * t2);
            X = x;
        }
    }
}

}  // namespace pd
