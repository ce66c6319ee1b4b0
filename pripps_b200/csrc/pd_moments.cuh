// Moment form of the pair sum (FP32 pair kernels) and the direction form (FP32 and
// FP64).
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
// moments: 8 lane operations per 8 moments, plus 4 for the turn (12 in all), against 3 per
// grid point in the direct form. The sines and cosines are kept divided by
// sin(φ/2) and cos(φ/2) in the long sequence (X, Y) and multiplied by them in
// the short one, which removes both square roots.
//
// The turn has full relative accuracy too: it is the sine, not the cosine, that is
// doubled (sin²2θ = 4 sin²θ cos²θ), and the steps are Reinsch differences in
// 4·sin²4φ = 2 − 2cos 8φ. In a long structure the close pairs have a small 8φ; a
// cosine of it rounded near 1 is a phase error of one sign for all of them
// (cos 8φ by three doublings of cos φ and a plain three-term recurrence: rods of
// 5,000 atoms, q_max·d = 258, and 6,000 atoms, 930: largest relative error of I(q)
// 1.3e-5 and 3.8e-5, root mean square 6e-6 and 1e-5).
//
// Direction form. The sum over all pairs is an average over directions,
//
//   Σ_ij a_i b_j sinc(q r_ij) = <A(q n) B*(q n)>,  A(k) = Σ_i a_i e^{i k·r_i},
//
// and the integrand is a polynomial of degree ~2·q·radius on the sphere up to a tail
// that falls off like J_ν: a Gauss–Legendre × equispaced rule with S ≈
// (2 q_max·radius)²/4·0.7 + … directions on a hemisphere integrates it to the same
// accuracy as above. The phase k·r expands in the same way,
// e^{i q x} = Σ_n i^n (2 − δ_n0) J_n(q r1) T_n(x/r1), |x| <= radius < r1, so that a
// thread sums T_n(x/r1) = cos(nφ), cos φ = x/r1, over the atoms for its
// direction with the same sequences as for the pairs, N·S of them instead of
// N²/2. The amplitudes come out relative to themselves, not to N²: at the
// deep minima of a profile this form is the more accurate one.
#pragma once

#include <cuda_runtime.h>

#include "pd_common.h"

namespace pd {

// First ν beyond which J_ν(z) stays below the bound: ν − z = a·(z/2)^{1/3} + b on
// the Airy tail; a and b were fitted to the exact tails for z from 0.01 to 900.
__device__ __forceinline__ double bessel_order(double z, double a, double b) {
    return z + a * cbrt(0.5 * z) + b;
}

// Moments that q_max·d = z needs: the tail Σ_{n>=M} |c_n| is below 1e-11 (FP32
// form, whose terms are rounded to 6e-8 each) or 1e-15 (FP64 form).
__device__ __forceinline__ int moments_needed(double z, bool fp64) {
    const double m = 0.5 * (fp64 ? bessel_order(z, 13.0, 3.0) : bessel_order(z, 9.7, 3.5));
    return m < 1e6 ? static_cast<int>(m) + 1 : 1000000;
}

// d = PD_MOM_STRETCH · 2·radius keeps φ away from π (φ <= 152°), where r²
// determines φ poorly, at the price of 3 % more moments; likewise r1.
constexpr double PD_MOM_STRETCH = 1.03;

// Direction form: orders kept of the rule and of the expansion; the tails are
// below 1e-9 (FP32 form) and 1e-17 (FP64 form) of one pair's or atom's term.
__device__ __forceinline__ double direction_order(double z, bool fp64) {
    return fp64 ? bessel_order(z, 15.0, 5.0) : bessel_order(z, 8.0, 2.0);
}

// A pair's sequences. U_j = (cos(cφ)/cos(φ/2), sin(cφ)/sin(φ/2)) at c = 8j + 3.5 steps by
// U_{j+1} = U_j + D_j, D_{j+1} = D_j − 4sin²4φ·U_{j+1}.
// V_t = (2cos((t+½)φ)cos(φ/2), −2sin((t+½)φ)sin(φ/2)), so that U.x·V.x = m_{c+b} + m_{c−b},
// U.y·V.y = m_{c+b} − m_{c−b}.
struct MomPair {
    float2 u, d;  // U at the first j of the block, and the step to the next
    float m4;     // −4sin²4φ
    float2 v[4];
};

// X, Y turned by an angle of θ = 2·half: t = sin²(half), T1 = sin θ·tan(φ/2) and
// T2 = sin θ/tan(φ/2): what it adds.
__device__ __forceinline__ float2 mom_turn(float X, float Y, float t, float T1, float T2) {
    const float m = -2.0f * t;
    return make_float2(fmaf(X, m, -(Y * T1)), fmaf(Y, m, X * T2));
}

// Scalar operations throughout: they cost the FP32 pipe the same lane slots as
// packed ones over two pairs would, and write the halves of the packed operands in place
// (packed over two pairs, the transposition was 90 register moves per pair:
// 20,000 atoms, 72 moments: 2.05 ms, FMA pipe 41 % and ALU pipe 48 % busy).
// s2 = sin²(φ/2). U is that of the first c of the block: turned by the angle of `rep`
// blocks, 8·2^dbl·φ each.
__device__ __forceinline__ void mom_seed(float s2, int rep, int dbl, bool valid, MomPair &P) {
    const float e = 1.0f - s2;             // cos²(φ/2)
    const float na = -4.0f * s2;           // −α
    const float d1 = -2.0f * s2;
    const float C1 = 1.0f + d1;            // cos φ
    // sin²(nφ), cos(nφ) and u_n = sin(nφ)/sin φ, n = 1, 2, 4, (8)
    const float t1 = -na * e;
    const float t2 = 4.0f * t1 * (C1 * C1), c2 = fmaf(-2.0f, t1, 1.0f);
    const float t4 = 4.0f * t2 * (c2 * c2), c4 = fmaf(-2.0f, t2, 1.0f);
    const float u8 = 8.0f * (C1 * c2) * c4;
    // cos tφ by Reinsch differences d_{t+1} = d_t − α cos tφ
    const float d2 = fmaf(na, C1, d1), C2 = C1 + d2;
    const float d3 = fmaf(na, C2, d2), C3 = C2 + d3;
    const float d4 = fmaf(na, C3, d3);
    P.v[0] = make_float2(1.0f + C1, d1);
    P.v[1] = make_float2(C1 + C2, d2);
    P.v[2] = make_float2(C2 + C3, d3);
    P.v[3] = make_float2(C3 + (C3 + d4), d4);
    // c = 3.5: cos(3.5φ)/cos(φ/2) and sin(3.5φ)/sin(φ/2), from the differences
    float X = fmaf(2.0f, d1 + d3, 1.0f);
    float Y = fmaf(2.0f, fmaf(3.0f, d1, fmaf(2.0f, d2, d3)), 7.0f);
    const float ts = s2 + s2, te = e + e;
    if (rep > 0) {
        float t = t4, c = c4, u = u8;  // sin²θ, cos θ, sin 2θ/sin φ at θ = 4φ
        for (int k = 0; k < dbl; ++k) {
            const float cn = fmaf(-2.0f, t, 1.0f);
            t = 4.0f * t * (c * c);
            c = cn;
            u = 2.0f * c * u;
        }
        for (int k = 0; k < rep; ++k) {
            const float2 step = mom_turn(X, Y, t, ts * u, te * u);
            X += step.x;
            Y += step.y;
        }
    }
    X = valid ? X : 0.0f;
    Y = valid ? Y : 0.0f;
    P.u = make_float2(X, Y);
    P.d = mom_turn(X, Y, t4, ts * u8, te * u8);
    P.m4 = -4.0f * t4;
}

template <int KM, bool WEIGHTED>
__device__ __forceinline__ void mom_accumulate(const MomPair &P, float w, int nj,
                                               float2 (&acc)[KM / 2],
                                               float2 (&accw)[WEIGHTED ? KM / 2 : 1]) {
    const float2 m4 = make_float2(P.m4, P.m4);
    float2 U = P.u, D = P.d;
    float2 WV[WEIGHTED ? 4 : 1];
    if constexpr (WEIGHTED)
#pragma unroll
        for (int t = 0; t < 4; ++t) WV[t] = __fmul2_rn(make_float2(w, w), P.v[t]);
#pragma unroll
    for (int jj = 0; jj < KM / 8; ++jj) {
        if (jj >= nj) break;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            acc[4 * jj + t] = __ffma2_rn(U, P.v[t], acc[4 * jj + t]);
            if constexpr (WEIGHTED) accw[4 * jj + t] = __ffma2_rn(U, WV[t], accw[4 * jj + t]);
        }
        if (jj + 1 < KM / 8) {
            if (jj > 0) D = __ffma2_rn(m4, U, D);
            U = __fadd2_rn(U, D);
        }
    }
}

// Moments of the pairs (i, j), j0 <= j < j1, j > i, of one thread's i into
// acc[4·jj + t] = (Σ U.x·V.x, Σ U.y·V.y), for the first nj groups of eight of
// the block. `at` holds the atoms [jbase, ...) in shared memory. Weighted mode
// (WEIGHTED): the sums weighted by the j atom's w in accw as well.
template <int KM, bool WEIGHTED>
__device__ __forceinline__ void moments_range(const float4 *__restrict__ at, int jbase, float4 pi,
                                              int i, bool ivalid, int j0, int j1, float inv_d2,
                                              int nj, int rep, int dbl, float2 (&acc)[KM / 2],
                                              float2 (&accw)[WEIGHTED ? KM / 2 : 1]) {
    for (int j = j0; j < j1; ++j) {
        const float4 pj = at[j - jbase];
        const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        MomPair P;
        mom_seed(r2 * inv_d2, rep, dbl, ivalid && j > i, P);
        mom_accumulate<KM, WEIGHTED>(P, pj.w, nj, acc, accw);
    }
}

constexpr int PD_DIR_LANES = PD_THREADS / PD_DIR_DIRS;   // atoms a unit takes at once

// A direction's first block sums products instead of the sequences of the pairs: with
// x = n·r/r1 = cos φ and T_n = cos(nφ), P_{j,t} = Σ T_8j·T_t, t < 8, from two plain
// three-term recurrences. T_8j·T_t = (T_8j+t + T_8j−t)/2, so the moments are sums of
// the P with alternating signs, which the coefficients take on
// (direction_fold): no half-angle seeds, 12 operations in front of the 10 for each
// eight moments instead of 44 (10,000 atoms, 40 moments: 50 -> 37 µs; 100,000 atoms,
// 112 moments: 5.2 -> 4.05 ms). Rounding of x costs 6e-8·r1 of a position, whatever
// the form; only pairs, whose distances may be short, need sin²(φ/2). w multiplies
// the atom's terms.
//
// P_{j,t} steps with j by the three-term recurrence P_{j+1} = 2T_8·P_j − P_{j−1}, kept as
// W_j = s_j·P_j with the signs s = + + − − + + − − …, which turns every step into one
// multiply-add, W_{j+1} = ±2T_8·W_j + W_{j−1} (+ for even j): no negation, no half
// swapped, the older of the two registers overwritten.
struct DirSeed {
    float2 w0, w1;  // W_0, W_1
    float cc;       // 2T_8
    float2 v[4];    // T_0 … T_7
};
__device__ __forceinline__ void dir_seed(float3 dv, float4 p, float w, DirSeed &P) {
    const float x2 = fmaf(dv.x, p.x, fmaf(dv.y, p.y, dv.z * p.z)) * 4.0f;  // 2x (dv is n/(2·r1))
    const float x = 0.5f * x2;
    const float T2 = fmaf(x2, x, -1.0f), T3 = fmaf(x2, T2, -x), T4 = fmaf(x2, T3, -T2);
    const float T5 = fmaf(x2, T4, -T3), T6 = fmaf(x2, T5, -T4), T7 = fmaf(x2, T6, -T5);
    const float T8 = fmaf(x2, T7, -T6);
    P.v[0] = make_float2(1.0f, x);
    P.v[1] = make_float2(T2, T3);
    P.v[2] = make_float2(T4, T5);
    P.v[3] = make_float2(T6, T7);
    const float w1 = w * T8;
    P.w0 = make_float2(w, w);
    P.w1 = make_float2(w1, w1);
    P.cc = T8 + T8;
}

// N atoms' terms at once, all KM sums: with two, their chains overlap.
template <int KM, int N>
__device__ __forceinline__ void dir_accumulate(const DirSeed (&P)[N], float2 (&acc)[KM / 2]) {
    float2 W[N][2];
#pragma unroll
    for (int n = 0; n < N; ++n) {
        W[n][0] = P[n].w0;
        W[n][1] = P[n].w1;
    }
#pragma unroll
    for (int jj = 0; jj < KM / 8; ++jj) {
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
            for (int t = 0; t < 4; ++t)
                acc[4 * jj + t] = __ffma2_rn(W[n][jj & 1], P[n].v[t], acc[4 * jj + t]);
        if (jj + 2 < KM / 8)
#pragma unroll
            for (int n = 0; n < N; ++n) {
                const float c = (jj & 1) ? P[n].cc : -P[n].cc;
                W[n][jj & 1] = __ffma2_rn(make_float2(c, c), W[n][(jj & 1) ^ 1], W[n][jj & 1]);
            }
    }
}

// A thread's atoms j0, j0 + PD_DIR_LANES, … < j1 of a block staged in shared memory,
// for its direction dv = n/(2·r1), weighted by w or not. With room in registers
// (ILP) two atoms at a time: their sequences' dependency chains overlap.
template <int KM, bool ILP>
__device__ __forceinline__ void direction_range(const float4 *__restrict__ at, float3 dv,
                                                bool weighted, int j0, int j1,
                                                float2 (&acc)[KM / 2]) {
    int j = j0;
    if constexpr (ILP)
        for (; j + PD_DIR_LANES < j1; j += 2 * PD_DIR_LANES) {
            const float4 pa = at[j], pb = at[j + PD_DIR_LANES];
            DirSeed S[2];
            dir_seed(dv, pa, weighted ? pa.w : 1.0f, S[0]);
            dir_seed(dv, pb, weighted ? pb.w : 1.0f, S[1]);
            dir_accumulate<KM, 2>(S, acc);
        }
    for (; j < j1; j += PD_DIR_LANES) {
        const float4 pa = at[j];
        DirSeed S[1];
        dir_seed(dv, pa, weighted ? pa.w : 1.0f, S[0]);
        dir_accumulate<KM, 1>(S, acc);
    }
}

// A later block (rep > 0): the pairs' sequences, turned to its first moment.
template <int KM>
__device__ __forceinline__ void direction_range_later(const float4 *__restrict__ at, float3 dv,
                                                      bool weighted, int j0, int j1, int nj,
                                                      int rep, float2 (&acc)[KM / 2]) {
    constexpr int DBL = KM == 128 ? 4 : 3;
    static_assert(KM == (8 << DBL), "blocks of 8·2^DBL moments");
    for (int j = j0; j < j1; j += PD_DIR_LANES) {
        const float4 p = at[j];
        // sin²(φ/2) = (1 − x/r1)/2
        const float s2 = fmaf(-dv.x, p.x, fmaf(-dv.y, p.y, fmaf(-dv.z, p.z, 0.5f)));
        MomPair A;
        mom_seed(s2, rep, DBL, true, A);
        const float w = weighted ? p.w : 1.0f;
        A.u = __fmul2_rn(make_float2(w, w), A.u);
        A.d = __fmul2_rn(make_float2(w, w), A.d);
        float2 none[1];
        mom_accumulate<KM, false>(A, 0.0f, nj, acc, none);
    }
}

// The same sequences in double for one s2 = sin²(φ/2) (a direction's later blocks; pairs
// in FP64 are summed at the grid points: their moments, sums of N² terms that cancel
// in a profile point, cost it up to three digits of its sixteen).
// acc[8·jj + 2t + {0, 1}] = scale·(Σ U.x·V.x, Σ U.y·V.y).
template <int KM>
__device__ __forceinline__ void mom_accumulate_f64(double s2, double scale, int nj, int rep,
                                                   int dbl, double (&acc)[KM]) {
    const double e = 1.0 - s2, na = -4.0 * s2;
    const double C1 = fma(-2.0, s2, 1.0);
    const double t1 = -na * e;
    const double t2 = 4.0 * t1 * (C1 * C1), c2 = fma(-2.0, t1, 1.0);
    const double t4 = 4.0 * t2 * (c2 * c2), c4 = fma(-2.0, t2, 1.0);
    const double u8 = 8.0 * (C1 * c2) * c4;
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
    double X = fma(2.0, vy[0] + vy[2], 1.0);
    double Y = fma(2.0, fma(3.0, vy[0], fma(2.0, vy[1], vy[2])), 7.0);
    const double ts = 2.0 * s2, te = 2.0 * e;
    if (rep > 0) {
        double t = t4, c = c4, u = u8;
        for (int k = 0; k < dbl; ++k) {
            const double cn = fma(-2.0, t, 1.0);
            t = 4.0 * t * (c * c);
            c = cn;
            u = 2.0 * c * u;
        }
        const double m = -2.0 * t, T1 = ts * u, T2 = te * u;
        for (int k = 0; k < rep; ++k) {
            const double x = fma(X, m, -(Y * T1));
            Y += fma(Y, m, X * T2);
            X += x;
        }
    }
    double UX = scale * X, UY = scale * Y;
    double DX = fma(UX, -2.0 * t4, -(UY * (ts * u8))), DY = fma(UY, -2.0 * t4, UX * (te * u8));
    const double m4 = -4.0 * t4;
#pragma unroll
    for (int jj = 0; jj < KM / 8; ++jj) {
        if (jj >= nj) break;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            acc[8 * jj + 2 * t] = fma(UX, vx[t], acc[8 * jj + 2 * t]);
            acc[8 * jj + 2 * t + 1] = fma(UY, vy[t], acc[8 * jj + 2 * t + 1]);
        }
        if (jj + 1 < KM / 8) {
            if (jj > 0) {
                DX = fma(m4, UX, DX);
                DY = fma(m4, UY, DY);
            }
            UX += DX;
            UY += DY;
        }
    }
}

// The first block of a direction in FP64: products of cosines (dir_seed), the same
// layout; two atoms at a time while their sequences fit.
struct DirSeed64 {
    double T[8], u[2], c;
};
__device__ __forceinline__ void dir_seed_f64(double4 dv, double4 p, bool weighted, DirSeed64 &S) {
    const double x2 = 4.0 * fma(dv.x, p.x, fma(dv.y, p.y, dv.z * p.z));
    S.T[0] = 1.0;
    S.T[1] = 0.5 * x2;
#pragma unroll
    for (int t = 2; t < 8; ++t) S.T[t] = fma(x2, S.T[t - 1], -S.T[t - 2]);
    const double T8 = fma(x2, S.T[7], -S.T[6]);
    S.c = T8 + T8;
    S.u[0] = weighted ? p.w : 1.0;
    S.u[1] = S.u[0] * T8;
}
template <int KM>
__device__ __forceinline__ void dir_accumulate_f64(DirSeed64 &S, int jj, double (&acc)[KM]) {
    const double u = S.u[jj & 1];
#pragma unroll
    for (int t = 0; t < 8; ++t) acc[8 * jj + t] = fma(u, S.T[t], acc[8 * jj + t]);
    // signs + + − − as in dir_accumulate
    if (jj + 2 < KM / 8) S.u[jj & 1] = fma((jj & 1) ? S.c : -S.c, S.u[(jj & 1) ^ 1], u);
}
template <int KM, bool ILP>
__device__ __forceinline__ void direction_range_f64(const double4 *__restrict__ at, double4 dv,
                                                    bool weighted, int j0, int j1,
                                                    double (&acc)[KM]) {
    int j = j0;
    if constexpr (ILP)
        for (; j + PD_DIR_LANES < j1; j += 2 * PD_DIR_LANES) {
            DirSeed64 A, C;
            dir_seed_f64(dv, at[j], weighted, A);
            dir_seed_f64(dv, at[j + PD_DIR_LANES], weighted, C);
#pragma unroll
            for (int jj = 0; jj < KM / 8; ++jj) {
                dir_accumulate_f64<KM>(A, jj, acc);
                dir_accumulate_f64<KM>(C, jj, acc);
            }
        }
    for (; j < j1; j += PD_DIR_LANES) {
        DirSeed64 A;
        dir_seed_f64(dv, at[j], weighted, A);
#pragma unroll
        for (int jj = 0; jj < KM / 8; ++jj) dir_accumulate_f64<KM>(A, jj, acc);
    }
}

// A later block (rep > 0): the pairs' sequences, turned to its first moment.
template <int KM>
__device__ __forceinline__ void direction_range_later_f64(const double4 *__restrict__ at,
                                                          double4 dv, bool weighted, int j0,
                                                          int j1, int nj, int rep,
                                                          double (&acc)[KM]) {
    constexpr int DBL = 3;
    static_assert(KM == (8 << DBL), "blocks of 8·2^DBL moments");
    for (int j = j0; j < j1; j += PD_DIR_LANES) {
        const double4 p = at[j];
        const double s2 = fma(-dv.x, p.x, fma(-dv.y, p.y, fma(-dv.z, p.z, 0.5)));
        mom_accumulate_f64<KM>(s2, weighted ? p.w : 1.0, nj, rep, DBL, acc);
    }
}

// Where a unit's sums go: [chunk][v][group][moment][32 directions].
__device__ __forceinline__ int64_t direction_slot(int chunk, int v, int grp, int nv2,
                                                  const PdFrameDev &fr) {
    return ((static_cast<int64_t>(chunk) * nv2 + v) * fr.n_grp + grp) * fr.n_amp * 32;
}

// Stored, or added to what earlier runs left: of the first block x = s_jj·P_{jj,2t}
// and y = s_jj·P_{jj,2t+1} in direction dir;
__device__ __forceinline__ void direction_put(double *__restrict__ out, int jj, int t, int dir,
                                              double x, double y, bool first) {
    double *o = out + static_cast<int64_t>(8 * jj + 2 * t) * 32 + dir;
    const double s = (jj & 2) ? -1.0 : 1.0;
    o[0] = (first ? 0.0 : o[0]) + s * x;
    o[32] = (first ? 0.0 : o[32]) + s * y;
}
// of a later one from moment n0 on, x = Σ U.x·V.x and y of group jj, element t: the
// moments of cos(nφ) are (x ± y)/2.
__device__ __forceinline__ void direction_put_later(double *__restrict__ out, int n0, int jj, int t,
                                                    int dir, double x, double y, bool first) {
    double *hi = out + static_cast<int64_t>(n0 + 8 * jj + 4 + t) * 32 + dir;
    double *lo = out + static_cast<int64_t>(n0 + 8 * jj + 3 - t) * 32 + dir;
    *hi = (first ? 0.0 : *hi) + 0.5 * (x + y);
    *lo = (first ? 0.0 : *lo) + 0.5 * (x - y);
}

}  // namespace pd
