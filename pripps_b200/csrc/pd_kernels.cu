// Device kernels of the Debye backend (sm_100a).
//
// A frame takes one of three forms, by the rule in frame_constants: class
// amplitudes over directions (pd_directions.cu, pd_direction_sums here), moments of
// the pairs (pd_moments.cuh, in the FP32 pair kernels), or, where they cost less and
// for the FP64 form, the grid points one by one:
//
// K1 (pd_pairs_fp32): for each tile (i-block × j-range × q-block) every thread
// owns one i atom and walks the j atoms of the range NP at a time. For a pair
// at distance r it needs sin(q_k r) for the K consecutive grid points
// q_k = q_s + k·Δq of the block. With x = Δq·r reduced as x = mπ + x'
// (|x'| <= π/2) the sequence is s_k = σ^k·u_k, σ = (-1)^m, where
// u_k = sin(θ + k x'), θ = q_s r. u_k follows the three-term recurrence
// u_{k+1} = 2cos(x')·u_k − u_{k−1}, evaluated in Reinsch's difference form
//   d_{k+1} = d_k − α·u_k,  u_{k+1} = u_k + d_{k+1},  α = 4 sin²(x'/2),
// which stays accurate for small x' (Reinsch's modification of the Goertzel
// recurrence; errors grow linearly in k). It is reseeded every K steps from
// sin θ and cos θ evaluated in FP32 with a double-float phase and our own
// fitted polynomials (see sincos_poly). One step plus the accumulation
// acc_k += σ^k u_k / r is FFMA + FADD + FADD, all on the FP32 pipes (the
// weight 1/r scales the pair's initial u and d, and the pairs' terms are
// summed before they reach acc_k; with the general step, σ alternating, the
// accumulation is an FFMA with ±1/r). acc_k sums sin(q_k r)/r over the
// thread's pairs; dividing by q_k in FP64 afterwards gives Σ sinc(q_k r).
// With a hydration weight per atom (weighted mode) a second accumulator sums
// the terms times w_j (one more FFMA). Both modes run the even and odd grid
// points of a pair as the two halves of packed FP32x2 instructions.
// Per-sub-chunk sums stay in FP32 registers; they are warp-reduced into FP64
// partial sums in shared memory, merged per atom class at the end of the
// tile into FP64 slots, and every later sum is FP64.
//
// K2 (pd_pairs_fp64): the same tiling with sin(q_k r) from the FP64 sin() for
// every pair and q, and FP64 accumulation throughout.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cmath>
#include <cstdio>
#include <mutex>
#include <vector>

#include "pd_common.h"
#include "pd_kernels.h"
#include "pd_launch.cuh"
#include "pd_moments.cuh"
#include "pripps_debye.h"

namespace pd {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// Reduce-scatter of 2·NT values per lane (NT packed pairs, NT a multiple of
// 32) over a warp: at each of five levels a lane keeps one half of its
// pairs, sends the other half to its partner lane^o and adds what the
// partner sends for the half it keeps. Afterwards lane l holds the warp sums
// of the values [l·2NT/32, (l+1)·2NT/32) in v[0 .. NT/32). About 2·NT
// shuffles and NT packed additions instead of the 10·NT shuffles and
// additions of one butterfly per value; the order of the additions is fixed,
// so the sums are deterministic.
#ifndef PD_FLUSH_RS
#define PD_FLUSH_RS 1
#endif
template <int NT>
__device__ __forceinline__ void warp_reduce_scatter(float2 (&v)[NT], int lane) {
    static_assert(NT % 32 == 0, "2·NT values must split evenly over 32 lanes in pairs");
#pragma unroll
    for (int lev = 0; lev < 5; ++lev) {
        const int o = 16 >> lev;
        const int h = (NT >> lev) / 2;  // packed pairs kept
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const float2 lo = v[k], hi = v[k + h];
            const float2 keep = up ? hi : lo;
            const float2 send = up ? lo : hi;
            const float2 got = make_float2(__shfl_xor_sync(0xffffffffu, send.x, o),
                                           __shfl_xor_sync(0xffffffffu, send.y, o));
            v[k] = __fadd2_rn(keep, got);
        }
    }
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// sin and cos on |t| <= π/4 (+ a few ulp) as polynomials in t² whose FP32
// coefficients we fitted (least squares on Chebyshev nodes, each coefficient
// rounded to FP32 before the next ones were refitted): |error| < 8e-11 for sin
// and < 1.1e-10 for cos in exact arithmetic, under the FP32 rounding of the
// result and oscillating in sign. Taylor coefficients rounded to FP32 would
// leave a one-signed error of ~1e-9, which a sum over 10^8 pairs turns into a
// bias.
__device__ __forceinline__ void sincos_poly(float t, float &s, float &c) {
    const float t2 = t * t;
    float ps = 2.789128530e-6f;
    ps = fmaf(ps, t2, -1.984876289e-4f);
    ps = fmaf(ps, t2, 8.333369158e-3f);
    ps = fmaf(ps, t2, -1.666666716e-1f);
    s = fmaf(t * t2, ps, t);
    float pc = 2.443297126e-5f;
    pc = fmaf(pc, t2, -1.388731296e-3f);
    pc = fmaf(pc, t2, 4.166664556e-2f);
    pc = fmaf(pc, t2, -0.5f);
    c = fmaf(t2, pc, 1.0f);
}

// Two-part π/2 for the reduction: C1 has 8 significant bits, so n·C1 and
// a_hi − n·C1 are exact for n < 2^15; C2 = fl32(π/2 − C1). The part of π/2
// below C2 (2.6e-12) scales every phase by the same 1 + 1.6e-12: a q-axis
// stretch far below anything the FP64 oracle comparison can see.
constexpr float kPio2C1 = 1.5703125f;
constexpr float kPio2C2 = 4.838267923333e-4f;
constexpr float kRoundMagic = 12582912.0f;  // 1.5·2^23: fma(a, 2/π, magic) rounds to an integer

// Reduction of an angle a = a_hi + a_lo (unevaluated sum, |a| <~ 1e4):
// a = n·π/2 + t with |t| <= π/4 + ε; returns t and the quadrant n mod 4.
//
// Why the low part: a_hi lies on the FP32 grid of its binade and a_hi − n·C1
// is exact, so rounding a_hi − n·π/2 to FP32 in one step would give the same
// rounding error to every pair of a quadrant and binade — a bias of ~2e-9 per
// sin that survives a sum over 10^7..10^10 pairs. a_lo carries the pair's own
// rounding residue of q·r, so the final rounding of t falls at a pair-
// specific place between grid points and averages out.
__device__ __forceinline__ float reduce_pio2(float a_hi, float a_lo, int &quadrant) {
    const float nm = fmaf(a_hi, 0.636619772f, kRoundMagic);
    const float n = nm - kRoundMagic;  // exact
    quadrant = __float_as_int(nm) & 3;  // the low mantissa bits hold n
    const float t1 = fmaf(-n, kPio2C1, a_hi);
    return t1 + fmaf(-n, kPio2C2, a_lo);
}

// sin and cos of n·π/2 + t from the polynomial values at t.
__device__ __forceinline__ void apply_quadrant(int q, float st, float ct, float &s, float &c) {
    const bool swap = (q & 1) != 0;
    const float a = swap ? ct : st;
    const float b = swap ? st : ct;
    s = (q & 2) ? -a : a;
    c = ((q + 1) & 2) ? -b : b;
}

// Seed of one pair for a q-block. The K values s_k = sin(θ + k x), θ = q_s r,
// x = Δq r, are produced as two interleaved sequences, even k and odd k, each
// a sinusoid in j = k/2 with step y = 2x: s_{2j} = sin(θ + j y) and
// s_{2j+1} = sin(θ + x + j y). With x = m·π/2 + h (|h| <= π/4), y = mπ + 2h
// and both sequences are σ^j·v_j, σ = (−1)^m, where v follows the Reinsch
// recurrence with step 2h: d_{j+1} = d_j − α v_j, v_{j+1} = v_j + d_{j+1},
// α = 4 sin²h. Two independent chains per pair halve the dependency stall of
// the FFMA → FADD step without adding instructions.
//
// GENERAL_STEP = false is the path every pair of a tile takes when
// Δq·(largest distance) <= π/4: then m = 0, h = x, σ = 1 and the step needs
// no reduction.
struct PairSeed {
    float ve, de, vo, dd, na, we, wo;
};

template <bool GENERAL_STEP>
__device__ __forceinline__ PairSeed pair_seed(float4 pi, float4 pj, bool valid, float qs_hi,
                                              float qs_lo, float dq_hi, float dq_lo) {
    const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
    float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    // Coincident points: sinc(0) = 1, i.e. sin(q r)/r -> q; r = 1e-6 Å gives
    // that limit to 1e-13 relative.
    r2 = fmaxf(r2, 1e-12f);
    float inv_r = rsqrtf(r2);
    // r = r_hi + r_lo to ~2^-44 relative: one Newton step on sqrt, its
    // correction kept apart.
    const float r_hi = r2 * inv_r;
    const float hinv = 0.5f * inv_r;
    const float r_lo = hinv * fmaf(-r_hi, r_hi, r2);
    // One Newton step on 1/r as well (1 − r2·inv² = 1 − r_hi·inv): the weight
    // multiplies every term of the pair, so its error must be unbiased, not
    // just small.
    inv_r = fmaf(hinv, fmaf(-r_hi, inv_r, 1.0f), inv_r);
    // θ = q_s·r as hi + lo (exact product residue plus the cross terms of the
    // two double-float factors).
    const float th_hi = qs_hi * r_hi;
    const float th_lo = fmaf(qs_lo, r_hi, fmaf(qs_hi, r_lo, fmaf(qs_hi, r_hi, -th_hi)));
    int qt;
    const float t = reduce_pio2(th_hi, th_lo, qt);
    float st, ct, s0, c0;
    sincos_poly(t, st, ct);
    apply_quadrant(qt, st, ct, s0, c0);
    const float w = valid ? inv_r : 0.0f;
    PairSeed ps;
    ps.ve = s0;  // v_0 even = sin θ
    if (!GENERAL_STEP) {
        // r_lo matters here: rsqrtf's error need not average to zero, and a
        // step biased by δ moves the phase of the k-th point by k·δ.
        const float x = fmaf(dq_hi, r_hi, fmaf(dq_hi, r_lo, dq_lo * r_hi));
        float sx, cx;
        sincos_poly(x, sx, cx);
        const float sx2 = 2.0f * sx;
        ps.de = sx2 * fmaf(c0, cx, s0 * sx);  // sin θ − sin(θ − 2x) = 2 sin x cos(θ − x)
        ps.vo = fmaf(s0, cx, c0 * sx);        // sin(θ + x)
        ps.dd = sx2 * c0;                     // sin(θ + x) − sin(θ − x) = 2 sin x cos θ
        ps.na = -sx2 * sx2;                   // −α = −4 sin² x
        ps.we = w;
        ps.wo = w;
    } else {
        const float x_hi = dq_hi * r_hi;
        const float x_lo = fmaf(dq_lo, r_hi, fmaf(dq_hi, r_lo, fmaf(dq_hi, r_hi, -x_hi)));
        int qm;
        const float h = reduce_pio2(x_hi, x_lo, qm);
        float sh, ch, sx, cx;
        sincos_poly(h, sh, ch);
        apply_quadrant(qm, sh, ch, sx, cx);
        const float s1 = fmaf(s0, cx, c0 * sx);   // sin(θ + x)
        const float c1 = fmaf(c0, cx, -s0 * sx);  // cos(θ + x)
        const float sh2 = 2.0f * sh;
        ps.de = sh2 * fmaf(c0, ch, s0 * sh);      // sin θ − sin(θ − 2h) = 2 sin h cos(θ − h)
        ps.vo = s1;
        ps.dd = sh2 * fmaf(c1, ch, s1 * sh);      // sin(θ + x) − sin(θ + x − 2h)
        ps.na = -sh2 * sh2;                       // −α = −4 sin² h
        ps.we = w;
        ps.wo = (qm & 1) ? -w : w;                // σ = (−1)^m
    }
    return ps;
}

// The seeds of two pairs at once on packed FP32x2 instructions: every
// operation of pair_seed, in the same order and with the same roundings (a
// negation is a multiplication by -1, exact), with pair 0 in the low and
// pair 1 in the high half. Half the issue slots of two scalar seeds, and the
// packed operations occupy both FP32 sub-pipes together instead of leaving
// one of them idle beside a scalar operation.
#ifndef PD_SEED_X2
#define PD_SEED_X2 1
#endif
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ void sincos_poly_x2(float2 t, float2 &s, float2 &c) {
    const float2 t2 = __fmul2_rn(t, t);
    float2 ps = f2(2.789128530e-6f);
    ps = __ffma2_rn(ps, t2, f2(-1.984876289e-4f));
    ps = __ffma2_rn(ps, t2, f2(8.333369158e-3f));
    ps = __ffma2_rn(ps, t2, f2(-1.666666716e-1f));
    s = __ffma2_rn(__fmul2_rn(t, t2), ps, t);
    float2 pc = f2(2.443297126e-5f);
    pc = __ffma2_rn(pc, t2, f2(-1.388731296e-3f));
    pc = __ffma2_rn(pc, t2, f2(4.166664556e-2f));
    pc = __ffma2_rn(pc, t2, f2(-0.5f));
    c = __ffma2_rn(t2, pc, f2(1.0f));
}
// reduce_pio2 on both halves; the quadrants come back as integers.
__device__ __forceinline__ float2 reduce_pio2_x2(float2 a_hi, float2 a_lo, int &q0, int &q1) {
    const float2 nm = __ffma2_rn(a_hi, f2(0.636619772f), f2(kRoundMagic));
    const float2 n = __fadd2_rn(nm, f2(-kRoundMagic));  // exact
    q0 = __float_as_int(nm.x) & 3;
    q1 = __float_as_int(nm.y) & 3;
    const float2 t1 = __ffma2_rn(n, f2(-kPio2C1), a_hi);
    return __fadd2_rn(t1, __ffma2_rn(n, f2(-kPio2C2), a_lo));
}

template <bool GENERAL_STEP>
__device__ __forceinline__ void pair_seed_x2(float4 pi, float4 pj0, float4 pj1, bool valid0,
                                             bool valid1, float qs_hi, float qs_lo, float dq_hi,
                                             float dq_lo, PairSeed &S0, PairSeed &S1) {
    const float2 M1 = f2(-1.0f);
    const float2 dx = __ffma2_rn(make_float2(pj0.x, pj1.x), M1, f2(pi.x));
    const float2 dy = __ffma2_rn(make_float2(pj0.y, pj1.y), M1, f2(pi.y));
    const float2 dz = __ffma2_rn(make_float2(pj0.z, pj1.z), M1, f2(pi.z));
    float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
    r2 = make_float2(fmaxf(r2.x, 1e-12f), fmaxf(r2.y, 1e-12f));
    float2 inv_r = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
    const float2 r_hi = __fmul2_rn(r2, inv_r);
    const float2 nr_hi = __fmul2_rn(r_hi, M1);
    const float2 hinv = __fmul2_rn(f2(0.5f), inv_r);
    const float2 r_lo = __fmul2_rn(hinv, __ffma2_rn(nr_hi, r_hi, r2));
    inv_r = __ffma2_rn(hinv, __ffma2_rn(nr_hi, inv_r, f2(1.0f)), inv_r);
    const float2 th_hi = __fmul2_rn(f2(qs_hi), r_hi);
    const float2 th_lo =
        __ffma2_rn(f2(qs_lo), r_hi,
                   __ffma2_rn(f2(qs_hi), r_lo,
                              __ffma2_rn(f2(qs_hi), r_hi, __fmul2_rn(th_hi, M1))));
    int qt0, qt1;
    const float2 t = reduce_pio2_x2(th_hi, th_lo, qt0, qt1);
    float2 st, ct;
    sincos_poly_x2(t, st, ct);
    float s0a, c0a, s0b, c0b;
    apply_quadrant(qt0, st.x, ct.x, s0a, c0a);
    apply_quadrant(qt1, st.y, ct.y, s0b, c0b);
    const float2 s0 = make_float2(s0a, s0b), c0 = make_float2(c0a, c0b);
    const float w0 = valid0 ? inv_r.x : 0.0f, w1 = valid1 ? inv_r.y : 0.0f;
    S0.ve = s0a;
    S1.ve = s0b;
    if (!GENERAL_STEP) {
        const float2 x = __ffma2_rn(f2(dq_hi), r_hi,
                                    __ffma2_rn(f2(dq_hi), r_lo, __fmul2_rn(f2(dq_lo), r_hi)));
        float2 sx, cx;
        sincos_poly_x2(x, sx, cx);
        const float2 sx2 = __fmul2_rn(f2(2.0f), sx);
        const float2 de = __fmul2_rn(sx2, __ffma2_rn(c0, cx, __fmul2_rn(s0, sx)));
        const float2 vo = __ffma2_rn(s0, cx, __fmul2_rn(c0, sx));
        const float2 dd = __fmul2_rn(sx2, c0);
        const float2 na = __fmul2_rn(__fmul2_rn(sx2, M1), sx2);
        S0.de = de.x; S1.de = de.y;
        S0.vo = vo.x; S1.vo = vo.y;
        S0.dd = dd.x; S1.dd = dd.y;
        S0.na = na.x; S1.na = na.y;
        S0.we = S0.wo = w0;
        S1.we = S1.wo = w1;
    } else {
        const float2 x_hi = __fmul2_rn(f2(dq_hi), r_hi);
        const float2 x_lo =
            __ffma2_rn(f2(dq_lo), r_hi,
                       __ffma2_rn(f2(dq_hi), r_lo,
                                  __ffma2_rn(f2(dq_hi), r_hi, __fmul2_rn(x_hi, M1))));
        int qm0, qm1;
        const float2 h = reduce_pio2_x2(x_hi, x_lo, qm0, qm1);
        float2 sh, ch;
        sincos_poly_x2(h, sh, ch);
        float sxa, cxa, sxb, cxb;
        apply_quadrant(qm0, sh.x, ch.x, sxa, cxa);
        apply_quadrant(qm1, sh.y, ch.y, sxb, cxb);
        const float2 sx = make_float2(sxa, sxb), cx = make_float2(cxa, cxb);
        const float2 s1 = __ffma2_rn(s0, cx, __fmul2_rn(c0, sx));
        const float2 c1 = __ffma2_rn(c0, cx, __fmul2_rn(__fmul2_rn(s0, M1), sx));
        const float2 sh2 = __fmul2_rn(f2(2.0f), sh);
        const float2 de = __fmul2_rn(sh2, __ffma2_rn(c0, ch, __fmul2_rn(s0, sh)));
        const float2 dd = __fmul2_rn(sh2, __ffma2_rn(c1, ch, __fmul2_rn(s1, sh)));
        const float2 na = __fmul2_rn(__fmul2_rn(sh2, M1), sh2);
        S0.de = de.x; S1.de = de.y;
        S0.vo = s1.x; S1.vo = s1.y;
        S0.dd = dd.x; S1.dd = dd.y;
        S0.na = na.x; S1.na = na.y;
        S0.we = w0;
        S1.we = w1;
        S0.wo = (qm0 & 1) ? -w0 : w0;
        S1.wo = (qm1 & 1) ? -w1 : w1;
    }
}

// Small-q residual form: where q·(2·radius) < 2 every pair has q·r < 2 and
// the terms sin(q r)/r lie within a factor 0.45..1 of q, so a sequential FP32
// sum of them rounds with a systematic bias. There the kernel accumulates
// sin(q r)/r − q and the reduction adds (pair count)·q back in FP64. Both
// kernels evaluate this predicate on the same FP64 values.
__host__ __device__ __forceinline__ bool residual_q(double q, double radius) {
    return q * (2.0 * radius) < 2.0;
}

// ------------------------------------------------- shared-memory staging (TMA)
// One-dimensional bulk copies (cp.async.bulk, no multicast) of j-atom chunks
// into shared memory, completed on an mbarrier. Every wait is bounded: a
// copy that does not land within its poll limit makes the wait return false;
// the pair kernel then stops issuing copies, waits (bounded) for the ones in
// flight, poisons its results with NaN and sets a status bit the host reads,
// instead of hanging the GPU.
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned long long *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
                 : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Thread 0 only: `bytes` (a multiple of 16, <= 2^20) from global `src`
// (16-byte aligned) to shared `dst` (16-byte aligned), completing on `bar`.
__device__ __forceinline__ void bulk_copy_to_shared(void *dst, const void *src, uint32_t bytes,
                                                    unsigned long long *bar) {
    // order earlier generic-proxy reads of dst before the async-proxy write
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, uint32_t phase, int polls) {
    for (int it = 0; it < polls; ++it) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(smem_addr(bar)), "r"(phase)
            : "memory");
        if (done) return true;
    }
    return false;
}

// ---------------------------------------------------------------- K1 (FP32)
// Seeds of NP consecutive j atoms (clamped reads past the range are masked).
template <int MODE, int NP, bool RESID, bool GENERAL_STEP>
struct SeedGroup {
    PairSeed S[NP];
    float wj[NP];
    float vsum, vwsum;

    // `at` holds the atoms [jbase, j1) (a chunk staged in shared memory).
    __device__ __forceinline__ void make(const float4 *__restrict__ at, int jbase, float4 pi,
                                         int i, bool ivalid, int j, int j1, float qs_hi,
                                         float qs_lo, float dq_hi, float dq_lo) {
        vsum = 0.0f;
        vwsum = 0.0f;
        if constexpr (PD_SEED_X2 && NP % 2 == 0) {
#pragma unroll
            for (int p = 0; p < NP; p += 2) {
                const int ja = j + p, jb = j + p + 1;
                const bool ina = ja < j1, inb = jb < j1;
                const float4 pja = at[(ina ? ja : j1 - 1) - jbase];
                const float4 pjb = at[(inb ? jb : j1 - 1) - jbase];
                const bool va = ivalid && ina && (ja > i), vb = ivalid && inb && (jb > i);
                pair_seed_x2<GENERAL_STEP>(pi, pja, pjb, va, vb, qs_hi, qs_lo, dq_hi, dq_lo,
                                           S[p], S[p + 1]);
                if (MODE == PD_MODE_WEIGHTED) {
                    wj[p] = pja.w;
                    wj[p + 1] = pjb.w;
                }
                if (RESID) {
                    vsum += (va ? 1.0f : 0.0f) + (vb ? 1.0f : 0.0f);
                    if (MODE == PD_MODE_WEIGHTED) {
                        vwsum += va ? pja.w : 0.0f;
                        vwsum += vb ? pjb.w : 0.0f;
                    }
                }
            }
            return;
        }
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const int jj = j + p;
            const bool inr = jj < j1;
            const float4 pj = at[(inr ? jj : j1 - 1) - jbase];
            const bool valid = ivalid && inr && (jj > i);
            S[p] = pair_seed<GENERAL_STEP>(pi, pj, valid, qs_hi, qs_lo, dq_hi, dq_lo);
            if (MODE == PD_MODE_WEIGHTED) wj[p] = pj.w;
            if (RESID) {
                vsum += valid ? 1.0f : 0.0f;
                if (MODE == PD_MODE_WEIGHTED) vwsum += valid ? pj.w : 0.0f;
            }
        }
    }
};

// NP pairs per thread per pass, two chains each: 2·NP independent
// recurrences. The seeds of the next pass are computed in the same straight-
// line block as the K steps of the current one, so their long dependency
// chains (sqrt, reductions, polynomials) overlap the recurrence instead of
// stalling the warp between passes.
template <int K, int MODE, int NP, bool RESID, bool GENERAL_STEP>
__device__ __forceinline__ void pairs_range(const float4 *__restrict__ at, int jbase, float4 pi,
                                            int i, bool ivalid, int j0, int j1, float qs_hi,
                                            float qs_lo, float dq_hi, float dq_lo,
                                            const float *__restrict__ s_qres,
                                            float (&acc)[(MODE == PD_MODE_WEIGHTED) ? 2 : 1][K]) {
    constexpr int NACC = (MODE == PD_MODE_WEIGHTED) ? 2 : 1;
    static_assert(K % 4 == 0, "K must be a multiple of 4");
    if (j0 >= j1) return;
    SeedGroup<MODE, NP, RESID, GENERAL_STEP> cur;
    cur.make(at, jbase, pi, i, ivalid, j0, j1, qs_hi, qs_lo, dq_hi, dq_lo);
    for (int j = j0; j < j1; j += NP) {
        SeedGroup<MODE, NP, RESID, GENERAL_STEP> nxt;  // unused after the last pass
        nxt.make(at, jbase, pi, i, ivalid, j + NP, j1, qs_hi, qs_lo, dq_hi, dq_lo);
        float we_w[NP], wo_w[NP];
        if (MODE == PD_MODE_WEIGHTED) {
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                we_w[p] = cur.S[p].we * cur.wj[p];
                wo_w[p] = cur.S[p].wo * cur.wj[p];
            }
        }
        // The q table is the same in every pass; an opaque zero offset keeps
        // the compiler from hoisting all K loads into registers.
        int qoff = 0;
        if (RESID) asm volatile("mov.b32 %0, %0;" : "+r"(qoff));
#pragma unroll
        for (int k = 0; k < K; k += 4) {
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const int kk = k + h;
                const bool odd_chain = (h & 1) != 0;  // k = 4t+1, 4t+3
                const bool odd_j = (h & 2) != 0;      // j = 2t+1: weight σ·w
                if (RESID) {
                    const float qk = s_qres[kk + qoff];
                    acc[0][kk] = fmaf(-cur.vsum, qk, acc[0][kk]);
                    if (MODE == PD_MODE_WEIGHTED)
                        acc[NACC - 1][kk] = fmaf(-cur.vwsum, qk, acc[NACC - 1][kk]);
                }
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    const float w = odd_j ? cur.S[p].wo : cur.S[p].we;
                    float &v = odd_chain ? cur.S[p].vo : cur.S[p].ve;
                    float &d = odd_chain ? cur.S[p].dd : cur.S[p].de;
                    acc[0][kk] = fmaf(w, v, acc[0][kk]);
                    if (MODE == PD_MODE_WEIGHTED)
                        acc[NACC - 1][kk] = fmaf(odd_j ? wo_w[p] : we_w[p], v, acc[NACC - 1][kk]);
                    d = fmaf(cur.S[p].na, v, d);
                    v += d;
                }
            }
        }
        cur = nxt;
    }
}

// Class mode on packed FP32x2 instructions (fma.rn.f32x2 / add.rn.f32x2,
// sm_100): the even and odd chain of a pair sit in the two halves of one
// register pair, V = (v_even, v_odd), D = (d_even, d_odd), and so do the
// accumulators of grid points 2t and 2t+1: one step t advances both chains
// and both accumulators with FFMA2 + FADD2 + FFMA2. The FP32 pipe does the
// same lane work as with scalar instructions, but a warp needs half the issue
// slots for it, which leaves the issue port to the seeds and lets the FMA
// pipe, not instruction issue, bound the kernel. Each half rounds exactly as
// the scalar fmaf/add would.
//
// A block runs only its first `nchunk` chunks of 16 grid points: the last
// q-block of a grid whose length is not a multiple of K skips the steps past
// the grid end instead of computing and discarding them. (One uniform branch
// per chunk in a single code path measured faster on B200 than a separate
// copy of the loop for tail blocks, which raised register spills.)
#ifndef PD_SCALED_V
#define PD_SCALED_V 1
#endif
// Where the seeds of a pass are computed. Computing each pass's seeds
// before its steps holds no next-pass seeds through the steps: fewer
// registers, so more resident CTAs or fewer spills, and the extra warps per
// scheduler hide the seeds' dependency chains. Measured on B200 (pair-kernel
// time): K = 128 with four pairs per thread fits 168 registers and three CTAs
// per SM instead of 255 and two, 546.7 ms against 556.0 ms on the
// 100,000-atom solve (558.5 ms with the seeds at the top but two CTAs); K = 64
// with four pairs loses its spills at four CTAs, 0.216 against 0.232 ms on
// 3,000 atoms at nq 300; the weighted mode's K = 64 fits three CTAs instead of
// two, 814 against 842 ms on the 100,000-atom solve with per-atom weights.
// The other shapes compute the next pass's seeds while the current pass
// steps (K = 128 with two pairs: 3.117 against 3.121 ms on 10,000 atoms).
#ifndef PD_SEED_TOP
#define PD_SEED_TOP 1
#endif
template <int K, int NP>
constexpr bool seeds_at_top() {
    return PD_SEED_TOP && (K == 64 || (K == 128 && NP == 4));
}
template <int K, int NP>
constexpr bool seeds_at_top_w() {
    return PD_SEED_TOP && K == 64;
}
// Instruction order within a step: 0 = d-steps, accumulations, v-steps;
// 1 = d-steps, then per pair its accumulation and v-step; 2 (with
// PD_SCALED_V, two or four pairs) = the pairs' scaled terms summed, then
// added to the accumulator (measured 1.5 % faster than 0 on the 100,000-atom
// solve: the accumulator's dependency chain is one add per step instead of
// one per pair).
#ifndef PD_STEP_ORDER
#define PD_STEP_ORDER 2
#endif
// Steps between two checks for the end of the grid (a chunk of 2·PD_CHUNK_T
// grid points).
#ifndef PD_CHUNK_T
#define PD_CHUNK_T 8
#endif
template <int K, int NP, bool RESID, bool GENERAL_STEP>
__device__ __forceinline__ void pairs_range_x2(const float4 *__restrict__ at, int jbase, float4 pi,
                                               int i, bool ivalid, int j0, int j1, float qs_hi,
                                               float qs_lo, float dq_hi, float dq_lo,
                                               const float2 *__restrict__ s_qres2,
                                               float2 (&acc)[K / 2], int nchunk,
                                               int rchunk = K / 16) {
    static_assert(K % 16 == 0, "K must be a multiple of 16");
    if (j0 >= j1) return;
    SeedGroup<PD_MODE_CLASS, NP, RESID, GENERAL_STEP> cur;
    constexpr bool TOP = seeds_at_top<K, NP>();
    if (!TOP) cur.make(at, jbase, pi, i, ivalid, j0, j1, qs_hi, qs_lo, dq_hi, dq_lo);
    for (int j = j0; j < j1; j += NP) {
        if (TOP) cur.make(at, jbase, pi, i, ivalid, j, j1, qs_hi, qs_lo, dq_hi, dq_lo);
        // SCALED: without the general step every term of a pair has the
        // weight w = 1/r, which the linear recurrence can carry in v and d
        // themselves; the accumulation is then a plain add.
        constexpr bool SCALED = PD_SCALED_V && !GENERAL_STEP;
        float2 V[NP], D[NP], NA[NP], WE[NP], WO[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            if (SCALED) {
                const float w = cur.S[p].we;
                V[p] = make_float2(w * cur.S[p].ve, w * cur.S[p].vo);
                D[p] = make_float2(w * cur.S[p].de, w * cur.S[p].dd);
            } else {
                V[p] = make_float2(cur.S[p].ve, cur.S[p].vo);
                D[p] = make_float2(cur.S[p].de, cur.S[p].dd);
                WE[p] = make_float2(cur.S[p].we, cur.S[p].we);
                WO[p] = GENERAL_STEP ? make_float2(cur.S[p].wo, cur.S[p].wo) : WE[p];
            }
            NA[p] = make_float2(cur.S[p].na, cur.S[p].na);
        }
        const float2 mvs = make_float2(-cur.vsum, -cur.vsum);
        // the next pass's seeds (unused after the last pass), computed in
        // place while the steps below run on this pass's copies
        if (!TOP) cur.make(at, jbase, pi, i, ivalid, j + NP, j1, qs_hi, qs_lo, dq_hi, dq_lo);
        int qoff = 0;  // opaque zero: keeps the K/2 q loads in the loop
        if (RESID) asm volatile("mov.b32 %0, %0;" : "+r"(qoff));
#pragma unroll
        for (int t = 0; t < K / 2; ++t) {
            if ((t % PD_CHUNK_T) == 0 && t / PD_CHUNK_T >= nchunk) break;
            // the residual points are a prefix of the block: only its first
            // rchunk 16-point chunks subtract q
            if (RESID && (t / 8) < rchunk) acc[t] = __ffma2_rn(mvs, s_qres2[t + qoff], acc[t]);
            // d-steps of all pairs, then the accumulations, then the
            // v-steps: every instruction's operands are a group old
            // (measured 0.5 % faster than the per-pair order).
#pragma unroll
            for (int p = 0; p < NP; ++p) D[p] = __ffma2_rn(NA[p], V[p], D[p]);
            if constexpr (SCALED && PD_STEP_ORDER == 2 && (NP == 2 || NP == 4)) {
                // the pairs' scaled terms added among themselves first, then
                // to the accumulator: one dependent add per step on acc[t]
                float2 sum = __fadd2_rn(V[0], V[1]);
                if constexpr (NP == 4) sum = __fadd2_rn(sum, __fadd2_rn(V[2], V[3]));
#pragma unroll
                for (int p = 0; p < NP; ++p) V[p] = __fadd2_rn(V[p], D[p]);
                acc[t] = __fadd2_rn(acc[t], sum);
            } else if constexpr (PD_STEP_ORDER == 0 || PD_STEP_ORDER == 2) {
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    if constexpr (SCALED)
                        acc[t] = __fadd2_rn(V[p], acc[t]);
                    else
                        acc[t] = __ffma2_rn((t & 1) ? WO[p] : WE[p], V[p], acc[t]);
                }
#pragma unroll
                for (int p = 0; p < NP; ++p) V[p] = __fadd2_rn(V[p], D[p]);
            } else {
                // each pair's accumulation, then its v-step
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    if constexpr (SCALED)
                        acc[t] = __fadd2_rn(V[p], acc[t]);
                    else
                        acc[t] = __ffma2_rn((t & 1) ? WO[p] : WE[p], V[p], acc[t]);
                    V[p] = __fadd2_rn(V[p], D[p]);
                }
            }
        }
    }
}

// Weighted mode on packed FP32x2 instructions: the same chains as
// pairs_range_x2 with two accumulators per grid point, Σ w d/r-terms (acc0)
// and Σ w_j·terms (acc1). Without the general step the weight 1/r rides in
// v and d (SCALED), acc0 takes the pairs' terms summed among themselves and
// acc1 one FFMA2 per pair with w_j: four FP32 lane slots per pair·q (d-step,
// v-step, the two accumulations), on half the issue slots of the scalar
// form.
#ifndef PD_WEIGHTED_X2
#define PD_WEIGHTED_X2 1
#endif
template <int K, int NP, bool RESID, bool GENERAL_STEP>
__device__ __forceinline__ void pairs_range_x2w(const float4 *__restrict__ at, int jbase,
                                                float4 pi, int i, bool ivalid, int j0, int j1,
                                                float qs_hi, float qs_lo, float dq_hi,
                                                float dq_lo, const float2 *__restrict__ s_qres2,
                                                float2 (&acc0)[K / 2], float2 (&acc1)[K / 2],
                                                int nchunk, int rchunk = K / 16) {
    static_assert(K % 16 == 0, "K must be a multiple of 16");
    if (j0 >= j1) return;
    constexpr bool SCALED = PD_SCALED_V && !GENERAL_STEP;
    SeedGroup<PD_MODE_WEIGHTED, NP, RESID, GENERAL_STEP> cur;
    constexpr bool TOP = seeds_at_top_w<K, NP>();
    if (!TOP) cur.make(at, jbase, pi, i, ivalid, j0, j1, qs_hi, qs_lo, dq_hi, dq_lo);
    for (int j = j0; j < j1; j += NP) {
        if (TOP) cur.make(at, jbase, pi, i, ivalid, j, j1, qs_hi, qs_lo, dq_hi, dq_lo);
        float2 V[NP], D[NP], NA[NP], WJ[NP], WE[NP], WO[NP], WJE[NP], WJO[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const float w = cur.S[p].we;
            if (SCALED) {
                V[p] = make_float2(w * cur.S[p].ve, w * cur.S[p].vo);
                D[p] = make_float2(w * cur.S[p].de, w * cur.S[p].dd);
                WJ[p] = make_float2(cur.wj[p], cur.wj[p]);
            } else {
                V[p] = make_float2(cur.S[p].ve, cur.S[p].vo);
                D[p] = make_float2(cur.S[p].de, cur.S[p].dd);
                const float wo = cur.S[p].wo;
                WE[p] = make_float2(w, w);
                WO[p] = make_float2(wo, wo);
                WJE[p] = make_float2(w * cur.wj[p], w * cur.wj[p]);
                WJO[p] = make_float2(wo * cur.wj[p], wo * cur.wj[p]);
            }
            NA[p] = make_float2(cur.S[p].na, cur.S[p].na);
        }
        const float2 mvs = make_float2(-cur.vsum, -cur.vsum);
        const float2 mvws = make_float2(-cur.vwsum, -cur.vwsum);
        if (!TOP) cur.make(at, jbase, pi, i, ivalid, j + NP, j1, qs_hi, qs_lo, dq_hi, dq_lo);
        int qoff = 0;  // opaque zero: keeps the K/2 q loads in the loop
        if (RESID) asm volatile("mov.b32 %0, %0;" : "+r"(qoff));
#pragma unroll
        for (int t = 0; t < K / 2; ++t) {
            if ((t % PD_CHUNK_T) == 0 && t / PD_CHUNK_T >= nchunk) break;
            if (RESID && (t / 8) < rchunk) {
                const float2 q2 = s_qres2[t + qoff];
                acc0[t] = __ffma2_rn(mvs, q2, acc0[t]);
                acc1[t] = __ffma2_rn(mvws, q2, acc1[t]);
            }
#pragma unroll
            for (int p = 0; p < NP; ++p) D[p] = __ffma2_rn(NA[p], V[p], D[p]);
            if constexpr (SCALED) {
                float2 sum = V[0];
#pragma unroll
                for (int p = 1; p < NP; ++p) sum = __fadd2_rn(sum, V[p]);
                float2 a1 = acc1[t];
#pragma unroll
                for (int p = 0; p < NP; ++p) a1 = __ffma2_rn(WJ[p], V[p], a1);
                acc1[t] = a1;
                acc0[t] = __fadd2_rn(acc0[t], sum);
            } else {
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    acc0[t] = __ffma2_rn((t & 1) ? WO[p] : WE[p], V[p], acc0[t]);
                    acc1[t] = __ffma2_rn((t & 1) ? WJO[p] : WJE[p], V[p], acc1[t]);
                }
            }
#pragma unroll
            for (int p = 0; p < NP; ++p) V[p] = __fadd2_rn(V[p], D[p]);
        }
    }
}

// Pairs a thread adds in FP32 before the warp's partial sums go into its
// FP64 slot. A j range of a tile is walked in sub-chunks of this length with
// fresh FP32 accumulators: FP32 running sums over thousands of terms lose
// ε·|running sum| per addition (and over same-sign terms that loss has a
// sign), which on sums of 10^9 pairs that cancel to 10^-5 of their scale
// shows up in the result; short FP32 runs keep it far below the profile.
#ifndef PD_JFLUSH
#define PD_JFLUSH 512
#endif
// The same for the moments: their low orders are sums of nearly equal terms at
// every grid point, so the rounding of long runs shows in the profile (largest error
// of a point against FP64, 8,000 atoms, q_max·d = 247: 1.1e-6 with 128 pairs, 4e-7 with
// 32; the grid points 2e-7). The shorter runs and their flushes cost 5 to 12 %.
#ifndef PD_MOM_FLUSH
#define PD_MOM_FLUSH 32
#endif
// j atoms per bulk copy into shared memory (two buffers of PD_JSTAGE float4,
// 64 KB of dynamic shared memory per CTA); a multiple of PD_JFLUSH. One CTA
// barrier per stage releases the buffer for the next copy.
#ifndef PD_JSTAGE_ATOMS
#define PD_JSTAGE_ATOMS 2048
#endif
constexpr int PD_JSTAGE = PD_JSTAGE_ATOMS;
static_assert(PD_JSTAGE % PD_JFLUSH == 0 && PD_JSTAGE % PD_MOM_FLUSH == 0,
              "stage must hold whole sub-chunks");
constexpr size_t PD_FP32_DYN_SMEM = 2 * PD_JSTAGE * sizeof(float4);

// Resident CTAs per SM each FP32 shape is compiled for (register budget
// 65536 / (128 · blocks) per thread).
constexpr int fp32_min_blocks(int K, int MODE, int NP) {
    return MODE == PD_MODE_CLASS
               ? (K <= 64 ? 4 : (K <= 128 && (NP <= 2 || (PD_SEED_TOP && K == 128 && NP == 4)) ? 3 : 2))
               : (K <= 32 ? 4 : (PD_SEED_TOP && K == 64 ? 3 : 2));
}

// Polls of a bulk-copy wait before it gives up: the normal limit, and the
// short one of the test hook (PD_REQF_TEST_EXPIRE), whose copy is never
// issued.
constexpr int PD_WAIT_POLLS = 1 << 22;
constexpr int PD_TEST_WAIT_POLLS = 1 << 10;

// Class-mode flush: the warp sums of acc, added to the warp's FP64 partials
// part[0 .. 2·NT) in the order of the values.
template <int NT>
__device__ __forceinline__ void flush_class(float2 (&acc)[NT], double *__restrict__ part, int lane,
                                            bool first) {
    if constexpr (NT % 32 == 0) {
        // reduce-scatter: lane l ends with the sums of values [l·NT/16, (l+1)·NT/16)
        warp_reduce_scatter<NT>(acc, lane);
#pragma unroll
        for (int m = 0; m < NT / 16; ++m) {
            double &d = part[lane * (NT / 16) + m];
            const float sum = (m & 1) ? acc[m >> 1].y : acc[m >> 1].x;
            d = (first ? 0.0 : d) + static_cast<double>(sum);
        }
    } else {
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const float v0 = warp_sum(acc[t].x);
            const float v1 = warp_sum(acc[t].y);
            if (lane == ((2 * t) & 31))
                part[2 * t] = (first ? 0.0 : part[2 * t]) + static_cast<double>(v0);
            if (lane == ((2 * t + 1) & 31))
                part[2 * t + 1] = (first ? 0.0 : part[2 * t + 1]) + static_cast<double>(v1);
        }
    }
}

// The same for moments: the lanes' sums meet in FP32 up to four of them, the rest in
// FP64 (low moments are sums of equal terms: all five levels in FP32 cost as much
// accuracy as runs four times as long).
template <int NT>
__device__ __forceinline__ void flush_moments(float2 (&acc)[NT], double *__restrict__ part,
                                              int lane, bool first) {
#pragma unroll
    for (int lev = 0; lev < 2; ++lev) {  // reduce-scatter, as warp_reduce_scatter
        const int o = 16 >> lev, h = (NT >> lev) / 2;
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const float2 keep = up ? acc[k + h] : acc[k], send = up ? acc[k] : acc[k + h];
            acc[k] = __fadd2_rn(keep, make_float2(__shfl_xor_sync(0xffffffffu, send.x, o),
                                                  __shfl_xor_sync(0xffffffffu, send.y, o)));
        }
    }
    double v[NT / 2];
#pragma unroll
    for (int k = 0; k < NT / 2; ++k) v[k] = static_cast<double>((k & 1) ? acc[k / 2].y : acc[k / 2].x);
#pragma unroll
    for (int lev = 0; lev < 3; ++lev) {
        const int o = 4 >> lev, h = (NT >> lev) / 4;
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const double keep = up ? v[k + h] : v[k], send = up ? v[k] : v[k + h];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (int m = 0; m < NT / 16; ++m) {  // values [l·NT/16, (l + 1)·NT/16) in lane l
        double &d = part[lane * (NT / 16) + m];
        d = (first ? 0.0 : d) + v[m];
    }
}

// The j range and moment block of a moment-form job (see PdFrameDev): part
// qb / n_mblk of the tile's range, cut at multiples of 32 atoms from its start.
struct MomJob {
    int j0, j1, mb;
};
__device__ __forceinline__ MomJob moment_job(int j0, int j1, int qb, int n_mblk, int n_parts) {
    const int part = qb / n_mblk;
    const int len = ((j1 - j0 + n_parts - 1) / n_parts + 31) & ~31;
    MomJob m;
    m.mb = qb - part * n_mblk;
    m.j0 = min(j1, j0 + part * len);
    m.j1 = part < n_parts ? min(j1, m.j0 + len) : m.j0;
    return m;
}

// Weighted-mode flush of one accumulator array: the warp sums of acc and of
// w_i·acc, added to part[k] and part[stride + k].
template <int K, bool MOMENTS>
__device__ __forceinline__ void flush_weighted(float2 (&acc)[K / 2], float wi,
                                               double *__restrict__ part, int stride, int lane,
                                               bool first) {
    const float2 wi2 = make_float2(wi, wi);
    float2 tw[K / 2];
#pragma unroll
    for (int t = 0; t < K / 2; ++t) tw[t] = __fmul2_rn(wi2, acc[t]);
    if constexpr (MOMENTS) {
        flush_moments<K / 2>(acc, part, lane, first);
        flush_moments<K / 2>(tw, part + stride, lane, first);
    } else {
        flush_class<K / 2>(acc, part, lane, first);
        flush_class<K / 2>(tw, part + stride, lane, first);
    }
}

// Moment form: a stage's j atoms [jss, jse) of a job that starts at tj0, in runs of
// PD_MOM_FLUSH. Not inlined: its accumulators would cost the grid points' steps
// registers (weighted mode, K = 64: 448 bytes of spills against 164).
template <int K, int MODE>
__device__ __noinline__ void moments_stage(const float4 *__restrict__ chunk, int jss, int jse,
                                           int tj0, float4 pi, int i, bool ivalid, float inv_d2,
                                           int nj, int mblk, double *__restrict__ part, int lane) {
    constexpr int KM = pd_moment_block(K);
    constexpr int DBL = KM == 128 ? 4 : (KM == 64 ? 3 : 2);
    for (int js = jss; js < jse; js += PD_MOM_FLUSH) {
        const int je = min(jse, js + PD_MOM_FLUSH);
        const bool first = js == tj0;
        float2 acc0[KM / 2];
#pragma unroll
        for (int t = 0; t < KM / 2; ++t) acc0[t] = make_float2(0.0f, 0.0f);
        if constexpr (MODE == PD_MODE_CLASS) {
            float2 none[1];
            moments_range<KM, false>(chunk, jss, pi, i, ivalid, js, je, inv_d2, nj, mblk, DBL, acc0,
                                     none);
            flush_moments<KM / 2>(acc0, part, lane, first);
        } else {
            float2 acc1[KM / 2];
#pragma unroll
            for (int t = 0; t < KM / 2; ++t) acc1[t] = make_float2(0.0f, 0.0f);
            moments_range<KM, true>(chunk, jss, pi, i, ivalid, js, je, inv_d2, nj, mblk, DBL, acc0,
                                    acc1);
            const float wi = ivalid ? pi.w : 0.0f;
            flush_weighted<KM, true>(acc0, wi, part, K, lane, first);
            flush_weighted<KM, true>(acc1, wi, part + 2 * K, K, lane, first);
        }
    }
}

// End of a tile: the warps' FP64 partial sums (part[w·nvk + e], e < nvk) of
// one class are added in warp order and written to that class's slot; a CTA
// whose copy wait expired writes NaN instead, and an empty tile zeros.
__device__ __forceinline__ void merge_tile_slots(const double *__restrict__ part, int nvk,
                                                 int64_t slot_word, double *__restrict__ slots,
                                                 bool dead, bool empty) {
    const int64_t slot0 = slot_word & PD_SLOT_MASK;
    const int smap = static_cast<int>(slot_word >> PD_SLOT_MAP_SHIFT) & 0xff;
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    for (int e = threadIdx.x; e < nvk; e += blockDim.x) {
        double a[PD_WARPS];
        int used = 0;
#pragma unroll
        for (int w = 0; w < PD_WARPS; ++w) {
            const int s = (smap >> (2 * w)) & 3;
            const double v = part[w * nvk + e];
            a[s] = (used & (1 << s)) ? a[s] + v : v;
            used |= 1 << s;
        }
#pragma unroll
        for (int s = 0; s < PD_WARPS; ++s)
            if (used & (1 << s))
                slots[(slot0 + s) * nvk + e] = dead ? nan : (empty ? 0.0 : a[s]);
    }
}

// Whether any frame of a request sums pairs: without one the pair kernel of a
// plan is left at once, its job list unread (uniform; the frames are read side by side).
__device__ __forceinline__ bool plan_sums_pairs(const PdReqDev &rq, int n_frames) {
    int any = 0;
    for (int f = threadIdx.x; f < n_frames; f += PD_THREADS) any |= rq.frames[f].n_grp == 0;
    return __syncthreads_or(any) != 0;
}

// The next job of a frame that sums pairs (one thread asks; n_jobs or more: none). The
// jobs of frames in the direction form are passed over here, where a branch around a
// whole tile cost the FP64 kernel's steps 13 % (5,000 atoms, 300 points: 13.3 ms
// against 11.7 ms). A block's first job is its own number: the longest come first, and
// blocks that wait for the frames' constants side by side would draw them in any order,
// two long ones for one SM (4 frames of 2,043 atoms, FP64, one grid block: 1.29 or
// 1.40 ms from one call to the next).
__device__ __forceinline__ int next_pair_job(const PdJob *__restrict__ jobs, int n_jobs,
                                             const PdReqDev *__restrict__ reqs,
                                             int *__restrict__ counter, bool first) {
    int jid = first ? blockIdx.x : gridDim.x + atomicAdd(counter, 1);
    while (jid < n_jobs && reqs[jobs[jid].req].frames[jobs[jid].frame].n_grp > 0)
        jid = gridDim.x + atomicAdd(counter, 1);
    return jid;
}

template <int K, int MODE, int NP>
__global__ void __launch_bounds__(PD_THREADS, fp32_min_blocks(K, MODE, NP))
    pd_pairs_fp32(const PdJob *__restrict__ jobs, const int *__restrict__ n_jobs_ptr,
                  const PdReqDev *__restrict__ reqs, int *__restrict__ counter, int plan_frames) {
    chain_enter();
    constexpr int NACC = (MODE == PD_MODE_WEIGHTED) ? 2 : 1;
    constexpr int NV = (MODE == PD_MODE_WEIGHTED) ? 4 : 1;  // FP64 values per q in a slot
    constexpr bool PACKED = (MODE == PD_MODE_CLASS);
    constexpr bool PACKED_W =
        (MODE == PD_MODE_WEIGHTED) && PD_WEIGHTED_X2 && (K / 2) % 32 == 0 && NP % 2 == 0;
    __shared__ int s_job;
    __shared__ __align__(16) float s_qres[K];
    // per-warp FP64 partial sums of the current tile, [warp][NV][K]
    __shared__ double s_part[PD_WARPS * NV * K];
    // j atoms of the current and the next stage, staged by bulk copies
    // (PD_FP32_DYN_SMEM bytes of dynamic shared memory)
    extern __shared__ __align__(128) float4 pd_dyn_atoms[];
    float4 *s_atoms[2] = {pd_dyn_atoms, pd_dyn_atoms + PD_JSTAGE};
    __shared__ __align__(8) unsigned long long s_bar[2];
    // Once a copy wait of this CTA expires the CTA is "dead" for the rest of
    // the launch: it issues no more copies, computes nothing, writes NaN to
    // the slots of every tile it still takes and flags each tile's request
    // in its status word. This state lives in shared memory, not registers,
    // so that it adds nothing to the register pressure of the steps.
    __shared__ int s_dead, s_polls, s_skip;
    __shared__ int s_empty;  // the job has no pairs: its slots are zeros
    __shared__ uint32_t s_inflight, s_par;  // thread 0: copies in flight, their parities
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int n_jobs = *n_jobs_ptr;
    if (threadIdx.x == 0) {
        mbar_init(&s_bar[0], 1);
        mbar_init(&s_bar[1], 1);
        mbar_init_fence();
        s_dead = 0;
    }
    __syncthreads();
    uint32_t phase = 0;  // bit b: parity of buffer b's next completion
    double *part = s_part + warp * NV * K;
    if (plan_frames > 0 && !plan_sums_pairs(reqs[0], plan_frames)) return;
    for (bool first = true;; first = false) {
        if (threadIdx.x == 0) s_job = next_pair_job(jobs, n_jobs, reqs, counter, first);
        __syncthreads();
        const int jid = s_job;
        if (jid >= n_jobs) break;
        const PdJob jb = jobs[jid];
        const PdReqDev rq = reqs[jb.req];
        const int kq0 = jb.qb * K;
        const PdFrameDev fr = rq.frames[jb.frame];
        const double radius = fr.radius;
        // moment form: this job's part of the j range and its moment block
        const bool moments = fr.n_mom > 0;
        int tj0 = jb.j0, tj1 = jb.j1, mblk = 0;
        if (moments) {
            const MomJob mj = moment_job(jb.j0, jb.j1, jb.qb, fr.n_mblk, fr.n_parts);
            tj0 = mj.j0;
            tj1 = mj.j1;
            mblk = mj.mb;
        }
        const bool resid = !moments && kq0 < rq.nq && residual_q(rq.qv[kq0], radius);
        int nres = 0;  // leading grid points of the block in the residual form
        if (resid) {
            for (int base = 0; base < K; base += PD_THREADS) {
                const int t = base + threadIdx.x;
                bool on = false;
                if (t < K) {
                    const int kq = kq0 + t;
                    on = kq < rq.nq && residual_q(rq.qv[kq], radius);
                    s_qres[t] = on ? static_cast<float>(rq.qv[kq]) : 0.0f;
                }
                nres += __syncthreads_count(on);
            }
        }
        const int rchunk = (nres + 15) >> 4;
        if (threadIdx.x == 0) {
            // test hook: the CTA that takes the launch's first tile waits for
            // a copy that is never issued, briefly, so that its wait expires
            // with no copy in flight
            s_skip = (rq.flags & PD_REQF_TEST_EXPIRE) != 0 && jid == 0;
            s_polls = s_skip ? PD_TEST_WAIT_POLLS : PD_WAIT_POLLS;
            s_inflight = 0;
            s_par = 0;
            s_empty = tj1 <= tj0;
        }
        __syncthreads();  // s_qres and the tile state ready; every thread has read s_job
        const float4 *__restrict__ at = rq.atoms32 + static_cast<size_t>(jb.frame) * rq.n_pad;
        const int i = jb.i0 + threadIdx.x;
        const float4 pi = at[i];
        const bool ivalid = lane < rq.gvalid[(jb.i0 >> 5) + warp];
        const double qs = rq.qmin + static_cast<double>(kq0) * rq.dq;
        const float qs_hi = static_cast<float>(qs);
        const float qs_lo = static_cast<float>(qs - static_cast<double>(qs_hi));
        const float dq_hi = static_cast<float>(rq.dq);
        const float dq_lo = static_cast<float>(rq.dq - static_cast<double>(dq_hi));
        // Every pair distance is at most 2·radius (positions are centred):
        // below π/4 for the step angle Δq·r the seeds skip its reduction.
        const bool general_step = rq.dq * (2.0 * radius) > 0.78;
        const int nstage = s_dead ? 0 : (tj1 - tj0 + PD_JSTAGE - 1) / PD_JSTAGE;
        if (threadIdx.x == 0 && nstage > 0 && !s_skip) {
            bulk_copy_to_shared(s_atoms[0], at + tj0,
                                static_cast<uint32_t>(min(tj1 - tj0, PD_JSTAGE)) * 16,
                                &s_bar[0]);
            s_inflight = 1u;
            s_par = phase & 1u;
        }
        for (int stg = 0; stg < nstage; ++stg) {
            const int jss = tj0 + stg * PD_JSTAGE;
            const int jse = min(tj1, jss + PD_JSTAGE);
            if (threadIdx.x == 0 && stg + 1 < nstage) {  // its buffer was released at stg - 1
                const int nb = (stg + 1) & 1;
                bulk_copy_to_shared(s_atoms[nb], at + jse,
                                    static_cast<uint32_t>(min(tj1 - jse, PD_JSTAGE)) * 16,
                                    &s_bar[nb]);
                s_inflight |= 1u << nb;
                s_par = (s_par & ~(1u << nb)) | (phase & (1u << nb));
            }
            const int b = stg & 1;
            const bool landed = mbar_wait(&s_bar[b], (phase >> b) & 1u, s_polls);
            phase ^= 1u << b;
            if (threadIdx.x == 0 && landed) s_inflight &= ~(1u << b);
            // A chunk that did not land is computed anyway (its shared memory
            // holds stale atoms, harmless to read) and the tile is poisoned
            // below: no branch around the steps.
            const float4 *chunk = s_atoms[b];
            {
                if (moments) {
                    constexpr int KM = pd_moment_block(K);
                    moments_stage<K, MODE>(chunk, jss, jse, tj0, pi, i, ivalid,
                                           static_cast<float>(fr.inv_d2),
                                           min(KM, fr.n_mom - mblk * KM) >> 3, mblk, part, lane);
                }
                for (int js = moments ? jse : jss; js < jse; js += PD_JFLUSH) {
                    const int je = min(jse, js + PD_JFLUSH);
                    const bool first = js == tj0;
                    if constexpr (PACKED) {
                        const float2 *q2 = reinterpret_cast<const float2 *>(s_qres);
                        // 16-point chunks of this block that lie on the grid.
                        // The small-q residual blocks (the first of a grid)
                        // run whole: a tail check there costs the register
                        // spills it saves in steps.
                        const int nchunk =
                            (min(K, rq.nq - kq0) + 2 * PD_CHUNK_T - 1) / (2 * PD_CHUNK_T);
                        float2 acc[K / 2];
#pragma unroll
                        for (int t = 0; t < K / 2; ++t) acc[t] = make_float2(0.0f, 0.0f);
                        if (resid) {
                            if (general_step)
                                pairs_range_x2<K, NP, true, true>(chunk, jss, pi, i, ivalid, js, je,
                                                                  qs_hi, qs_lo, dq_hi, dq_lo, q2,
                                                                  acc, K / (2 * PD_CHUNK_T), rchunk);
                            else
                                pairs_range_x2<K, NP, true, false>(chunk, jss, pi, i, ivalid, js,
                                                                   je, qs_hi, qs_lo, dq_hi, dq_lo,
                                                                   q2, acc, K / (2 * PD_CHUNK_T),
                                                                   rchunk);
                        } else {
                            if (general_step)
                                pairs_range_x2<K, NP, false, true>(chunk, jss, pi, i, ivalid, js,
                                                                   je, qs_hi, qs_lo, dq_hi, dq_lo,
                                                                   q2, acc, nchunk);
                            else
                                pairs_range_x2<K, NP, false, false>(chunk, jss, pi, i, ivalid, js,
                                                                    je, qs_hi, qs_lo, dq_hi, dq_lo,
                                                                    q2, acc, nchunk);
                        }
                        // Warp-reduce and add into this warp's partial sums,
                        // in sub-chunk order (one warp owns them).
                        flush_class<K / 2>(acc, part, lane, first);
                    } else if constexpr (PACKED_W) {
                        const float2 *q2 = reinterpret_cast<const float2 *>(s_qres);
                        const int nchunk =
                            (min(K, rq.nq - kq0) + 2 * PD_CHUNK_T - 1) / (2 * PD_CHUNK_T);
                        float2 acc0[K / 2], acc1[K / 2];
#pragma unroll
                        for (int t = 0; t < K / 2; ++t) {
                            acc0[t] = make_float2(0.0f, 0.0f);
                            acc1[t] = make_float2(0.0f, 0.0f);
                        }
                        if (resid) {
                            if (general_step)
                                pairs_range_x2w<K, NP, true, true>(
                                    chunk, jss, pi, i, ivalid, js, je, qs_hi, qs_lo, dq_hi, dq_lo,
                                    q2, acc0, acc1, K / (2 * PD_CHUNK_T), rchunk);
                            else
                                pairs_range_x2w<K, NP, true, false>(
                                    chunk, jss, pi, i, ivalid, js, je, qs_hi, qs_lo, dq_hi, dq_lo,
                                    q2, acc0, acc1, K / (2 * PD_CHUNK_T), rchunk);
                        } else {
                            if (general_step)
                                pairs_range_x2w<K, NP, false, true>(chunk, jss, pi, i, ivalid, js,
                                                                    je, qs_hi, qs_lo, dq_hi, dq_lo,
                                                                    q2, acc0, acc1, nchunk);
                            else
                                pairs_range_x2w<K, NP, false, false>(
                                    chunk, jss, pi, i, ivalid, js, je, qs_hi, qs_lo, dq_hi, dq_lo,
                                    q2, acc0, acc1, nchunk);
                        }
                        // the four warp sums of each grid point: Σ acc0,
                        // Σ w_i·acc0, Σ acc1, Σ w_i·acc1
                        const float wi = ivalid ? pi.w : 0.0f;
                        flush_weighted<K, false>(acc0, wi, part, K, lane, first);
                        flush_weighted<K, false>(acc1, wi, part + 2 * K, K, lane, first);
                    } else {
                        const float wi = ivalid ? pi.w : 0.0f;
                        float acc[NACC][K];
#pragma unroll
                        for (int a = 0; a < NACC; ++a)
#pragma unroll
                            for (int k = 0; k < K; ++k) acc[a][k] = 0.0f;
                        if (resid) {
                            if (general_step)
                                pairs_range<K, MODE, NP, true, true>(chunk, jss, pi, i, ivalid, js,
                                                                     je, qs_hi, qs_lo, dq_hi,
                                                                     dq_lo, s_qres, acc);
                            else
                                pairs_range<K, MODE, NP, true, false>(chunk, jss, pi, i, ivalid, js,
                                                                      je, qs_hi, qs_lo, dq_hi,
                                                                      dq_lo, s_qres, acc);
                        } else {
                            if (general_step)
                                pairs_range<K, MODE, NP, false, true>(chunk, jss, pi, i, ivalid, js,
                                                                      je, qs_hi, qs_lo, dq_hi,
                                                                      dq_lo, s_qres, acc);
                            else
                                pairs_range<K, MODE, NP, false, false>(chunk, jss, pi, i, ivalid,
                                                                       js, je, qs_hi, qs_lo, dq_hi,
                                                                       dq_lo, s_qres, acc);
                        }
                        // Warp-reduce into this warp's [4][K] partial sums.
#pragma unroll
                        for (int k = 0; k < K; ++k) {
                            const float t0 = warp_sum(acc[0][k]);
                            const float ti = warp_sum(wi * acc[0][k]);
                            const float tj = warp_sum(acc[NACC - 1][k]);
                            const float tij = warp_sum(wi * acc[NACC - 1][k]);
                            if (lane == (k & 31)) {
                                part[k] = (first ? 0.0 : part[k]) + static_cast<double>(t0);
                                part[K + k] = (first ? 0.0 : part[K + k]) + static_cast<double>(ti);
                                part[2 * K + k] =
                                    (first ? 0.0 : part[2 * K + k]) + static_cast<double>(tj);
                                part[3 * K + k] =
                                    (first ? 0.0 : part[3 * K + k]) + static_cast<double>(tij);
                            }
                        }
                    }
                }
            }
            // every read of buffer b done before it is refilled; an expired
            // wait in any thread makes the whole CTA dead
            if (__syncthreads_or(!landed)) {
                if (threadIdx.x == 0) s_dead = 1;
                break;
            }
        }
        __syncthreads();  // every warp's partial sums are complete; s_dead final
        {
            // The job and request fields of the epilogue are loaded again here
            // (an opaque index keeps the compiler from holding them in
            // registers through the steps).
            int jid2 = s_job;
            asm volatile("" : "+r"(jid2));
            const int64_t slot_word = jobs[jid2].slot;
            const PdReqDev *rq2 = reqs + jobs[jid2].req;
            const bool dead = s_dead != 0;
            if (dead && threadIdx.x == 0) {
                // no copy of this CTA may land in shared memory after it
                // moves on: wait (bounded) for the ones still in flight
                for (int b = 0; b < 2; ++b)
                    if (s_inflight & (1u << b))
                        mbar_wait(&s_bar[b], (s_par >> b) & 1u, PD_WAIT_POLLS);
                atomicOr(rq2->status, PD_DEV_WAIT_EXPIRED);
            }
            merge_tile_slots(s_part, NV * K, slot_word, rq2->slots, dead, s_empty && !dead);
        }
        __syncthreads();  // s_qres, s_part, s_job and the tile state are rewritten next
    }
}

// ---------------------------------------------------------------- K2 (FP64)
template <int K, int MODE>
__global__ void __launch_bounds__(PD_THREADS) pd_pairs_fp64(const PdJob *__restrict__ jobs,
                                                            const int *__restrict__ n_jobs_ptr,
                                                            const PdReqDev *__restrict__ reqs,
                                                            int *__restrict__ counter,
                                                            int plan_frames) {
    chain_enter();
    constexpr int NACC = (MODE == PD_MODE_WEIGHTED) ? 2 : 1;
    constexpr int NV = (MODE == PD_MODE_WEIGHTED) ? 4 : 1;
    __shared__ int s_job;
    __shared__ double s_q[K];
    __shared__ double s_part[PD_WARPS * NV * K];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int n_jobs = *n_jobs_ptr;
    double *part = s_part + warp * NV * K;
    if (plan_frames > 0 && !plan_sums_pairs(reqs[0], plan_frames)) return;
    for (bool first = true;; first = false) {
        if (threadIdx.x == 0) s_job = next_pair_job(jobs, n_jobs, reqs, counter, first);
        __syncthreads();
        const int jid = s_job;
        if (jid >= n_jobs) break;
        const PdJob jb = jobs[jid];
        const PdReqDev rq = reqs[jb.req];
        if (threadIdx.x < K) {
            const int kq = jb.qb * K + threadIdx.x;
            s_q[threadIdx.x] = kq < rq.nq ? rq.qv[kq] : 0.0;
        }
        __syncthreads();
        const double4 *__restrict__ at = rq.atoms64 + static_cast<size_t>(jb.frame) * rq.n_pad;
        const int i = jb.i0 + threadIdx.x;
        const double4 pi = at[i];
        const bool ivalid = lane < rq.gvalid[(jb.i0 >> 5) + warp];

        double acc[NACC][K];
#pragma unroll
        for (int a = 0; a < NACC; ++a)
#pragma unroll
            for (int k = 0; k < K; ++k) acc[a][k] = 0.0;

        for (int j = jb.j0; j < jb.j1; ++j) {
            const double4 pj = at[j];
            const double dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            double r2 = dx * dx + dy * dy + dz * dz;
            r2 = fmax(r2, 1e-24);
            const double r = sqrt(r2);
            const double w0 = (ivalid && j > i) ? 1.0 / r : 0.0;
            const double w1 = w0 * pj.w;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const double s = sin(s_q[k] * r);
                acc[0][k] = fma(w0, s, acc[0][k]);
                if (MODE == PD_MODE_WEIGHTED) acc[NACC - 1][k] = fma(w1, s, acc[NACC - 1][k]);
            }
        }

        const double wi = ivalid ? pi.w : 0.0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const double t0 = warp_sum(acc[0][k]);
            if (MODE == PD_MODE_CLASS) {
                if (lane == (k & 31)) part[k] = t0;
            } else {
                const double ti = warp_sum(wi * acc[0][k]);
                const double tj = warp_sum(acc[NACC - 1][k]);
                const double tij = warp_sum(wi * acc[NACC - 1][k]);
                if (lane == (k & 31)) {
                    part[k] = t0;
                    part[K + k] = ti;
                    part[2 * K + k] = tj;
                    part[3 * K + k] = tij;
                }
            }
        }
        __syncthreads();  // every warp's partial sums are complete
        merge_tile_slots(s_part, NV * K, jb.slot, rq.slots, false, false);
        __syncthreads();  // s_q, s_part and s_job are rewritten by the next tile
    }
}

// ------------------------------------------------------- pack and centroid
// Per-frame centroid of the input positions, FP64: every block adds a fixed
// run of atoms in a fixed tree and the frame's last block adds the blocks'
// sums in block order, so the centroid does not depend on which block ends
// last. One block per frame of up to PD_CENT_RUN atoms, more for larger frames (a
// single block took 150 µs to read 100,000 atoms twice; now 8 µs).
constexpr int PD_CENT_THREADS = 256;
constexpr int64_t PD_CENT_RUN = 2048;

__global__ void __launch_bounds__(PD_CENT_THREADS)
    pd_centroid(const double *__restrict__ xyz, int64_t n_atoms, int32_t n_blk,
                double *__restrict__ part, unsigned int *__restrict__ done,
                double *__restrict__ centroid, int32_t *__restrict__ status) {
    chain_enter();
    __shared__ double red[3][PD_CENT_THREADS];
    __shared__ bool s_last;
    const int f = blockIdx.x / n_blk, b = blockIdx.x % n_blk;
    const double *p = xyz + static_cast<size_t>(f) * n_atoms * 3;
    if (blockIdx.x == 0 && threadIdx.x == 0 && status) *status = 0;
    const int64_t i0 = n_atoms * b / n_blk, i1 = n_atoms * (b + 1) / n_blk;
    double sx = 0, sy = 0, sz = 0;
#pragma unroll 4
    for (int64_t i = i0 + threadIdx.x; i < i1; i += PD_CENT_THREADS) {
        sx += p[3 * i];
        sy += p[3 * i + 1];
        sz += p[3 * i + 2];
    }
    red[0][threadIdx.x] = sx;
    red[1][threadIdx.x] = sy;
    red[2][threadIdx.x] = sz;
    __syncthreads();
    for (int s = PD_CENT_THREADS / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            red[0][threadIdx.x] += red[0][threadIdx.x + s];
            red[1][threadIdx.x] += red[1][threadIdx.x + s];
            red[2][threadIdx.x] += red[2][threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        for (int a = 0; a < 3; ++a) part[3 * blockIdx.x + a] = red[a][0];
        __threadfence();
        s_last = atomicAdd(&done[f], 1u) == static_cast<unsigned>(n_blk - 1);
    }
    __syncthreads();
    if (s_last && threadIdx.x < 96) {  // a warp per axis, lanes added in a fixed tree
        __threadfence();
        const int ax = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const double *q = part + 3 * static_cast<size_t>(f) * n_blk + ax;
        double s = 0;
        for (int k = lane; k < n_blk; k += 32) s += __ldcg(q + 3 * k);
        s = warp_sum(s);
        if (lane == 0) centroid[3 * f + ax] = s / static_cast<double>(n_atoms);
    }
}

// Gather positions into the class-sorted, padded layout, centred per frame.
// The largest distance from the centroid is collected on the way, and the
// frame's last block turns it into the frame's constants (PdFrameDev): which form
// its pairs are summed in, the expansion's size and the direction table.
//
// The rule counts FP32 lane operations: a pair costs about 44 for its sequences and 12
// for its share of the flushes (in each moment block) and 1.5 per moment, an atom in
// one direction 14 (44 more for each later block) and 1.25 per moment, a direction
// also n_cls·M terms per node in FP64, and the class pairs' products there. The costs of
// the tiles, of the pairs at the grid points and as moments, which decide between those
// two, of the class pairs' products and of the chains are the plan's (set_reduction).
// Whole solves on both sides (vacuum, µs): FP32, moments of the pairs / directions,
// q_max 0.5, 200 / 300 / 600 / 1,200 atoms 68/65, 80/66, 83/70, 90/84, q_max 1.0 71/75,
// 84/72, 89/82, 97/89, elongated 2.5 : 1, q_max 1.0, 300 / 500 / 800 atoms 73/79, 82/92, 101/122; FP64, grid points / directions, 100 points, 100 / 300 / 600 atoms
// 233/59, 559/74, 983/75.
constexpr int PD_PACK_THREADS = 256;

// Nodes and weights of the 2h-point Gauss–Legendre rules, upper half
// (x > 0, ascending), h = 1 … PD_GL_MAX: rule h at h·(h − 1)/2. The weights of
// a half add up to 1. Filled once per device (prepare_direction_rules).
constexpr int PD_GL_MAX = 128;
__device__ double2 pd_gl_rules[PD_GL_MAX * (PD_GL_MAX + 1) / 2];

__device__ __forceinline__ int ring_points(double z_sin, bool fp64) {
    return max(4, static_cast<int>(direction_order(z_sin, fp64)) + 1);
}

// The direction of length sqrt(len2) in FP32: of the eight roundings of its components
// the one whose length is nearest. Each to nearest would stretch all distances along
// the direction by up to 6e-8 — and a ring's directions share their z —, which the
// moments, expanded for the exact length, cannot tell from another structure; a
// turn by as much is harmless. (10,000-atom sphere against FP64: 2-norm error 5.4e-9 ->
// 7.6e-10, largest error of a profile point 6.8e-7 -> 1.5e-7.)
__device__ __forceinline__ double4 round_direction(double4 d, double len2) {
    const double lo[3] = {__double2float_rd(d.x), __double2float_rd(d.y), __double2float_rd(d.z)};
    const double hi[3] = {__double2float_ru(d.x), __double2float_ru(d.y), __double2float_ru(d.z)};
    double best = 1e300;
    double4 r = d;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const double x = (k & 1) ? hi[0] : lo[0], y = (k & 2) ? hi[1] : lo[1],
                     z = (k & 4) ? hi[2] : lo[2];
        const double e = fabs(fma(x, x, fma(y, y, fma(z, z, -len2))));
        if (e < best) {
            best = e;
            r = make_double4(x, y, z, d.w);
        }
    }
    return r;
}

// A frame's constants (PdFrameDev) from its radius: which form its pairs are summed
// in, the expansion's size, and the direction table, whose entries the n_part blocks
// share. T threads, all of each block.
template <int T>
__device__ __forceinline__ void frame_constants(double radius, const PdMomentRule &rule, int f,
                                                int part, int n_part,
                                                PdFrameDev *__restrict__ frames,
                                                double4 *__restrict__ dirs,
                                                double2 *__restrict__ node_tab) {
    static_assert(T >= PD_GL_MAX, "a thread per ring");
    __shared__ int s_off[PD_GL_MAX + 1];  // first direction of each ring
    const bool fp64 = rule.fp64 != 0;
    PdFrameDev fr{};
    fr.radius = radius;
    // d follows the FP32 value of 1/d² that the pairs are scaled with: rounding
    // 1/d² alone would stretch every distance by the same 1 + 3e-8
    fr.d = fmax(2.0 * PD_MOM_STRETCH * radius, 1e-6);
    fr.inv_d2 = static_cast<double>(static_cast<float>(1.0 / (fr.d * fr.d)));
    fr.d = 1.0 / sqrt(fr.inv_d2);
    fr.r1 = fmax(PD_MOM_STRETCH * radius, 1e-6);
    double pair_cost = rule.grid_dir_cost;
    if (rule.block > 0) {
        const int m8 = (moments_needed(rule.qmax * fr.d, false) + 7) & ~7;
        const int blocks = (m8 + rule.block - 1) / rule.block;
        if (m8 <= rule.max_moments && blocks <= rule.nqb &&
            rule.mom_cost * m8 + rule.mom_block_cost * blocks < rule.grid_cost) {
            fr.n_mom = m8;
            fr.n_mblk = blocks;
            fr.n_parts = rule.nqb / blocks;
            pair_cost = 56.0 * blocks + 1.5 * m8;
        }
    }
    pair_cost *= rule.n_tile_pairs;
    pair_cost += rule.tile_cost + (fr.n_mom > 0 ? rule.mom_latency : rule.grid_latency);
    // ---- directions: 2h Gauss rings (upper half: h), enough points on each
    if (rule.dir_cap == 0) {
        if (part == 0 && threadIdx.x == 0) frames[f] = fr;
        return;
    }
    const double z = 2.0 * radius * rule.qmax;
    const double order = direction_order(z, fp64);
    const int h = order < 4.0 * PD_GL_MAX - 4.0 ? static_cast<int>(order * 0.25) + 1 : 0;
    const double2 *gl = pd_gl_rules + h * (h - 1) / 2;
    if (threadIdx.x < h) {
        const double x = gl[threadIdx.x].x;
        s_off[threadIdx.x + 1] = ring_points(z * sqrt(1.0 - x * x), fp64);
    }
    __syncthreads();
    for (int o = 1; o < h; o <<= 1) {  // inclusive scan of s_off[1 .. h]
        const int k = threadIdx.x + 1;
        const int v = (k <= h && k > o) ? s_off[k - o] : 0;
        __syncthreads();
        if (k <= h) s_off[k] += v;
        __syncthreads();
    }
    if (threadIdx.x == 0) s_off[0] = 0;
    __syncthreads();
    const int S = h > 0 ? s_off[h] : 0;
    const int groups = (S + 31) / 32;
    const int mine = rule.rank < groups ? (groups - rule.rank + rule.world - 1) / rule.world : 0;
    const double mo = direction_order(fr.r1 * rule.qmax, fp64);
    const int m8 = mo < 1e6 ? ((static_cast<int>(mo) + 8) & ~7) : 1000000;
    const int ablk = (m8 + rule.dir_block - 1) / rule.dir_block;
    const int nodes = fp64 ? rule.nq : moments_needed(2.0 * fr.r1 * rule.qmax, true);
    const double dir_cost =
        static_cast<double>(S) * ((static_cast<double>(rule.n_atoms) +
                                   (fp64 ? PD_DIR_CHUNK64 * rule.n_chunk : 0.0)) * rule.nv2 *
                                      (44.0 * ablk - 30.0 + 1.25 * m8) +
                                  4.0 * rule.n_cls * m8 * nodes) +
        rule.dir_pair_cost * fmax(static_cast<double>(S) * nodes, PD_DIR_LEAST);
    const bool use = S > 0 && groups * 32 <= rule.dir_cap && mine > 0 &&
                     (groups + rule.world - 1) / rule.world <= rule.grp_cap &&
                     m8 <= rule.amp_cap && nodes <= rule.node_cap &&
                     static_cast<int64_t>(rule.n_chunk) * rule.nv2 *
                             ((groups + rule.world - 1) / rule.world) * m8 * 32 <= rule.slot_cap &&
                     groups >= rule.world && (rule.dir_only || dir_cost < pair_cost);
    if (use) {
        fr.n_grp = mine;
        fr.n_amp = m8;
        fr.n_node = nodes;
        // Chebyshev nodes of the q range: y_k and the barycentric weight
        for (int k = part * T + threadIdx.x; k < nodes && !fp64; k += n_part * T) {
            double sn, cs;
            sincospi((2 * k + 1) / (2.0 * nodes), &sn, &cs);
            node_tab[static_cast<int64_t>(f) * rule.node_cap + k] =
                make_double2(cs, (k & 1) ? -sn : sn);
        }
        const double sc = 0.5 / fr.r1;
        double4 *o = dirs + static_cast<int64_t>(f) * rule.dir_cap;
        for (int s = part * T + threadIdx.x; s < groups * 32; s += n_part * T) {
            double4 d = make_double4(0.0, 0.0, 0.0, 0.0);
            if (s < S) {
                int lo = 0, hi = h;  // ring with s_off[lo] <= s < s_off[lo + 1]
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (s_off[mid] <= s) lo = mid; else hi = mid;
                }
                const double2 nw = gl[lo];
                const int n = s_off[lo + 1] - s_off[lo];
                const double st = sqrt(1.0 - nw.x * nw.x) * sc;
                double sn, cs;
                sincospi(2.0 * (s - s_off[lo]) / n, &sn, &cs);
                d = make_double4(st * cs, st * sn, nw.x * sc, nw.y / n);
                if (!fp64) d = round_direction(d, sc * sc);
            }
            o[s] = d;
        }
    }
    if (part == 0 && threadIdx.x == 0) frames[f] = fr;
}

__global__ void __launch_bounds__(PD_PACK_THREADS)
    pd_pack(const double *__restrict__ xyz, const double *__restrict__ weights,
            const int32_t *__restrict__ perm, const double *__restrict__ centroid,
            int64_t n_atoms, int32_t n_pad, int32_t n_blk, float4 *__restrict__ out32,
            double4 *__restrict__ out64, PdMomentRule rule, unsigned long long *__restrict__ rad2,
            unsigned int *__restrict__ done, PdFrameDev *__restrict__ frames,
            double4 *__restrict__ dirs, double2 *__restrict__ node_tab) {
    chain_enter();
    __shared__ double s_max[PD_PACK_THREADS / 32];
    __shared__ bool s_last;
    __shared__ double s_radius;
    const int f = blockIdx.x / n_blk, b = blockIdx.x % n_blk;
    const int p = b * PD_PACK_THREADS + threadIdx.x;
    double r2 = 0.0;
    if (p < n_pad) {
        const int src = perm[p];
        double x = 0, y = 0, z = 0, w = 0;
        if (src >= 0) {
            const double *s = xyz + (static_cast<size_t>(f) * n_atoms + src) * 3;
            x = s[0] - centroid[3 * f];
            y = s[1] - centroid[3 * f + 1];
            z = s[2] - centroid[3 * f + 2];
            w = weights ? weights[src] : 0.0;
            r2 = x * x + y * y + z * z;
        }
        const size_t t = static_cast<size_t>(f) * n_pad + p;
        if (out32) out32[t] = make_float4(static_cast<float>(x), static_cast<float>(y),
                                          static_cast<float>(z), static_cast<float>(w));
        if (out64) out64[t] = make_double4(x, y, z, w);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r2 = fmax(r2, __shfl_xor_sync(0xffffffffu, r2, o));
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = r2;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < PD_PACK_THREADS / 32; ++k) r2 = fmax(r2, s_max[k]);
        // non-negative doubles order as their bit patterns; the maximum is exact
        atomicMax(&rad2[f], static_cast<unsigned long long>(__double_as_longlong(r2)));
        __threadfence();
        s_last = atomicAdd(&done[f], 1u) == static_cast<unsigned>(n_blk - 1);
        if (s_last) {
            __threadfence();
            s_radius = sqrt(__longlong_as_double(
                static_cast<long long>(atomicMax(&rad2[f], 0ull))));
        }
    }
    __syncthreads();
    if (!s_last) return;

    frame_constants<PD_PACK_THREADS>(s_radius, rule, f, 0, 1, frames, dirs, node_tab);
}

// Centroid, pack and constants of a frame in one kernel: a cluster of PD_FRAME_CTAS
// blocks per frame, whose partial sums and maxima meet in distributed shared memory. For
// frames of up to PD_FRAME_MAX padded atoms, where the two kernels are latency (8
// SMs read the frame here): 300 atoms 15.7 -> 7.5 µs, 3,000 atoms 18.3 -> 12.0 µs;
// whole executions at the line, 16,000 atoms (one kernel) 116 µs, 17,000 (two) 126 µs.
constexpr int PD_FRAME_CTAS = 8, PD_FRAME_THREADS = 512;
constexpr int32_t PD_FRAME_MAX = 16384;

__global__ void __cluster_dims__(PD_FRAME_CTAS, 1, 1) __launch_bounds__(PD_FRAME_THREADS)
    pd_pack_frames(const double *__restrict__ xyz, const double *__restrict__ weights,
                   const int32_t *__restrict__ perm, int32_t n_atoms, int32_t n_pad,
                   float4 *__restrict__ out32, double4 *__restrict__ out64, PdMomentRule rule,
                   PdFrameDev *__restrict__ frames, double4 *__restrict__ dirs,
                   double2 *__restrict__ node_tab, int32_t *__restrict__ status) {
    chain_enter();
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ double s_red[PD_FRAME_THREADS / 32][3];
    __shared__ double s_mine[4];  // this block's sums and maximum, read by the cluster
    constexpr int STEP = PD_FRAME_CTAS * PD_FRAME_THREADS;
    const int f = blockIdx.x / PD_FRAME_CTAS, rank = blockIdx.x % PD_FRAME_CTAS;
    const int first = rank * PD_FRAME_THREADS + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double *p = xyz + static_cast<size_t>(f) * n_atoms * 3;
    if (blockIdx.x == 0 && threadIdx.x == 0 && status) *status = 0;
    double sum[3] = {0.0, 0.0, 0.0};
#pragma unroll 4
    for (int i = first; i < n_atoms; i += STEP)
#pragma unroll
        for (int a = 0; a < 3; ++a) sum[a] += p[3 * static_cast<size_t>(i) + a];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        sum[a] = warp_sum(sum[a]);
        if (lane == 0) s_red[warp][a] = sum[a];
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double s = 0.0;
        for (int w = 0; w < PD_FRAME_THREADS / 32; ++w) s += s_red[w][threadIdx.x];
        s_mine[threadIdx.x] = s;
    }
    cluster.sync();
    double c[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int b = 0; b < PD_FRAME_CTAS; ++b) {
        const double *o = cluster.map_shared_rank(s_mine, b);
#pragma unroll
        for (int a = 0; a < 3; ++a) c[a] += o[a];
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) c[a] /= static_cast<double>(n_atoms);
    double r2 = 0.0;
#pragma unroll 2
    for (int k = first; k < n_pad; k += STEP) {
        const int src = perm[k];
        double x = 0, y = 0, z = 0, w = 0;
        if (src >= 0) {
            const double *s = p + static_cast<size_t>(src) * 3;
            x = s[0] - c[0];
            y = s[1] - c[1];
            z = s[2] - c[2];
            w = weights ? weights[src] : 0.0;
            r2 = fmax(r2, x * x + y * y + z * z);
        }
        const size_t t = static_cast<size_t>(f) * n_pad + k;
        if (out32) out32[t] = make_float4(static_cast<float>(x), static_cast<float>(y),
                                          static_cast<float>(z), static_cast<float>(w));
        if (out64) out64[t] = make_double4(x, y, z, w);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r2 = fmax(r2, __shfl_xor_sync(0xffffffffu, r2, o));
    if (lane == 0) s_red[warp][0] = r2;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < PD_FRAME_THREADS / 32; ++w) r2 = fmax(r2, s_red[w][0]);
        s_mine[3] = r2;
    }
    cluster.sync();
    r2 = 0.0;
#pragma unroll
    for (int b = 0; b < PD_FRAME_CTAS; ++b) r2 = fmax(r2, cluster.map_shared_rank(s_mine, b)[3]);
    cluster.sync();  // the blocks' shared memory is read
    frame_constants<PD_FRAME_THREADS>(sqrt(r2), rule, f, rank, PD_FRAME_CTAS, frames, dirs,
                                      node_tab);
}

// ------------------------------------------------------------ reductions
// Sums the slots of every (frame, class pair) in a fixed order. A block owns
// 128 values (grid points, or moments) of one class pair: its groups of 128
// threads, and the n_chunk blocks along y, each add a contiguous run of the
// slot list, and the runs' sums are added in run order (by the block that ends
// last where there are several).
//  - grid points: the slots hold Σ sin(q r)/r; the sums are divided by q,
//    and the residual form and q = 0 take their exact pair sums;
//  - moments: value e of block mb collects the lists of all the parts.
// red is [frame][pair][nv][width].
constexpr int PD_RED_GROUPS = 4;
constexpr int PD_RED_THREADS = 128 * PD_RED_GROUPS;

template <int NV>
__device__ __forceinline__ void sum_slots(const double *__restrict__ slots,
                                          const int64_t *__restrict__ lidx, int64_t e0, int64_t e1,
                                          int64_t fbase, int64_t stride, int K, int kk,
                                          double (&s)[NV]) {
    int64_t e = e0;
    for (; e + 8 <= e1; e += 8) {  // eight slots in flight, added in list order
        double x[8][NV];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const double *sl = slots + (fbase + lidx[e + u]) * stride + kk;
#pragma unroll
            for (int v = 0; v < NV; ++v) x[u][v] = sl[v * K];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
            for (int v = 0; v < NV; ++v) s[v] += x[u][v];
    }
    for (; e < e1; ++e) {
        const double *sl = slots + (fbase + lidx[e]) * stride + kk;
#pragma unroll
        for (int v = 0; v < NV; ++v) s[v] += sl[v * K];
    }
}

template <int NV>
__global__ void __launch_bounds__(PD_RED_THREADS)
    pd_reduce_pairs(const double *__restrict__ slots, const int64_t *__restrict__ lptr,
                    const int64_t *__restrict__ lidx, const PdPairDev *__restrict__ pairs,
                    const double *__restrict__ qv, const PdFrameDev *__restrict__ frames,
                    PdReduceShape sh, int32_t residual_form, int32_t add_exact,
                    double *__restrict__ chunk_sums, unsigned int *__restrict__ done,
                    double *__restrict__ red) {
    chain_enter();
    __shared__ double s_run[PD_RED_GROUPS][NV][128];
    __shared__ bool s_last;
    const int z = blockIdx.x % sh.n_z;
    const int p = blockIdx.x / sh.n_z % sh.n_pairs;
    const int f = blockIdx.x / sh.n_z / sh.n_pairs;
    const int tl = threadIdx.x & 127, grp = threadIdx.x >> 7;
    const int k = z * 128 + tl;
    const PdFrameDev fr = frames[f];
    const bool moments = fr.n_mom > 0;
    if (fr.n_grp > 0) return;  // direction form
    if (z * 128 >= (moments ? fr.n_mom : sh.nq)) return;
    const int64_t fbase = static_cast<int64_t>(f) * sh.slots_per_frame;
    const int64_t stride = static_cast<int64_t>(NV) * sh.K;
    const int run = blockIdx.y * PD_RED_GROUPS + grp, n_runs = gridDim.y * PD_RED_GROUPS;
    double s[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) s[v] = 0.0;
    const double qval = (!moments && k < sh.nq) ? qv[k] : 0.0;
    if (moments) {
        if (k < fr.n_mom) {
            const int mb = k / sh.block, kk = k - mb * sh.block;
            for (int part = 0; part < fr.n_parts; ++part) {
                const int64_t *lp = lptr + p * sh.nqb + part * fr.n_mblk + mb;
                const int64_t l0 = lp[0], len = lp[1] - l0;
                sum_slots<NV>(slots, lidx, l0 + len * run / n_runs, l0 + len * (run + 1) / n_runs,
                              fbase, stride, sh.K, kk, s);
            }
        }
    } else if (qval > 0.0) {
        const int64_t *lp = lptr + p * sh.nqb + k / sh.K;
        const int64_t l0 = lp[0], len = lp[1] - l0;
        sum_slots<NV>(slots, lidx, l0 + len * run / n_runs, l0 + len * (run + 1) / n_runs, fbase,
                      stride, sh.K, k % sh.K, s);
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) s_run[grp][v][tl] = s[v];
    __syncthreads();
    if (grp == 0) {
#pragma unroll
        for (int v = 0; v < NV; ++v)
#pragma unroll
            for (int g = 1; g < PD_RED_GROUPS; ++g) s[v] += s_run[g][v][tl];
    }
    if (gridDim.y > 1) {
        // [block][chunk][nv][128]
        double *cs = chunk_sums + static_cast<size_t>(blockIdx.x) * gridDim.y * NV * 128;
        if (grp == 0) {
#pragma unroll
            for (int v = 0; v < NV; ++v) cs[(blockIdx.y * NV + v) * 128 + tl] = s[v];
            __threadfence();
        }
        __syncthreads();
        if (threadIdx.x == 0)
            s_last = atomicAdd(&done[blockIdx.x], 1u) == gridDim.y - 1;
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        if (grp == 0) {
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const volatile double *c = cs + v * 128 + tl;
                double t = 0.0;
                for (unsigned y = 0; y < gridDim.y; ++y) t += c[y * NV * 128];
                s[v] = t;
            }
        }
    }
    if (grp != 0 || k >= sh.width) return;
    if (!moments) {
        if (k >= sh.nq) return;
        if (qval > 0.0) {
#pragma unroll
            for (int v = 0; v < NV; ++v) s[v] /= qval;
            if (add_exact && residual_form && residual_q(qval, fr.radius))
#pragma unroll
                for (int v = 0; v < NV; ++v) s[v] += pairs[p].q0[v];
        } else {
#pragma unroll
            for (int v = 0; v < NV; ++v) s[v] = add_exact ? pairs[p].q0[v] : 0.0;
        }
    }
    double *o = red + (static_cast<int64_t>(f) * sh.n_pairs + p) * NV * sh.width + k;
#pragma unroll
    for (int v = 0; v < NV; ++v) o[static_cast<int64_t>(v) * sh.width] = s[v];
}

// Direction form: class-pair sums at Chebyshev nodes of the q range, or at the grid
// points.
//
// S_ab(q) = Σ sinc(q r) is an even entire function of q whose expansion in
// T_2k(q/q_max) ends, like the moments, at k ≈ q_max·d/2 + …: its values at that many
// nodes q_k = q_max·cos((2k+1)π/4M) give every grid point by interpolation (pd_profiles), so
// the amplitudes are formed at 30 to 120 nodes instead of 200 to 1,000 grid
// points. The interpolation mixes values from N² to N: it keeps 1e-16 of N², which at
// a deep minimum is up to 1e-11 of the point, far below the FP32 moments' rounding.
// The FP64 form takes the grid points themselves (qv; largest error of a point, 30,000
// atoms to q = 2: 8.7e-12 -> 4e-15; 6,001 atoms, 301 points: 8e-15 -> 5e-15 for 234 ->
// 296 us). A block takes 32 directions and PD_DNODE_T nodes (fewer where many
// classes share its memory): E_c = Σ_n g_n(q_k r1)·m_n, g_n = i^n (2 − δ_n0) J_n, of every class in
// FP64 — the sums of the class's chunks added in chunk order, the zeroth
// moment the exact atom count or weight sum — then Σ w·Re(E_a E_b*) over the directions
// of every class pair. The frame's last block of these nodes adds the groups in
// group order and takes the i = j terms out of the self sums.
//
// Bound: latency — a chain of loads, a Bessel recurrence, two short FP64
// contractions and the last block's sum. 512 threads: 256 took 20.0 µs per frame
// more at 20,000 atoms (whole execution 425 against 403 µs), the same at 3,000.
constexpr int PD_DNODE_T = 16;
constexpr int PD_DSUM_THREADS = 512;
constexpr int PD_DSUM_WARPS = PD_DSUM_THREADS / 32;

// (2 − δ_n0)·J_n(y)·(sign of i^n) for n < n_mom, unnormalised, into g[n·stride];
// returns the factor that normalises them (J_0 + 2ΣJ_2k = 1, Miller's recurrence).
__device__ double direction_coefficients(double y, int n_mom, double *__restrict__ g, int stride) {
    if (!(y > 1e-8)) {
        for (int n = 0; n < n_mom; ++n) g[n * stride] = n == 0 ? 1.0 : 0.0;
        return 1.0;
    }
    const double ty = 2.0 / y;
    const int top = static_cast<int>(bessel_order(y, 16.0, 10.0)) | 1;
    for (int n = top + 1; n < n_mom; ++n) g[n * stride] = 0.0;
    double hi = 0.0, cur = 1e-200, even = 0.0;
    for (int n = top; n > 0; --n) {  // cur = J_n
        if (n < n_mom) g[n * stride] = (n & 2) ? -2.0 * cur : 2.0 * cur;
        if (!(n & 1)) even += cur;
        const double lower = fma(n * ty, cur, -hi);
        hi = cur;
        cur = lower;
    }
    g[0] = cur;
    return 1.0 / fma(2.0, even, cur);
}

// The coefficients of the first block's product sums from those of its moments (n <
// lim, a multiple of 8): m_8j+t = 2·P_{j,t} − m_8j−t, so a coefficient passes on
// with the other sign from n = 8j + t to 8j − t, a chain of 8(j − 1) + (8 − t) next:
// seven chains, one for a thread (t: the chain's element of the last eight).
__device__ void direction_fold(double *__restrict__ g, int lim, int t, int stride) {
    double prev = 0.0;
#pragma unroll 4
    for (int j = lim / 8 - 1; j >= 0; --j) {
        double &c = g[(8 * j + t) * stride];
        const double v = c - prev;
        c = j > 0 ? 2.0 * v : v;
        prev = v;
        t = 8 - t;
    }
}

// Node k of n on the q range [0, qmax]: q = qmax·cos((2k+1)π/4n).
__device__ __forceinline__ double direction_node(int k, int n, double qmax) {
    return qmax * cospi((2 * k + 1) / (4.0 * n));
}

template <int NV2>
__global__ void __launch_bounds__(PD_DSUM_THREADS)
    pd_direction_sums(const double *__restrict__ slots, const double4 *__restrict__ dirs,
                      const PdFrameDev *__restrict__ frames, PdAmpShape sh, double qmax,
                      const double *__restrict__ qv,
                      const PdClassDev *__restrict__ cls, const PdPairDev *__restrict__ pairs,
                      int32_t n_pairs, const int32_t *__restrict__ cls_ptr,
                      const int32_t *__restrict__ cls_chunk, int32_t width,
                      int32_t add_exact, double *__restrict__ part, unsigned int *__restrict__ done,
                      double *__restrict__ red) {
    chain_enter();
    extern __shared__ double s_dyn[];
    __shared__ double s_scale[PD_DNODE_T], s_w[32];
    __shared__ bool s_last;
    const int f = blockIdx.y;
    const PdFrameDev fr = frames[f];
    const int NT = sh.node_tile;
    const int n_nt = (sh.node_cap + NT - 1) / NT;
    const int tile = blockIdx.x % n_nt, grp = blockIdx.x / n_nt;
    if (grp >= fr.n_grp || tile * NT >= fr.n_node) return;
    const int M = fr.n_amp, nn = min(NT, fr.n_node - tile * NT);
    const int ncv = sh.n_cls * NV2;             // class sums (plain, weighted)
    double *s_g = s_dyn;                        // [M][NT]
    double *s_e = s_g + M * NT;                 // [n_cls][NV2][NT][2][32]
    double *s_m = s_e + ncv * NT * 64;          // [batch][M][32]
    const int batch = min(ncv, (sh.sum_smem - M * NT - ncv * NT * 64) / (M * 32));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int LOADERS = PD_DSUM_WARPS - 1;
    if (warp == LOADERS) {  // one warp: the coefficients, while the others load
        if (lane < nn) {
            const int k = tile * NT + lane;
            const double q = qv ? qv[k] : direction_node(k, fr.n_node, qmax);
            s_scale[lane] = direction_coefficients(q * fr.r1, M, s_g + lane, NT);
        }
        __syncwarp();
        for (int k = lane; k < 7 * nn; k += 32)
            direction_fold(s_g + k % nn, min(M, sh.dir_block), 1 + k / nn, NT);
        s_w[lane] = dirs[static_cast<int64_t>(f) * sh.dir_cap +
                         (static_cast<int64_t>(grp) * sh.world + sh.rank) * 32 + lane].w;
    }
    const double *sl = slots + static_cast<int64_t>(f) * sh.slot_cap;
    for (int c0 = 0; c0 < ncv; c0 += batch) {  // as many classes at once as fit
        const int nb = min(batch, ncv - c0);
        if (c0) __syncthreads();  // the previous classes' moments are read
        // (class, 8 moments) per warp and step: rows of 32 directions, those of four
        // chunks in flight
        const int n8 = M / 8;
        for (int k = warp; k < nb * n8 && warp < LOADERS; k += LOADERS) {
            const int cb = k / n8, r0 = (k - cb * n8) * 8;
            const int c = (c0 + cb) / NV2, v = (c0 + cb) % NV2;
            const int e0 = cls_ptr[c], n = cls_ptr[c + 1] - e0;
            const double *src = sl + direction_slot(0, v, grp, NV2, fr) + r0 * 32 + lane;
            const int64_t step = static_cast<int64_t>(NV2) * fr.n_grp * M * 32;  // of a chunk
            double m[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) m[u] = 0.0;
#pragma unroll 4
            for (int e = 0; e < n; ++e) {
                const double *row = src + cls_chunk[e0 + e] * step;
#pragma unroll
                for (int u = 0; u < 8; ++u) m[u] += __ldg(row + u * 32);
            }
            if (r0 == 0) m[0] = v ? cls[c].w1 : cls[c].n;
            double *dst = s_m + (cb * M + r0) * 32 + lane;
#pragma unroll
            for (int u = 0; u < 8; ++u) dst[u * 32] = m[u];
        }
        __syncthreads();
        // (class, four nodes) per warp and step
        const int n4 = (nn + 3) / 4;
        for (int k = warp; k < nb * n4; k += PD_DSUM_WARPS) {
            const int cb = k / n4, t0 = (k - cb * n4) * 4;
            const double *mm = s_m + cb * (M * 32) + lane;
            const double *g = s_g + t0;
            double er[4] = {0, 0, 0, 0}, ei[4] = {0, 0, 0, 0};
#pragma unroll 2
            for (int n = 0; n < M; n += 2) {  // M is a multiple of 8
                const double m0 = mm[n * 32], m1 = mm[(n + 1) * 32];
#pragma unroll
                for (int t = 0; t < 4; ++t) {  // NT is a multiple of 4: rows past nn are unused
                    er[t] = fma(g[n * NT + t], m0, er[t]);
                    ei[t] = fma(g[(n + 1) * NT + t], m1, ei[t]);
                }
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                if (t0 + t >= nn) break;
                double *o = s_e + ((c0 + cb) * NT + t0 + t) * 64 + lane;
                o[0] = er[t] * s_scale[t0 + t];
                o[32] = ei[t] * s_scale[t0 + t];
            }
        }
    }
    __syncthreads();
    constexpr int NV = NV2 == 2 ? 4 : 1;
    // [frame][group][pair][nv][node]
    const int64_t row = static_cast<int64_t>(n_pairs) * NV * sh.node_cap;
    double *pt = part + (static_cast<int64_t>(f) * sh.grp_cap + grp) * row;
    // a thread per (pair, node); each starts at a direction of its own, so that
    // the 32 reads of a warp touch all banks (tiles of 4, 8 or 16 nodes: the
    // pair's bits reversed). The start depends on the pair and the node alone: the
    // order of a sum, and so its rounding, does not follow the tile size.
    for (int k = threadIdx.x; k < n_pairs * nn; k += PD_DSUM_THREADS) {
        const int p = k / nn, t = k - p * nn;
        const int a = pairs[p].a, b = pairs[p].b;
        const double *Ea = s_e + (a * NV2 * NT + t) * 64, *Eb = s_e + (b * NV2 * NT + t) * 64;
        const int rot = tile * NT + t + static_cast<int>(__brev(p) >> 27);
        double x[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) x[v] = 0.0;
#pragma unroll 4
        for (int i = 0; i < 32; ++i) {
            const int d = (i + rot) & 31;
            const double w = s_w[d];
            const double ar = w * Ea[d], ai = w * Ea[32 + d], br = Eb[d], bi = Eb[32 + d];
            x[0] = fma(ar, br, fma(ai, bi, x[0]));
            if constexpr (NV == 4) {  // weighted amplitudes
                const double *Fa = Ea + NT * 64, *Fb = Eb + NT * 64;
                const double fr_ = w * Fa[d], fi_ = w * Fa[32 + d], gr = Fb[d], gi = Fb[32 + d];
                x[1] = fma(fr_, br, fma(fi_, bi, x[1]));
                x[2] = fma(ar, gr, fma(ai, gi, x[2]));
                x[3] = fma(fr_, gr, fma(fi_, gi, x[3]));
            }
        }
#pragma unroll
        for (int v = 0; v < NV; ++v)
            pt[(static_cast<int64_t>(p) * NV + v) * sh.node_cap + tile * NT + t] = x[v];
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        s_last = atomicAdd(&done[f * n_nt + tile], 1u) == static_cast<unsigned>(fr.n_grp - 1);
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const double *p0 = part + static_cast<int64_t>(f) * sh.grp_cap * row;
    for (int k = threadIdx.x; k < n_pairs * NV * nn; k += PD_DSUM_THREADS) {
        const int pv = k / nn, t = k - pv * nn, p = pv / NV, v = pv % NV;
        const double *q = p0 + static_cast<int64_t>(pv) * sh.node_cap + tile * NT + t;
        double s = 0.0;
        int g = 0;
        for (; g + 8 <= fr.n_grp; g += 8) {
            double x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) x[u] = __ldcg(q + (g + u) * row);
#pragma unroll
            for (int u = 0; u < 8; ++u) s += x[u];
        }
        for (; g < fr.n_grp; ++g) s += __ldcg(q + g * row);
        const PdPairDev pr = pairs[p];
        if (pr.a == pr.b) {  // all (i, j) of the class: i < j is half of the rest
            const PdClassDev cl = cls[pr.a];
            const double diag = v == 0 ? cl.n : (v == 3 ? cl.w2 : cl.w1);
            s = 0.5 * (s - (add_exact ? diag : 0.0));
        }
        red[(static_cast<int64_t>(f) * n_pairs * NV + pv) * width + tile * NT + t] = s;
    }
}

// c_n(z)·z/4 (c_0·z/2) unnormalised for n < n_mom into coef[n·stride], z = q·d (see
// pd_moments.cuh); returns the factor that makes them c_n. J_ν(z) by Miller's
// downward recurrence, normalised with J_0 + 2ΣJ_2k = 1; it starts a few terms
// beyond the moments z needs, where the value it drops is below the last bit.
__device__ double moment_coefficients(double z, int n_mom, double *__restrict__ coef, int stride) {
    if (!(z > 1e-8)) {  // sinc = 1 to the last bit
        for (int n = 0; n < n_mom; ++n) coef[n * stride] = n == 0 ? 1.0 : 0.0;
        return 1.0;
    }
    const double tz = 2.0 / z;
    const int top = min(moments_needed(z, true) + 4, n_mom + 8);
    for (int n = top + 1; n < n_mom; ++n) coef[n * stride] = 0.0;
    double hi = 0.0, cur = 1e-200;  // J_{ν+1}, J_ν at ν = 2·top + 1
    double even = 0.0, odd = 0.0;   // ΣJ_2k (k >= 1), ΣJ_{2k+1}
    for (int n = top; n > 0; --n) {
        odd += cur;  // ν = 2n + 1
        if (n < n_mom) coef[n * stride] = odd;
        const double nu = 2.0 * n;
        const double lower = fma((nu + 1.0) * tz, cur, -hi);  // J_2n
        even += lower;
        cur = fma(nu * tz, lower, -cur);                      // J_{2n−1}
        hi = lower;
    }
    odd += cur;
    coef[0] = 0.5 * odd;
    const double j0 = fma(tz, cur, -hi);
    return 2.0 * tz / fma(2.0, even, j0);
}

// Six profiles of PD_PROF_Q grid points of one frame: the class-pair sums
// Σ sinc(q r) (read, formed from the moments, or interpolated from the nodes),
// times the class factors, all in FP64. 32 groups of eight threads (one per
// grid point) share the class pairs, and where there are fewer pairs than
// groups also the moments; their partial profiles are added in a fixed order. The rows
// of as many pairs as fit are staged in shared memory with all loads in flight,
// and so are the class factors (STAGED) unless there are too many classes for
// that: the species are not bounded, only (species, weight) classes are. Then
// they are read where they are used (from L2; profile_smem draws the line).
constexpr int PD_PROF_Q = 8;
constexpr int PD_PROF_THREADS = 256;
constexpr int PD_PROF_GROUPS = PD_PROF_THREADS / PD_PROF_Q;
// Doubles of pair rows staged at once. A step waits for its copies and two barriers, so
// where the pairs take more than a few steps the steps are longer: 7,260 class pairs of
// 5,346 atoms at 393 points take 3.0 ms in steps of 16,384 and 4.6 in steps of 2,048 (5.8
// with loads through registers), 465 pairs of weighted atoms at 544 points 0.23 and 0.30
// (0.43), 435 pairs of 32 frames, 2,048 on both sides, 0.52 (0.59). The middle size
// leaves room for three blocks on an SM; above that many blocks others run while one
// waits, and the short steps win by 2-4 % of a whole solve.
constexpr int PD_PROF_ROWS = 2048, PD_PROF_ROWS_MANY = 6144, PD_PROF_ROWS_MOST = 16384;
constexpr size_t PD_PROF_SMEM = 64 * 1024;  // with the class factors, at PD_PROF_ROWS

// Its shared memory: pair rows, class factors and the coefficients of the most
// moments a frame may have (up to 16, 9 for 48 classes, and 32 KB).
static size_t profile_smem(const PdReduceShape &sh, int rows, int32_t n_cls_staged) {
    return (rows + static_cast<size_t>(n_cls_staged) * 3 * PD_PROF_Q +
            static_cast<size_t>(sh.max_moments) * PD_PROF_Q) * sizeof(double);
}

template <int NV, bool STAGED>
__global__ void __launch_bounds__(PD_PROF_THREADS)
    pd_profiles(const double *__restrict__ red, const double *__restrict__ lat_sums,
                const PdClassDev *__restrict__ cls, const PdPairDev *__restrict__ pairs,
                int32_t n_cls, PdReduceShape sh, const double *__restrict__ qv,
                const PdFrameDev *__restrict__ frames, const double2 *__restrict__ node_tab,
                const double *__restrict__ ffA, const double *__restrict__ ffC,
                const double *__restrict__ ffW, int32_t add_diag, double qmax, int32_t n_rows,
                const int *__restrict__ err, double *__restrict__ terms) {
    chain_enter();
    extern __shared__ double s_dyn[];
    __shared__ double s_c0[PD_PROF_Q], s_scale[PD_PROF_Q];
    __shared__ double s_sum[PD_PROF_THREADS / 32][6][PD_PROF_Q];
    double *s_row = s_dyn;                                 // [pair][nv][M]
    double *s_fac = s_row + n_rows;                        // [class][A, C, B][PD_PROF_Q]
    double *s_coef = s_fac + (STAGED ? n_cls * 3 * PD_PROF_Q : 0);  // [M][PD_PROF_Q]
    const int n_qt = (sh.nq + PD_PROF_Q - 1) / PD_PROF_Q;
    const int f = blockIdx.x / n_qt;
    const int ql = threadIdx.x % PD_PROF_Q, g = threadIdx.x / PD_PROF_Q;
    const int q = (blockIdx.x % n_qt) * PD_PROF_Q + ql;
    const bool ok = q < sh.nq;
    constexpr bool weighted = NV == 4;
    const PdFrameDev fr = frames[f];
    // M values per class-pair row: nodes, or moments of the pairs; 0: grid points
    const bool dirs = fr.n_grp > 0, nodes = dirs && !sh.fp64;
    const int M = nodes ? fr.n_node : (dirs ? 0 : fr.n_mom);
    const double *rows = red + static_cast<int64_t>(f) * sh.n_pairs * NV * sh.width;
    // the rows of pairs [p0, p0 + n): n·NV rows of M
    const int fit = M > 0 ? min(sh.n_pairs, n_rows / (NV * M)) : 0;
    auto stage_rows = [&](int p0, int n) {
        const int dr = PD_PROF_THREADS / M, dm = PD_PROF_THREADS - dr * M;
        int r = threadIdx.x / M, m = threadIdx.x - r * M;
        const double *from = rows + static_cast<int64_t>(p0) * NV * sh.width;
        const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(s_row));
        for (int k = threadIdx.x; k < n * NV * M; k += PD_PROF_THREADS) {
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to + 8 * k),
                         "l"(from + static_cast<int64_t>(r) * sh.width + m)
                         : "memory");
            r += dr;
            m += dm;
            if (m >= M) m -= M, ++r;
        }
    };
    auto rows_staged = [] { asm volatile("cp.async.wait_all;" ::: "memory"); };
    if (M > 0) stage_rows(0, fit);
    // factor w (atom, excluded, hydration) of class c at grid point qq
    auto factor = [&](int c, int w, int qq) {
        double v = 0.0;
        if (qq < sh.nq) {
            const int64_t at = static_cast<int64_t>(cls[c].species) * sh.nq + qq;
            if (w == 0) v = ffA[at];
            if (w == 1 && ffC) v = ffC[at];
            if (w == 2 && ffW) v = weighted ? ffW[qq] : cls[c].w * ffW[qq];
        }
        return v;
    };
    if constexpr (STAGED)
        for (int k = threadIdx.x; k < n_cls * 3 * PD_PROF_Q; k += PD_PROF_THREADS)
            s_fac[k] = factor(k / (3 * PD_PROF_Q), k / PD_PROF_Q % 3, q - ql + k % PD_PROF_Q);
    auto own_factor = [&](int c, int w) {
        if constexpr (STAGED) return s_fac[(c * 3 + w) * PD_PROF_Q + ql];
        return factor(c, w, q);
    };
    const double qval = ok ? qv[q] : 0.0;
    if (nodes) {
        // interpolation from the Chebyshev nodes y_k = cos((2k+1)π/2M) of
        // y = 2(q/qmax)² − 1, barycentric form
        const double y = qmax > 0.0 ? 2.0 * (qval / qmax) * (qval / qmax) - 1.0 : -1.0;
        double sum = 0.0;
        int hit = 0;
        for (int k = g; k < M; k += PD_PROF_GROUPS) {
            const double2 nd = __ldg(node_tab + static_cast<int64_t>(f) * sh.node_cap + k);
            const double dy = y - nd.x;
            const double l = dy != 0.0 ? nd.y / dy : 0.0;
            if (dy == 0.0) hit = k + 1;
            s_coef[k * PD_PROF_Q + ql] = l;
            sum += l;
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 8);
        sum += __shfl_xor_sync(0xffffffffu, sum, 16);
        hit = max(hit, __shfl_xor_sync(0xffffffffu, hit, 8));
        hit = max(hit, __shfl_xor_sync(0xffffffffu, hit, 16));
        if ((threadIdx.x & 31) < PD_PROF_Q) {
            s_sum[threadIdx.x >> 5][0][ql] = sum;
            s_sum[threadIdx.x >> 5][1][ql] = hit;
        }
        __syncthreads();
        double v = 0.0, h = 0.0;
#pragma unroll
        for (int w = 0; w < PD_PROF_THREADS / 32; ++w) {
            v += s_sum[w][0][ql];
            h = fmax(h, s_sum[w][1][ql]);  // the grid point's own node + 1, or 0
        }
        const double scale = 1.0 / v;
        for (int k = g; k < M; k += PD_PROF_GROUPS) {
            double &c = s_coef[k * PD_PROF_Q + ql];
            c = h > 0.0 ? (k + 1 == static_cast<int>(h) ? 1.0 : 0.0) : c * scale;
        }
    } else if (M > 0) {
        if (threadIdx.x < PD_PROF_Q) {
            s_scale[ql] = moment_coefficients(qval * fr.d, M, s_coef + ql, PD_PROF_Q);
            s_c0[ql] = s_coef[ql] * s_scale[ql];
        }
        __syncthreads();
        // the factors of the tiles' sums e = 8j + 2t + {0, 1}, Σ X·vx and Σ Y·vy:
        // (c_lo + c_hi)/2 and (c_hi − c_lo)/2 of the moments lo = 8j + 3 − t and
        // hi = 8j + 4 + t
        for (int j = g; j < M / 8; j += PD_PROF_GROUPS) {
            double c[8];
#pragma unroll
            for (int n = 0; n < 8; ++n)
                c[n] = 0.5 * s_scale[ql] * s_coef[(8 * j + n) * PD_PROF_Q + ql];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                s_coef[(8 * j + 2 * t) * PD_PROF_Q + ql] = c[3 - t] + c[4 + t];
                s_coef[(8 * j + 2 * t + 1) * PD_PROF_Q + ql] = c[4 + t] - c[3 - t];
            }
        }
    }
    rows_staged();
    __syncthreads();
    double AA = 0, CC = 0, BB = 0, AC = 0, AB = 0, CB = 0;
    if (add_diag) {  // i = j terms
        for (int c = g; c < n_cls; c += PD_PROF_GROUPS) {
            const PdClassDev cl = cls[c];
            const double fa = own_factor(c, 0), ca = own_factor(c, 1), b = own_factor(c, 2);
            AA += cl.n * fa * fa;
            CC += cl.n * ca * ca;
            AC += cl.n * fa * ca;
            BB += (weighted ? cl.w2 : cl.n) * b * b;
            AB += (weighted ? cl.w1 : cl.n) * fa * b;
            CB += (weighted ? cl.w1 : cl.n) * ca * b;
        }
    }
    for (int p0 = 0; p0 < sh.n_pairs;) {
        // M = 0 (grid points summed directly): one value per pair, not staged
        const int n = M > 0 ? min(fit, sh.n_pairs - p0) : sh.n_pairs;
        if (p0 > 0) {
            __syncthreads();  // the previous pairs' rows are read
            stage_rows(p0, n);
            rows_staged();
            __syncthreads();
        }
        // groups per class pair (they share its moments)
        const int per = n >= PD_PROF_GROUPS ? 1 : PD_PROF_GROUPS / n;
        const int sub = g % per;
        for (int pl = g / per; pl < n; pl += PD_PROF_GROUPS / per) {
            const int p = p0 + pl;
            const PdPairDev pr = pairs[p];
            double s[NV];
#pragma unroll
            for (int v = 0; v < NV; ++v) s[v] = 0.0;
            const int lat = pr.a == pr.b ? cls[pr.a].lat : -1;
            if (lat >= 0) {  // from the lattice set's pair counts (class mode, one frame)
                if (sub == 0 && ok) s[0] = lat_sums[static_cast<int64_t>(lat) * sh.nq + q];
            } else if (!(qval > 0.0)) {  // exact pair sums
                if (sub == 0 && add_diag)
#pragma unroll
                    for (int v = 0; v < NV; ++v) s[v] = pr.q0[v];
            } else if (M == 0) {
                if (sub == 0 && ok)
#pragma unroll
                    for (int v = 0; v < NV; ++v)
                        s[v] = rows[static_cast<int64_t>(p * NV + v) * sh.width + q];
            } else {
                const double *r = s_row + pl * NV * M;
#pragma unroll 4
                for (int e = sub; e < M; e += per) {
                    const double c = s_coef[e * PD_PROF_Q + ql];
#pragma unroll
                    for (int v = 0; v < NV; ++v) s[v] = fma(c, r[v * M + e], s[v]);
                }
                // the zeroth moment is the exact pair sum at q = 0, not the
                // tiles' rounded (Σ X·vx − Σ Y·vy)/2
                if (!nodes && sub == 0)
#pragma unroll
                    for (int v = 0; v < NV; ++v)
                        s[v] = fma(s_c0[ql],
                                   (add_diag ? pr.q0[v] : 0.0) - 0.5 * (r[v * M + 6] - r[v * M + 7]),
                                   s[v]);
            }
            const double fa = own_factor(pr.a, 0), fb = own_factor(pr.b, 0);
            const double ca = own_factor(pr.a, 1), cb = own_factor(pr.b, 1);
            const double ba = own_factor(pr.a, 2), bb = own_factor(pr.b, 2);
            AA += 2.0 * fa * fb * s[0];
            CC += 2.0 * ca * cb * s[0];
            AC += (fa * cb + ca * fb) * s[0];
            if constexpr (weighted) {  // ba = bb = F_water
                BB += 2.0 * ba * ba * s[3];
                AB += ba * (fa * s[2] + fb * s[1]);
                CB += ba * (ca * s[2] + cb * s[1]);
            } else {
                BB += 2.0 * ba * bb * s[0];
                AB += (fa * bb + ba * fb) * s[0];
                CB += (ca * bb + ba * cb) * s[0];
            }
        }
        p0 += n;
    }
    double out[6] = {AA, CC, BB, AC, AB, CB};
#pragma unroll
    for (int t = 0; t < 6; ++t) {
        out[t] += __shfl_xor_sync(0xffffffffu, out[t], 8);
        out[t] += __shfl_xor_sync(0xffffffffu, out[t], 16);
    }
    __syncthreads();  // s_sum's earlier use is over
    if ((threadIdx.x & 31) < PD_PROF_Q)
#pragma unroll
        for (int t = 0; t < 6; ++t) s_sum[threadIdx.x >> 5][t][ql] = out[t];
    __syncthreads();
    if (threadIdx.x < 6 * PD_PROF_Q) {
        const int t = threadIdx.x / PD_PROF_Q;
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < PD_PROF_THREADS / 32; ++w) v += s_sum[w][t][ql];
        // a point off its lattice, or a frame whose form the plan has nothing for
        if ((err && *err) || (sh.dir_only && !dirs)) v = __longlong_as_double(0x7ff8000000000000ll);
        if (ok) terms[(static_cast<int64_t>(f) * 6 + t) * sh.nq + q] = v;
    }
}

// ------------------------------------------------------------ lattice sets
// Integer lattice coordinates of every point of every lattice set, from the
// FP64 input positions (frame 0): i = rint((x - origin)/spacing) per axis. A
// point farther than 1e-6·spacing from its lattice node, or outside the
// extents, sets *err (the profiles of the request then become NaN).
__global__ void pd_lattice_index(const double *__restrict__ xyz, const int32_t *__restrict__ perm,
                                 const PdLatDev *__restrict__ lat, int4 *__restrict__ idx,
                                 int *__restrict__ err) {
    const PdLatDev d = lat[blockIdx.y];
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < d.n; r += gridDim.x * blockDim.x) {
        const int p = d.start + r;
        const int64_t src = perm[p];
        int c[3] = {0, 0, 0};  // an invalid point counts at the origin node (in range)
        bool ok = src >= 0;
        for (int a = 0; a < 3 && ok; ++a) {
            const double x = xyz[3 * src + a];
            const double u = (x - d.origin[a]) / d.spacing;
            const double ur = rint(u);
            ok = fabs(x - (d.origin[a] + ur * d.spacing)) <= 1e-6 * d.spacing && ur >= 0.0 &&
                 ur < static_cast<double>(d.ext[a]);
            c[a] = ok ? static_cast<int>(ur) : 0;
        }
        if (!ok) atomicOr(err, 1);
        idx[p] = make_int4(c[0], c[1], c[2], 0);
    }
}

// Exact pair counts per integer squared offset n = |Δ(i, j, k)|² of a
// lattice set: one CTA per tile (128 i points, a range of j points, j > i),
// counted in a shared-memory histogram (32-bit: a tile holds at most
// 128 × 8192 pairs) and added to the FP64-free 64-bit global histogram at the
// end. Integer sums: the counts do not depend on the order the CTAs run in.
// With more bins than fit in shared memory (`shared_bins` = 0) the CTA adds
// straight to the global histogram.
__global__ void __launch_bounds__(128) pd_lattice_hist(const PdLatTile *__restrict__ tiles,
                                                       const PdLatDev *__restrict__ lat,
                                                       const int4 *__restrict__ idx,
                                                       unsigned long long *__restrict__ hist,
                                                       int shared_bins) {
    extern __shared__ unsigned int s_hist[];
    const PdLatTile t = tiles[blockIdx.x];
    const PdLatDev d = lat[t.lat];
    const bool use_shared = shared_bins > 0;
    if (use_shared)
        for (int b = threadIdx.x; b < d.n_bins; b += blockDim.x) s_hist[b] = 0u;
    __syncthreads();
    const int i = t.i0 + threadIdx.x;
    if (i < d.n) {
        const int4 a = idx[d.start + i];
        for (int j = max(t.j0, i + 1); j < t.j1; ++j) {
            const int4 b = idx[d.start + j];
            const int dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
            const int n = dx * dx + dy * dy + dz * dz;  // < n_bins: both points in the extents
            if (use_shared)
                atomicAdd(&s_hist[n], 1u);
            else
                atomicAdd(&hist[d.hist_off + n], 1ull);
        }
    }
    __syncthreads();
    if (use_shared)
        for (int b = threadIdx.x; b < d.n_bins; b += blockDim.x) {
            const unsigned int v = s_hist[b];
            if (v) atomicAdd(&hist[d.hist_off + b], static_cast<unsigned long long>(v));
        }
}

// Self pair sums of the lattice sets from their pair counts:
// Σ_{i<j} sinc(q r_ij) = Σ_n count(n)·sinc(q·spacing·√n), FP64, one CTA per
// (q, lattice); each thread adds the bins n ≡ thread (mod 256) in ascending
// order and a fixed tree adds the threads, so the sum is deterministic. The
// values are sums[lattice][q] (the pair tiles skip those pairs; where directions are
// summed, whose FP32 terms these counts are exact beside, their own sum goes unused). Only the rank
// that adds the exact terms writes a sum; the others write 0. *err set: NaN.
__global__ void __launch_bounds__(256) pd_lattice_sums(const unsigned long long *__restrict__ hist,
                                                       const PdLatDev *__restrict__ lat,
                                                       const double *__restrict__ qv, int32_t nq,
                                                       int32_t add_exact,
                                                       const int *__restrict__ err,
                                                       double *__restrict__ sums) {
    __shared__ double s_part[256];
    const int q = blockIdx.x;
    const PdLatDev d = lat[blockIdx.y];
    const double qval = qv[q];
    double acc = 0.0;
    for (int n = 1 + threadIdx.x; n < d.n_bins; n += 256) {
        const unsigned long long c = hist[d.hist_off + n];
        if (c == 0ull) continue;
        const double x = qval * d.spacing * sqrt(static_cast<double>(n));
        // sinc as the reference defines it (src/debye.rs:17-24)
        const double sc = fabs(x) < 1e-8 ? 1.0 : sin(x) / x;
        acc += static_cast<double>(c) * sc;
    }
    s_part[threadIdx.x] = acc;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) s_part[threadIdx.x] += s_part[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        double v = add_exact ? s_part[0] : 0.0;
        if (*err) v = __longlong_as_double(0x7ff8000000000000ll);  // NaN
        sums[static_cast<int64_t>(blockIdx.y) * nq + q] = v;
    }
}

// Frame-weighted mean of the six profiles, frames added in order.
__global__ void pd_frame_mean(const double *__restrict__ terms, const double *__restrict__ fw,
                              int32_t n_frames, int32_t nq, int32_t normalize,
                              double *__restrict__ out) {
    chain_enter();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 6 * nq) return;
    double s = 0.0, wsum = 0.0;
    for (int f = 0; f < n_frames; ++f) {
        const double w = fw ? fw[f] : 1.0;
        s += w * terms[static_cast<int64_t>(f) * 6 * nq + t];
        wsum += w;
    }
    out[t] = normalize ? s / wsum : s;
}

// Streamed trajectories: acc += batch, where batch is one batch's
// unnormalised Σ_f w_f·T_f (or, for a one-frame batch, T times its weight).
// Batches are added in submission order.
__global__ void pd_stream_accumulate(const double *__restrict__ batch, double scale, int32_t n,
                                     double *__restrict__ acc) {
    chain_enter();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) acc[t] += scale * batch[t];
}

// ------------------------------------------------------------ Direct transform
// Amplitudes of a periodic box at explicit q-vectors (the reference's
// DirectTransform, src/explicit.rs:138-147 and :208-230), FP64 throughout:
// F(q) = Σ_j f_j(q)·e^{i q·r_j} with q·r evaluated as q_x·x + q_y·y + q_z·z and
// one sincos per (vector, point). The points are split into chunks that never
// straddle a molecule: groups of whole molecules (molecules of at most
// a chunk length of points), for which the chunk also forms Σ_m |F_m|², or
// slices of that many points of one molecule (the last one shorter), whose
// partial amplitudes the reduction joins per molecule. The chunk length is
// 1,024, 512 or 256 points: the longest that still gives PD_DIRECT_BLOCKS
// blocks, so that the last wave of blocks is a small part of the launch.
//
// A block of 128 threads owns 2 × 128 q-vectors (two independent sincos
// chains per thread) and walks its chunk in stages of PD_DIRECT_STAGE points
// copied to shared memory (coordinates, weight, kind), which every thread then
// reads as broadcasts; the form factors of up to PD_DIRECT_SMEM_KINDS kinds for
// the block's vectors sit in shared memory as well, so the inner loop reads no
// global memory.
constexpr int PD_DIRECT_CHUNK_MAX = 1024, PD_DIRECT_CHUNK_MIN = 256;
constexpr int64_t PD_DIRECT_BLOCKS = 4096;  // about 6 waves of 148 SMs x 5 blocks
constexpr int PD_DIRECT_THREADS = 128;
constexpr int PD_DIRECT_V = 2;  // q-vectors per thread
constexpr int PD_DIRECT_STAGE = 256;
constexpr int PD_DIRECT_SMEM_KINDS = 16;

__global__ void __launch_bounds__(PD_DIRECT_THREADS)
    pd_direct_chunks(const double *__restrict__ xyz, const uint32_t *__restrict__ kind,
                     const double *__restrict__ weight, const double *__restrict__ ff,
                     const double *__restrict__ qvec, int64_t n_vec, int64_t n_vblocks,
                     int64_t mol_size, int64_t chunk_points, int64_t slices_per_mol,
                     int64_t n_points, int32_t n_kinds, double *__restrict__ part) {
    constexpr int V = PD_DIRECT_V, T = PD_DIRECT_THREADS;
    __shared__ double s_x[PD_DIRECT_STAGE], s_y[PD_DIRECT_STAGE], s_z[PD_DIRECT_STAGE],
        s_w[PD_DIRECT_STAGE];
    __shared__ uint32_t s_k[PD_DIRECT_STAGE];
    __shared__ double s_f[PD_DIRECT_SMEM_KINDS][V * T];
    const int tid = threadIdx.x;
    // consecutive blocks: the vector blocks of one chunk (its points stay in L2)
    const int64_t c = blockIdx.x / n_vblocks, vb = blockIdx.x % n_vblocks;
    int64_t v[V];
    bool ok[V];
    double qx[V], qy[V], qz[V];
#pragma unroll
    for (int j = 0; j < V; ++j) {
        v[j] = vb * (V * T) + j * T + tid;
        ok[j] = v[j] < n_vec;
        qx[j] = ok[j] ? qvec[3 * v[j]] : 0.0;
        qy[j] = ok[j] ? qvec[3 * v[j] + 1] : 0.0;
        qz[j] = ok[j] ? qvec[3 * v[j] + 2] : 0.0;
    }
    const bool smem_ff = n_kinds <= PD_DIRECT_SMEM_KINDS;
    if (smem_ff)
        for (int k = 0; k < n_kinds; ++k)
#pragma unroll
            for (int j = 0; j < V; ++j)
                s_f[k][j * T + tid] = ok[j] ? ff[static_cast<int64_t>(k) * n_vec + v[j]] : 0.0;
    int64_t p0, p1;
    if (slices_per_mol == 1) {  // whole molecules
        p0 = c * chunk_points;
        p1 = min(n_points, p0 + chunk_points);
    } else {                    // slice s of molecule m
        const int64_t m = c / slices_per_mol, sl = c % slices_per_mol;
        p0 = m * mol_size + sl * chunk_points;
        p1 = min((m + 1) * mol_size, p0 + chunk_points);
    }
    const bool whole = slices_per_mol == 1;
    int64_t mol_end = (p0 / mol_size + 1) * mol_size;  // first molecule end after p0
    double ar[V], ai[V], self[V], fr[V], fi[V];
#pragma unroll
    for (int j = 0; j < V; ++j) ar[j] = ai[j] = self[j] = fr[j] = fi[j] = 0.0;
    for (int64_t s0 = p0; s0 < p1; s0 += PD_DIRECT_STAGE) {
        const int ns = static_cast<int>(min(static_cast<int64_t>(PD_DIRECT_STAGE), p1 - s0));
        __syncthreads();  // the previous stage is read (and s_f written)
        for (int t = tid; t < ns; t += T) {
            const int64_t p = s0 + t;
            s_x[t] = xyz[3 * p];
            s_y[t] = xyz[3 * p + 1];
            s_z[t] = xyz[3 * p + 2];
            s_w[t] = weight ? weight[p] : 1.0;
            s_k[t] = kind[p];
        }
        __syncthreads();
        for (int t = 0; t < ns; ++t) {
            const double x = s_x[t], y = s_y[t], z = s_z[t], w = s_w[t];
            const uint32_t k = s_k[t];
#pragma unroll
            for (int j = 0; j < V; ++j) {
                double f = smem_ff ? s_f[k][j * T + tid]
                                   : (ok[j] ? ff[static_cast<int64_t>(k) * n_vec + v[j]] : 0.0);
                if (weight) f = w * f;  // DummySet::Weighted: w·F
                const double qr = qx[j] * x + qy[j] * y + qz[j] * z;
                double sn, cs;
                sincos(qr, &sn, &cs);
                fr[j] += f * cs;
                fi[j] += f * sn;
            }
            if (whole && s0 + t + 1 == mol_end) {  // a molecule ends inside this chunk
#pragma unroll
                for (int j = 0; j < V; ++j) {
                    ar[j] += fr[j];
                    ai[j] += fi[j];
                    self[j] += fr[j] * fr[j] + fi[j] * fi[j];
                    fr[j] = 0.0;
                    fi[j] = 0.0;
                }
                mol_end += mol_size;
            }
        }
    }
    // whole molecules: (A, Σ|F_m|²); a slice of a molecule: its open partial F
#pragma unroll
    for (int j = 0; j < V; ++j) {
        if (!ok[j]) continue;
        double *o = part + (c * n_vec + v[j]) * 5;
        o[0] = ar[j];
        o[1] = ai[j];
        o[2] = self[j];
        o[3] = fr[j];
        o[4] = fi[j];
    }
}

// Direct transform at reciprocal-lattice vectors q = 2π·(h, k, l)/L: the phase
// of a term is e^{i2πh·x/Lx}·e^{i2πk·y/Ly}·e^{i2πl·z/Lz}. Per stage of points
// the block builds, in shared memory, each point's powers e^{i2πn·x_a/L_a} for
// n = 0..nmax on every axis (segments of a row start from a sincos and step by
// products with e^{i2π·x_a/L_a}; negative n by conjugation: the reference's
// PhaseTable, src/explicit.rs:85-135). A term then costs three table reads and two
// complex products instead of a sincos. Same chunks, partial layout and
// reduction as pd_direct_chunks; 256 threads own 3 × 256 vectors.
constexpr int PD_DTAB_THREADS = 256;
constexpr int PD_DTAB_V = 3;
constexpr int PD_DTAB_MAX_POINTS = 64;
constexpr int PD_DTAB_TABLE_BYTES = 96 * 1024;

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// a, or its conjugate when neg is the sign bit of the high word
__device__ __forceinline__ double2 conj_if(double2 a, int neg) {
    return make_double2(a.x, __hiloint2double(__double2hiint(a.y) ^ neg, __double2loint(a.y)));
}

__global__ void __launch_bounds__(PD_DTAB_THREADS, 2)
    pd_direct_table(const double *__restrict__ xyz, const uint32_t *__restrict__ kind,
                    const double *__restrict__ weight, const double *__restrict__ ff,
                    const int32_t *__restrict__ hkl, double lx, double ly, double lz,
                    int32_t stride, int32_t npts, int64_t n_vec, int64_t n_vblocks,
                    int64_t mol_size, int64_t chunk_points, int64_t slices_per_mol,
                    int64_t n_points, double *__restrict__ part) {
    constexpr int V = PD_DTAB_V, T = PD_DTAB_THREADS;
    extern __shared__ __align__(16) double2 pd_dtab[];  // [npts][3][stride]
    __shared__ double s_w[PD_DTAB_MAX_POINTS];
    __shared__ uint32_t s_k[PD_DTAB_MAX_POINTS];
    const int tid = threadIdx.x;
    const int64_t c = blockIdx.x / n_vblocks, vb = blockIdx.x % n_vblocks;
    int64_t v[V];
    bool ok[V];
    int ox[V], oy[V], oz[V], sx[V], sy[V], sz[V];
#pragma unroll
    for (int j = 0; j < V; ++j) {
        v[j] = vb * (V * T) + j * T + tid;
        ok[j] = v[j] < n_vec;
        const int h = ok[j] ? hkl[3 * v[j]] : 0, k = ok[j] ? hkl[3 * v[j] + 1] : 0,
                  l = ok[j] ? hkl[3 * v[j] + 2] : 0;
        ox[j] = abs(h);
        oy[j] = stride + abs(k);
        oz[j] = 2 * stride + abs(l);
        sx[j] = h < 0 ? static_cast<int>(0x80000000u) : 0;
        sy[j] = k < 0 ? static_cast<int>(0x80000000u) : 0;
        sz[j] = l < 0 ? static_cast<int>(0x80000000u) : 0;
    }
    int64_t p0, p1;
    if (slices_per_mol == 1) {
        p0 = c * chunk_points;
        p1 = min(n_points, p0 + chunk_points);
    } else {
        const int64_t m = c / slices_per_mol, sl = c % slices_per_mol;
        p0 = m * mol_size + sl * chunk_points;
        p1 = min((m + 1) * mol_size, p0 + chunk_points);
    }
    const bool whole = slices_per_mol == 1;
    int64_t mol_end = (p0 / mol_size + 1) * mol_size;
    double ar[V], ai[V], self[V], fr[V], fi[V];
#pragma unroll
    for (int j = 0; j < V; ++j) ar[j] = ai[j] = self[j] = fr[j] = fi[j] = 0.0;
    for (int64_t s0 = p0; s0 < p1; s0 += npts) {
        const int ns = static_cast<int>(min(static_cast<int64_t>(npts), p1 - s0));
        __syncthreads();  // the previous stage's table is read
        // the rows e^{i2πn·x_a/L_a}, n = 0..stride-1, one per (point, axis),
        // each cut into up to 16-entry segments so that every thread takes
        // part: a segment starts from its own sincos and steps by products
        const int rows = 3 * ns;
        const int nseg = max(1, min((stride + 15) / 16, T / rows));
        const int seglen = (stride + nseg - 1) / nseg;
        for (int t = tid; t < rows * nseg; t += T) {
            const int rw = t / nseg, sg = t - rw * nseg;
            const int pt = rw / 3, a = rw - 3 * pt;
            const int n0 = sg * seglen, n1 = min(stride, n0 + seglen);
            const double x = xyz[3 * (s0 + pt) + a];
            const double L = a == 0 ? lx : (a == 1 ? ly : lz);
            const double th = 2.0 * 3.141592653589793 * x / L;
            double sn, cs;
            sincos(th, &sn, &cs);
            const double2 step = make_double2(cs, sn);
            double2 e = make_double2(1.0, 0.0);
            if (n0 > 0) {
                sincos(static_cast<double>(n0) * th, &sn, &cs);
                e = make_double2(cs, sn);
            }
            double2 *row = pd_dtab + rw * stride;
            for (int n = n0; n < n1; ++n) {
                row[n] = e;
                e = cmul(e, step);
            }
        }
        for (int t = tid; t < ns; t += T) {
            s_w[t] = weight ? weight[s0 + t] : 1.0;
            s_k[t] = kind[s0 + t];
        }
        __syncthreads();
        for (int pt = 0; pt < ns; ++pt) {
            const double2 *row = pd_dtab + 3 * pt * stride;
            const double w = s_w[pt];
            const uint32_t k = s_k[pt];
#pragma unroll
            for (int j = 0; j < V; ++j) {
                double f = ok[j] ? ff[static_cast<int64_t>(k) * n_vec + v[j]] : 0.0;
                if (weight) f = w * f;  // DummySet::Weighted: w·F
                const double2 ph = cmul(cmul(conj_if(row[ox[j]], sx[j]), conj_if(row[oy[j]], sy[j])),
                                        conj_if(row[oz[j]], sz[j]));
                fr[j] += f * ph.x;
                fi[j] += f * ph.y;
            }
            if (whole && s0 + pt + 1 == mol_end) {
#pragma unroll
                for (int j = 0; j < V; ++j) {
                    ar[j] += fr[j];
                    ai[j] += fi[j];
                    self[j] += fr[j] * fr[j] + fi[j] * fi[j];
                    fr[j] = 0.0;
                    fi[j] = 0.0;
                }
                mol_end += mol_size;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < V; ++j) {
        if (!ok[j]) continue;
        double *o = part + (c * n_vec + v[j]) * 5;
        o[0] = ar[j];
        o[1] = ai[j];
        o[2] = self[j];
        o[3] = fr[j];
        o[4] = fi[j];
    }
}

// Direct transform at lattice vectors that lie on lines n0 + j·δ (the Miller grid's
// multiples of a direction, or consecutive indices along an axis): a thread owns
// a segment of PD_DLINE_J vectors of one line and needs, per point, only the
// phases of its start and step — two products of table entries — instead of three
// table reads and two complex products per vector (pd_direct_table: the reads
// bound it, 0.50 ms for 128,000 points × 1,300 vectors; this kernel: 0.123 ms).
// With E = e^{iφ} at the segment's index 4 (and 12) and
// V_k = e^{ikδ·r}, the vectors ±k around it share four products,
//   Re = x·c ∓ y·s, Im = y·c ± x·s,
// accumulated separately: 4.6 FP64 operations per (vector, point). The points of
// a molecule are sorted by kind, so the form factors enter once per kind of a chunk
// (flush), not per point. A table holds the distinct |indices| that starts and steps
// use on each axis. Chunks are slices of one molecule.
constexpr int PD_DLINE_J = 16;
constexpr int PD_DLINE_THREADS = 128;
constexpr int PD_DLINE_MAX_POINTS = 64;
constexpr int PD_DLINE_TABLE_BYTES = 40 * 1024;

__device__ __forceinline__ double2 csqr(double2 a) {
    return make_double2(fma(a.x, a.x, -a.y * a.y), 2.0 * a.x * a.y);
}

__global__ void __launch_bounds__(PD_DLINE_THREADS, 3)
    pd_direct_lines(const double *__restrict__ xyz, const uint32_t *__restrict__ kind,
                    const double *__restrict__ weight, const double *__restrict__ ff,
                    const PdLine *__restrict__ lines, const int32_t *__restrict__ index,
                    int3 n_index, double lx, double ly, double lz, int32_t npts, int32_t n_line,
                    int32_t n_vblocks, int64_t mol_size, int64_t chunk_points,
                    int64_t slices_per_mol, double *__restrict__ part) {
    constexpr int J = PD_DLINE_J;
    extern __shared__ __align__(16) double2 pd_dl_tab[];  // [npts][entries], then [J][2][threads]
    __shared__ double s_w[PD_DLINE_MAX_POINTS], s_u[3 * PD_DLINE_MAX_POINTS];
    __shared__ uint32_t s_k[PD_DLINE_MAX_POINTS];
    const int T = blockDim.x, tid = threadIdx.x;
    const int n_ent = n_index.x + n_index.y + n_index.z;
    double *s_f = reinterpret_cast<double *>(pd_dl_tab + npts * n_ent);
    const int64_t c = blockIdx.x / n_vblocks;
    const int seg = static_cast<int>(blockIdx.x % n_vblocks) * T + tid;
    const bool ok = seg < n_line;
    const PdLine ln = lines[ok ? seg : 0];
    const int64_t m = c / slices_per_mol, sl = c % slices_per_mol;
    const int64_t p0 = m * mol_size + sl * chunk_points,
                  p1 = min((m + 1) * mol_size, p0 + chunk_points);
    // sums over the points of one kind: center h: x, y; pairs ±k: x·c, y·s, y·c,
    // x·s; index −4: re, im
    double a[2][16];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 16; ++e) a[h][e] = 0.0;
    for (int j = 0; j < 2 * J; ++j) s_f[j * T + tid] = 0.0;
    auto flush = [&](uint32_t k) {
        const double *f = ff + static_cast<int64_t>(k) * J * n_line + (ok ? seg : 0);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int b = -4; b < 4; ++b) {
                double re, im;
                if (b == -4) {
                    re = a[h][14];
                    im = a[h][15];
                } else if (b == 0) {
                    re = a[h][0];
                    im = a[h][1];
                } else {
                    const int q = 2 + 4 * ((b < 0 ? -b : b) - 1);
                    re = b > 0 ? a[h][q] - a[h][q + 1] : a[h][q] + a[h][q + 1];
                    im = b > 0 ? a[h][q + 2] + a[h][q + 3] : a[h][q + 2] - a[h][q + 3];
                }
                const int j = 8 * h + 4 + b;
                const double fj = f[static_cast<int64_t>(j) * n_line];
                s_f[(2 * j) * T + tid] = fma(fj, re, s_f[(2 * j) * T + tid]);
                s_f[(2 * j + 1) * T + tid] = fma(fj, im, s_f[(2 * j + 1) * T + tid]);
            }
#pragma unroll
            for (int e = 0; e < 16; ++e) a[h][e] = 0.0;
        }
    };
    uint32_t cur = 0xffffffffu;
    for (int64_t s0 = p0; s0 < p1; s0 += npts) {
        const int ns = static_cast<int>(min(static_cast<int64_t>(npts), p1 - s0));
        __syncthreads();  // the previous stage's table is read
        for (int t = tid; t < 3 * ns; t += T) {
            const int ax = t % 3;
            s_u[t] = xyz[3 * s0 + t] / (ax == 0 ? lx : (ax == 1 ? ly : lz));
        }
        __syncthreads();
        for (int t = tid; t < ns * n_ent; t += T) {
            const int pt = t / n_ent, e = t - pt * n_ent;
            const int ax = e < n_index.x ? 0 : (e < n_index.x + n_index.y ? 1 : 2);
            // n·x/L reduced to half a turn before the multiplication by 2π
            const double u = static_cast<double>(index[e]) * s_u[3 * pt + ax];
            double sn, cs;
            sincospi(2.0 * (u - rint(u)), &sn, &cs);
            pd_dl_tab[t] = make_double2(cs, sn);
        }
        for (int t = tid; t < ns; t += T) {
            s_w[t] = weight ? weight[s0 + t] : 1.0;
            s_k[t] = kind[s0 + t];
        }
        __syncthreads();
        for (int pt = 0; pt < ns; ++pt) {
            const uint32_t k = s_k[pt];
            if (k != cur) {
                if (cur != 0xffffffffu) flush(cur);
                cur = k;
            }
            const double2 *row = pd_dl_tab + pt * n_ent;
            // a negative index is the conjugate entry (sign bit of the member)
            auto at = [&](int32_t m) {
                return conj_if(row[m & 0x7fffffff], m & static_cast<int>(0x80000000u));
            };
            const double2 st = cmul(cmul(at(ln.sx), at(ln.sy)), at(ln.sz));
            double2 e0 = cmul(cmul(at(ln.x), at(ln.y)), at(ln.z));
            if (weight) {
                const double w = s_w[pt];
                e0.x *= w;
                e0.y *= w;
            }
            double2 v[4];
            v[0] = st;
            v[1] = csqr(st);
            v[2] = cmul(v[1], st);
            v[3] = csqr(v[1]);
            double2 E = cmul(e0, v[3]);
            const double2 v8 = csqr(v[3]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                a[h][0] += E.x;
                a[h][1] += E.y;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    a[h][2 + 4 * q] = fma(E.x, v[q].x, a[h][2 + 4 * q]);
                    a[h][3 + 4 * q] = fma(E.y, v[q].y, a[h][3 + 4 * q]);
                    a[h][4 + 4 * q] = fma(E.y, v[q].x, a[h][4 + 4 * q]);
                    a[h][5 + 4 * q] = fma(E.x, v[q].y, a[h][5 + 4 * q]);
                }
                a[h][14] = fma(E.x, v[3].x, fma(E.y, v[3].y, a[h][14]));
                a[h][15] = fma(E.y, v[3].x, fma(-E.x, v[3].y, a[h][15]));
                if (h == 0) E = cmul(E, v8);
            }
        }
    }
    if (cur != 0xffffffffu) flush(cur);
    if (!ok) return;
    double *o = part + c * 2 * J * n_line + seg;  // [chunk][j][re, im][line]
    for (int j = 0; j < 2 * J; ++j) o[static_cast<int64_t>(j) * n_line] = s_f[j * T + tid];
}

// The points of each molecule in stable order of their kinds, within pieces of up to
// PD_DSORT_PIECE points (a block each; a slice of the line kernel meets a kind once per
// piece): every thread counts the kinds of a contiguous run, the counts are scanned kind
// by kind, and the runs are scattered in order. One piece of a whole molecule would
// leave a large one to a single SM (1,000,000 points, whole call: 9.2 -> 5.1 ms).
constexpr int64_t PD_DSORT_PIECE = 4096;
constexpr int PD_DSORT_THREADS = 256;

__global__ void __launch_bounds__(PD_DSORT_THREADS)
    pd_direct_sort(const double *__restrict__ xyz, const uint32_t *__restrict__ kind,
                   const double *__restrict__ weight, int64_t mol_size, int32_t n_piece,
                   int32_t n_kinds, double *__restrict__ xyz_out,
                   uint32_t *__restrict__ kind_out, double *__restrict__ weight_out) {
    constexpr int T = PD_DSORT_THREADS;
    extern __shared__ uint32_t s_cnt[];  // [kind][thread]
    __shared__ uint32_t s_scan[T];
    const int64_t mol = blockIdx.x / n_piece, part = blockIdx.x % n_piece;
    const int64_t m0 = mol * mol_size + mol_size * part / n_piece;
    const int64_t size = mol * mol_size + mol_size * (part + 1) / n_piece - m0;
    const int t = threadIdx.x;
    const int64_t i0 = m0 + size * t / T, i1 = m0 + size * (t + 1) / T;
    for (int k = 0; k < n_kinds; ++k) s_cnt[k * T + t] = 0;
    for (int64_t i = i0; i < i1; ++i) ++s_cnt[kind[i] * T + t];
    __syncthreads();
    // exclusive scan of the flattened counts: n_kinds consecutive ones per thread
    uint32_t sum = 0;
    for (int k = 0; k < n_kinds; ++k) sum += s_cnt[t * n_kinds + k];
    s_scan[t] = sum;
    __syncthreads();
    for (int o = 1; o < T; o <<= 1) {
        const uint32_t v = t >= o ? s_scan[t - o] : 0;
        __syncthreads();
        s_scan[t] += v;
        __syncthreads();
    }
    uint32_t at = s_scan[t] - sum;
    for (int k = 0; k < n_kinds; ++k) {
        const uint32_t v = s_cnt[t * n_kinds + k];
        s_cnt[t * n_kinds + k] = at;
        at += v;
    }
    __syncthreads();
    for (int64_t i = i0; i < i1; ++i) {
        const uint32_t k = kind[i];
        const int64_t o = m0 + s_cnt[k * T + t]++;
        xyz_out[3 * o] = xyz[3 * i];
        xyz_out[3 * o + 1] = xyz[3 * i + 1];
        xyz_out[3 * o + 2] = xyz[3 * i + 2];
        kind_out[o] = k;
        if (weight) weight_out[o] = weight[i];
    }
}

// Per vector of pd_direct_lines (j·n_line + line): the slices of a molecule joined,
// A = Σ F_m and Σ_m |F_m|². 32 lanes are 32 vectors, the warps 32 fixed runs of
// molecules, added in run order.
__global__ void __launch_bounds__(1024)
    pd_direct_lines_reduce(const double *__restrict__ part, int32_t n_line, int64_t n_mol,
                           int64_t slices_per_mol, double *__restrict__ out) {
    __shared__ double s_run[32][3][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int n_vec = PD_DLINE_J * n_line;
    const int v = blockIdx.x * 32 + lane;
    const bool ok = v < n_vec;
    const int j = ok ? v / n_line : 0, l = ok ? v - j * n_line : 0;
    const int64_t u0 = n_mol * w / 32, u1 = n_mol * (w + 1) / 32;
    double ar = 0.0, ai = 0.0, self = 0.0;
    for (int64_t m = u0; ok && m < u1; ++m) {
        double fr = 0.0, fi = 0.0;
#pragma unroll 4
        for (int64_t s = 0; s < slices_per_mol; ++s) {
            const double *o = part + ((m * slices_per_mol + s) * 2 * PD_DLINE_J + 2 * j) * n_line + l;
            fr += o[0];
            fi += o[n_line];
        }
        ar += fr;
        ai += fi;
        self += fr * fr + fi * fi;
    }
    s_run[w][0][lane] = ar;
    s_run[w][1][lane] = ai;
    s_run[w][2][lane] = self;
    __syncthreads();
    if (w == 0 && ok) {
        double x = 0.0, y = 0.0, sf = 0.0;
        for (int r = 0; r < 32; ++r) {
            x += s_run[r][0][lane];
            y += s_run[r][1][lane];
            sf += s_run[r][2][lane];
        }
        out[4 * static_cast<int64_t>(v)] = x;
        out[4 * static_cast<int64_t>(v) + 1] = y;
        out[4 * static_cast<int64_t>(v) + 2] = x * x + y * y;
        out[4 * static_cast<int64_t>(v) + 3] = sf;
    }
}

// Per q-vector: A = Σ chunks, Σ_m |F_m|² with the slices of a molecule joined
// first. out[v] = (Re A, Im A, |A|², Σ_m |F_m|²). A block takes 32 vectors (a
// lane each); its 32 warps sum 32 fixed runs of whole molecules' chunks, each in
// chunk order, and the run totals are added in run order: the same sums, in
// the same order, on every call.
constexpr int PD_DIRECT_RED_WARPS = 32;

__global__ void __launch_bounds__(32 * PD_DIRECT_RED_WARPS)
    pd_direct_reduce(const double *__restrict__ part, int64_t n_vec, int64_t n_chunks,
                     int64_t slices_per_mol, double *__restrict__ out) {
    __shared__ double s_run[PD_DIRECT_RED_WARPS][3][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t v = static_cast<int64_t>(blockIdx.x) * 32 + lane;
    const bool ok = v < n_vec;
    // runs of whole molecules: chunks [u0·spm, u1·spm)
    const int64_t units = n_chunks / slices_per_mol;
    const int64_t u0 = units * w / PD_DIRECT_RED_WARPS, u1 = units * (w + 1) / PD_DIRECT_RED_WARPS;
    double ar = 0.0, ai = 0.0, self = 0.0, fr = 0.0, fi = 0.0;
    if (ok) {
        for (int64_t c = u0 * slices_per_mol; c < u1 * slices_per_mol; ++c) {
            const double *o = part + (c * n_vec + v) * 5;
            ar += o[0];
            ai += o[1];
            self += o[2];
            if (slices_per_mol > 1) {
                fr += o[3];
                fi += o[4];
                if ((c + 1) % slices_per_mol == 0) {
                    ar += fr;
                    ai += fi;
                    self += fr * fr + fi * fi;
                    fr = 0.0;
                    fi = 0.0;
                }
            }
        }
    }
    s_run[w][0][lane] = ar;
    s_run[w][1][lane] = ai;
    s_run[w][2][lane] = self;
    __syncthreads();
    if (w == 0 && ok) {
        double a = 0.0, b = 0.0, sf = 0.0;
        for (int r = 0; r < PD_DIRECT_RED_WARPS; ++r) {
            a += s_run[r][0][lane];
            b += s_run[r][1][lane];
            sf += s_run[r][2][lane];
        }
        out[4 * v] = a;
        out[4 * v + 1] = b;
        out[4 * v + 2] = a * a + b * b;
        out[4 * v + 3] = sf;
    }
}

// ------------------------------------------------------------ form factors
// One thread per (form factor, grid point): the reference's FormFactor::eval
// (src/formfactor.rs:188-201) in FP64 on q_k = qmin + (qmax - qmin)·k/denom.
// Descriptor d: type, n, offset of its parameters in `params`; range [lo, hi].
// A point outside the range records the form factor's index + 1 in *bad.
__global__ void pd_ff_eval(const int32_t *__restrict__ desc, const double *__restrict__ range,
                           const double *__restrict__ params, int32_t n_ff, double qmin,
                           double qmax, int64_t nq, int *__restrict__ bad,
                           double *__restrict__ out) {
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (t >= n_ff * nq) return;
    const int f = static_cast<int>(t / nq);
    const int64_t k = t % nq;
    const double denom = static_cast<double>(nq > 1 ? nq - 1 : 1);
    const double q = qmin + (qmax - qmin) * static_cast<double>(k) / denom;
    const int type = desc[3 * f], n = desc[3 * f + 1];
    const double *p = params + desc[3 * f + 2];
    double v = 0.0;
    if (!(range[2 * f] <= q && q <= range[2 * f + 1])) {
        atomicMax(bad, f + 1);
    } else if (type == PD_FF_CONSTANT) {
        v = p[0];
    } else if (type == PD_FF_GAUSSIAN) {
        const double PI = 3.14159265358979323846;
        const double s2 = q * q / (16.0 * PI * PI);
        double sum = 0.0;
        for (int i = 0; i < n; ++i) sum += p[1 + 2 * i] * exp(-p[2 + 2 * i] * s2);
        v = sum + p[0];
    } else if (type == PD_FF_SINGLE_GAUSSIAN) {
        v = p[0] * exp(-p[1] * q * q);
    } else if (type == PD_FF_POLYNOMIAL) {
        double sum = 0.0;
        for (int i = 0; i < n; ++i) {
            double pw = 1.0;
            for (int e = 0; e < i; ++e) pw *= q;  // q^i by repeated products (Rust powi)
            sum += p[i] * pw;
        }
        v = sum;
    } else if (type == PD_FF_TABLE) {
        const double *xs = p, *ys = p + n;
        int low = 0, high = n - 1;
        bool hit = false;
        while (low < high) {
            const int mid = (low + high) / 2;
            if (q < xs[mid]) {
                high = mid;
            } else if (q > xs[mid]) {
                low = mid + 1;
            } else {
                v = ys[mid];
                hit = true;
                break;
            }
        }
        if (!hit) {
            if (low == 0) {  // q == xs[0] is a hit; below xs[0] is out of range
                v = ys[0];
            } else {
                const double x0 = xs[low - 1], y0 = ys[low - 1], x1 = xs[low], y1 = ys[low];
                v = y0 + (q - x0) * (y1 - y0) / (x1 - x0);
            }
        }
    }
    out[t] = v;
}

// ------------------------------------------------------------ FP32 probe
// Register-only FFMA throughput: 8 independent chains per thread.
__global__ void pd_ffma_probe(float *out, int iters, float a, float b) {
    float v[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = threadIdx.x * 1e-3f + c;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int u = 0; u < 16; ++u)
#pragma unroll
            for (int c = 0; c < 8; ++c) v[c] = fmaf(v[c], a, b);
    }
    float s = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) s += v[c];
    if (s == 12345.678f) out[0] = s;
}

// Same with packed FP32x2 FMAs (fma.rn.f32x2, sm_100a).
__global__ void pd_ffma2_probe(float *out, int iters, float a, float b) {
    unsigned long long v[8];
    float2 init;
    unsigned long long av, bv;
    {
        float2 t = make_float2(a, a);
        av = *reinterpret_cast<unsigned long long *>(&t);
        t = make_float2(b, b);
        bv = *reinterpret_cast<unsigned long long *>(&t);
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        init = make_float2(threadIdx.x * 1e-3f + c, c * 0.5f);
        v[c] = *reinterpret_cast<unsigned long long *>(&init);
    }
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int u = 0; u < 16; ++u)
#pragma unroll
            for (int c = 0; c < 8; ++c)
                asm volatile("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(v[c]) : "l"(av), "l"(bv));
    }
    float s = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        float2 t = *reinterpret_cast<float2 *>(&v[c]);
        s += t.x + t.y;
    }
    if (s == 12345.678f) out[0] = s;
}

// ------------------------------------------------------------ launchers
template <int K, int MODE, int NP>
static cudaError_t fp32_smem_attr() {
    // Above 48 KB of dynamic shared memory needs the opt-in attribute, set
    // once per device (the occupancy query sets it before any stream capture).
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = dev < 64 ? (uint64_t{1} << dev) : 0;
    if (bit && (done.load() & bit)) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(pd_pairs_fp32<K, MODE, NP>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(PD_FP32_DYN_SMEM));
    if (e == cudaSuccess && bit) done.fetch_or(bit);
    return e;
}
template <int K, int MODE, int NP>
static cudaError_t launch_fp32_t(const PdJob *jobs, const int *n_jobs, const PdReqDev *reqs,
                                 int *counter, int plan_frames, int grid, cudaStream_t st,
                                 bool after) {
    cudaError_t e = fp32_smem_attr<K, MODE, NP>();
    if (e != cudaSuccess) return e;
    return chain_launch(after, pd_pairs_fp32<K, MODE, NP>, grid, PD_THREADS, PD_FP32_DYN_SMEM, st,
                        jobs, n_jobs, reqs, counter, plan_frames);
}
template <int K, int MODE>
static cudaError_t launch_fp64_t(const PdJob *jobs, const int *n_jobs, const PdReqDev *reqs,
                                 int *counter, int plan_frames, int grid, cudaStream_t st,
                                 bool after) {
    return chain_launch(after, pd_pairs_fp64<K, MODE>, grid, PD_THREADS, 0, st, jobs, n_jobs, reqs,
                        counter, plan_frames);
}
template <int K, int MODE, int NP>
static int occupancy_fp32() {
    int n = 0;
    if (fp32_smem_attr<K, MODE, NP>() != cudaSuccess) return 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, pd_pairs_fp32<K, MODE, NP>, PD_THREADS,
                                                  PD_FP32_DYN_SMEM);
    return n;
}
template <int K, int MODE>
static int occupancy_fp64() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, pd_pairs_fp64<K, MODE>, PD_THREADS, 0);
    return n;
}

// (K, NP) shapes instantiated for the FP32 form; the weighted mode (two
// accumulators per q) only up to K = 64 to stay within 255 registers.
bool valid_shape(int precision, int mode, int K, int NP) {
    if (precision == 1) return (K == 16 || K == 32) && NP == 1;
    if (mode == PD_MODE_WEIGHTED) return (K == 32 && NP == 2) || (K == 64 && (NP == 2 || NP == 4));
    return (K == 32 && NP == 4) || (K == 64 && NP >= 1 && NP != 3) || (K == 96 && NP == 2) ||
           (K == 128 && NP >= 1 && NP != 3) || ((K == 160 || K == 192) && NP == 1);
}

bool valid_q_block(int precision, int K) {
    if (precision == 1) return K == 16 || K == 32;
    return K == 32 || K == 64 || K == 96 || K == 128 || K == 160 || K == 192;
}

#define PD_F32(K, M, NP)                                                                 \
    if (K_ == K && mode == M && NP_ == NP)                                               \
        return launch_fp32_t<K, M, NP>(jobs, n_jobs, reqs, counter, plan_frames, grid, st, after);
#define PD_F64(K, M) \
    if (K_ == K && mode == M) \
        return launch_fp64_t<K, M>(jobs, n_jobs, reqs, counter, plan_frames, grid, st, after);

cudaError_t launch_pairs(int precision, int K_, int NP_, int mode, const PdJob *jobs,
                         const int *n_jobs, const PdReqDev *reqs, int *counter, int plan_frames,
                         int grid, cudaStream_t st, bool after) {
    if (precision == 1) {
        PD_F64(16, 0) PD_F64(16, 1) PD_F64(32, 0) PD_F64(32, 1)
        return cudaErrorInvalidValue;
    }
    PD_F32(32, 0, 4) PD_F32(64, 0, 1) PD_F32(64, 0, 2) PD_F32(64, 0, 4) PD_F32(96, 0, 2)
    PD_F32(128, 0, 1) PD_F32(128, 0, 2) PD_F32(128, 0, 4) PD_F32(160, 0, 1) PD_F32(192, 0, 1)
    PD_F32(32, 1, 2) PD_F32(64, 1, 2) PD_F32(64, 1, 4)
    return cudaErrorInvalidValue;
}

#define PD_O32(K, M, NP) \
    if (K_ == K && mode == M && NP_ == NP) return occupancy_fp32<K, M, NP>();
#define PD_O64(K, M) \
    if (K_ == K && mode == M) return occupancy_fp64<K, M>();

int pairs_blocks_per_sm(int precision, int K_, int NP_, int mode) {
    if (precision == 1) {
        PD_O64(16, 0) PD_O64(16, 1) PD_O64(32, 0) PD_O64(32, 1)
        return 0;
    }
    PD_O32(32, 0, 4) PD_O32(64, 0, 1) PD_O32(64, 0, 2) PD_O32(64, 0, 4) PD_O32(96, 0, 2)
    PD_O32(128, 0, 1) PD_O32(128, 0, 2) PD_O32(128, 0, 4) PD_O32(160, 0, 1) PD_O32(192, 0, 1)
    PD_O32(32, 1, 2) PD_O32(64, 1, 2) PD_O32(64, 1, 4)
    return 0;
}

cudaError_t prepare_pair_kernels() {
    const int shapes[][3] = {{32, 0, 4},  {64, 0, 1},  {64, 0, 2},  {64, 0, 4},
                             {96, 0, 2},  {128, 0, 1}, {128, 0, 2}, {128, 0, 4},
                             {160, 0, 1}, {192, 0, 1}, {32, 1, 2},  {64, 1, 2},
                             {64, 1, 4}};
    for (const auto &sh : shapes)
        if (pairs_blocks_per_sm(0, sh[0], sh[2], sh[1]) <= 0) return cudaErrorInvalidValue;
    for (const int v : {0, 64, 128})
        if (directions_blocks_per_sm(v) <= 0) return cudaErrorInvalidValue;
    return cudaSuccess;
}

int32_t centroid_blocks(int64_t n_atoms) {
    return static_cast<int32_t>(
        std::min<int64_t>(std::max<int64_t>((n_atoms + PD_CENT_RUN - 1) / PD_CENT_RUN, 1), 256));
}

cudaError_t launch_pack(const double *xyz, const double *weights, const int32_t *perm,
                        int64_t n_atoms, int32_t n_pad, int32_t n_frames, double *part,
                        unsigned int *cent_done, double *centroid, int32_t *status, float4 *out32,
                        double4 *out64, const PdMomentRule &rule, unsigned long long *rad2,
                        unsigned int *done, PdFrameDev *frames, double4 *dirs, double2 *node_tab,
                        cudaStream_t st, int *launches) {
    if (n_pad <= PD_FRAME_MAX && n_frames <= 0x7fffffff / PD_FRAME_CTAS) {
        *launches = 1;
        return chain_launch(false, pd_pack_frames, static_cast<unsigned>(n_frames) * PD_FRAME_CTAS,
                            PD_FRAME_THREADS, 0, st, xyz, weights, perm,
                            static_cast<int32_t>(n_atoms), n_pad, out32, out64, rule, frames, dirs,
                            node_tab, status);
    }
    *launches = 2;
    const int32_t nc = centroid_blocks(n_atoms);
    const int64_t nb = (static_cast<int64_t>(n_pad) + PD_PACK_THREADS - 1) / PD_PACK_THREADS;
    if (nb * n_frames > 0x7fffffffLL) return cudaErrorInvalidValue;
    const cudaError_t e =
        chain_launch(false, pd_centroid, static_cast<unsigned>(n_frames) * nc, PD_CENT_THREADS, 0,
                     st, xyz, n_atoms, nc, part, cent_done, centroid, status);
    if (e != cudaSuccess) return e;
    return chain_launch(true, pd_pack, static_cast<unsigned>(nb * n_frames), PD_PACK_THREADS, 0, st,
                        xyz, weights, perm, centroid, n_atoms, n_pad, static_cast<int32_t>(nb),
                        out32, out64, rule, rad2, done, frames, dirs, node_tab);
}

// Gauss–Legendre rules: Newton's method on P_2h from Tricomi's estimate, in
// long double, once per process; copied to each device that asks.
cudaError_t prepare_direction_rules() {
    static std::mutex mu;
    static std::vector<double2> rules;
    static uint64_t done = 0;
    std::lock_guard<std::mutex> g(mu);
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = dev < 64 ? (uint64_t{1} << dev) : 0;
    if (bit && (done & bit)) return cudaSuccess;
    if (rules.empty()) {
        rules.resize(PD_GL_MAX * (PD_GL_MAX + 1) / 2);
        for (int h = 1; h <= PD_GL_MAX; ++h) {
            const int n = 2 * h;
            for (int i = 0; i < h; ++i) {  // i-th largest node
                long double x = cosl(3.14159265358979323846264L * (i + 0.75L) / (n + 0.5L));
                long double dp = 1.0L;
                for (int it = 0; it < 6; ++it) {
                    long double p0 = 1.0L, p1 = x;
                    for (int k = 2; k <= n; ++k) {
                        const long double p2 = ((2 * k - 1) * x * p1 - (k - 1) * p0) / k;
                        p0 = p1;
                        p1 = p2;
                    }
                    dp = n * (x * p1 - p0) / (x * x - 1.0L);
                    const long double dx = p1 / dp;
                    x -= dx;
                    if (fabsl(dx) < 1e-12L) break;  // quadratic: the next step is below the last bit
                }
                {
                    long double p0 = 1.0L, p1 = x;
                    for (int k = 2; k <= n; ++k) {
                        const long double p2 = ((2 * k - 1) * x * p1 - (k - 1) * p0) / k;
                        p0 = p1;
                        p1 = p2;
                    }
                    dp = n * (x * p1 - p0) / (x * x - 1.0L);
                }
                double2 &r = rules[h * (h - 1) / 2 + (h - 1 - i)];
                r.x = static_cast<double>(x);
                r.y = static_cast<double>(2.0L / ((1.0L - x * x) * dp * dp));
            }
            long double sum = 0.0L;
            for (int i = 0; i < h; ++i) sum += rules[h * (h - 1) / 2 + i].y;
            for (int i = 0; i < h; ++i)
                rules[h * (h - 1) / 2 + i].y = static_cast<double>(rules[h * (h - 1) / 2 + i].y / sum);
        }
    }
    const cudaError_t e =
        cudaMemcpyToSymbol(pd_gl_rules, rules.data(), rules.size() * sizeof(double2));
    if (e == cudaSuccess) done |= bit;
    return e;
}

cudaError_t launch_direction_sums(const double *slots, const double4 *dirs,
                                  const PdFrameDev *frames, const PdAmpShape &sh, double qmax,
                                  const double *qv, int32_t n_frames, const PdClassDev *cls,
                                  const PdPairDev *pairs,
                                  int32_t n_pairs, const int32_t *cls_ptr,
                                  const int32_t *cls_chunk, int32_t width,
                                  int add_exact, double *part, unsigned int *done, double *red,
                                  cudaStream_t st, bool after) {
    const size_t smem = static_cast<size_t>(sh.sum_smem) * sizeof(double);
    auto kern = sh.nv2 == 2 ? pd_direction_sums<2> : pd_direction_sums<1>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         PD_DIR_SMEM);
    if (e != cudaSuccess) return e;
    if (smem > PD_DIR_SMEM) return cudaErrorInvalidValue;
    const int64_t n_nt = (sh.node_cap + sh.node_tile - 1) / sh.node_tile;
    const int64_t nv = sh.nv2 == 2 ? 4 : 1;
    for (int32_t f0 = 0; f0 < n_frames; f0 += 65535) {  // grid.y limit
        const dim3 grid(static_cast<unsigned>(n_nt * sh.grp_cap),
                        static_cast<unsigned>(std::min(n_frames - f0, 65535)));
        e = chain_launch(
            after, kern, grid, PD_DSUM_THREADS, smem, st, slots + f0 * sh.slot_cap,
            dirs + static_cast<int64_t>(f0) * sh.dir_cap, frames + f0, sh,
            qmax, qv, cls, pairs, n_pairs, cls_ptr, cls_chunk, width, add_exact,
            part + f0 * static_cast<int64_t>(sh.grp_cap) * n_pairs * nv * sh.node_cap,
            done + f0 * n_nt, red + f0 * static_cast<int64_t>(n_pairs) * nv * width);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_reduce(const double *slots, const int64_t *lptr, const int64_t *lidx,
                          const PdPairDev *pairs, const double *qv, const PdFrameDev *frames,
                          const PdReduceShape &sh, int32_t nv, int32_t n_frames, int residual_form,
                          int add_exact, double *chunk_sums, unsigned int *done, double *red,
                          cudaStream_t st, bool after) {
    const int64_t blocks = static_cast<int64_t>(n_frames) * sh.n_pairs * sh.n_z;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    const dim3 grid(static_cast<unsigned>(blocks), static_cast<unsigned>(sh.n_chunk));
    return chain_launch(after, nv == 4 ? pd_reduce_pairs<4> : pd_reduce_pairs<1>, grid,
                        PD_RED_THREADS, 0, st, slots, lptr, lidx, pairs, qv, frames, sh,
                        residual_form, add_exact, chunk_sums, done, red);
}

cudaError_t launch_profiles(const double *red, const double *lat_sums, const PdClassDev *cls,
                            const PdPairDev *pairs, int32_t n_cls, const PdReduceShape &sh,
                            int32_t nv, int32_t n_frames, const double *qv,
                            const PdFrameDev *frames, const double2 *node_tab, const double *ffA,
                            const double *ffC, const double *ffW, int add_diag, double qmax, const int *err,
                            double *terms, cudaStream_t st, bool after) {
    const int64_t blocks =
        static_cast<int64_t>(n_frames) * ((sh.nq + PD_PROF_Q - 1) / PD_PROF_Q);
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    const bool staged = profile_smem(sh, PD_PROF_ROWS, n_cls) <= PD_PROF_SMEM;
    const int64_t all = static_cast<int64_t>(sh.n_pairs) * nv * sh.max_moments;
    const int rows = all <= 4 * PD_PROF_ROWS || blocks > 3 * 148 ? PD_PROF_ROWS
                     : blocks > 148                              ? PD_PROF_ROWS_MANY
                                                                 : PD_PROF_ROWS_MOST;
    const size_t smem = profile_smem(sh, rows, staged ? n_cls : 0);
    auto kern = nv == 4 ? (staged ? pd_profiles<4, true> : pd_profiles<4, false>)
                        : (staged ? pd_profiles<1, true> : pd_profiles<1, false>);
    if (smem > 44 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(
            kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e != cudaSuccess) return e;
    }
    return chain_launch(after, kern, static_cast<unsigned>(blocks), PD_PROF_THREADS, smem, st, red,
                        lat_sums, cls, pairs, n_cls, sh, qv, frames, node_tab, ffA, ffC, ffW,
                        add_diag, qmax, rows, err, terms);
}

cudaError_t launch_lattice(const double *xyz, const int32_t *perm, const PdLatDev *lat_dev,
                           const PdLatDev *lat_host, int n_lat, const PdLatTile *tiles,
                           int64_t n_tiles, int4 *idx, unsigned long long *hist, int64_t n_bins,
                           int *err, cudaStream_t st) {
    if (n_lat == 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(hist, 0, static_cast<size_t>(n_bins) * 8, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    int max_n = 1, max_bins = 1;
    for (int l = 0; l < n_lat; ++l) {
        max_n = max(max_n, lat_host[l].n);
        max_bins = max(max_bins, lat_host[l].n_bins);
    }
    const dim3 g1(static_cast<unsigned>(min((max_n + 255) / 256, 4096)), n_lat);
    pd_lattice_index<<<g1, 256, 0, st>>>(xyz, perm, lat_dev, idx, err);
    if ((e = cudaGetLastError()) != cudaSuccess || n_tiles == 0) return e;
    // shared-memory histogram when the bins fit (opt-in limit of the device)
    int dev = 0, smem_optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const size_t need = static_cast<size_t>(max_bins) * 4;
    int shared_bins = need <= static_cast<size_t>(smem_optin) ? max_bins : 0;
    size_t smem = shared_bins ? need : 0;
    if (smem > 48 * 1024) {
        e = cudaFuncSetAttribute(pd_lattice_hist, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem));
        if (e != cudaSuccess) {
            (void)cudaGetLastError();
            shared_bins = 0;
            smem = 0;
        }
    }
    pd_lattice_hist<<<static_cast<unsigned>(n_tiles), 128, smem, st>>>(tiles, lat_dev, idx, hist,
                                                                        shared_bins);
    return cudaGetLastError();
}

cudaError_t launch_lattice_sums(const unsigned long long *hist, const PdLatDev *lat, int n_lat,
                                const double *qv, int32_t nq, int add_exact, const int *err,
                                double *sums, cudaStream_t st) {
    if (n_lat == 0) return cudaSuccess;
    pd_lattice_sums<<<dim3(nq, n_lat), 256, 0, st>>>(hist, lat, qv, nq, add_exact, err, sums);
    return cudaGetLastError();
}

cudaError_t launch_frame_mean(const double *terms, const double *fw, int32_t n_frames, int32_t nq,
                              double *out, cudaStream_t st, bool normalize, bool after) {
    const int grid = (6 * nq + 127) / 128;
    return chain_launch(after, pd_frame_mean, grid, 128, 0, st, terms, fw, n_frames, nq,
                        normalize ? 1 : 0, out);
}

cudaError_t launch_stream_accumulate(const double *batch, double scale, int32_t n, double *acc,
                                     cudaStream_t st) {
    pd_stream_accumulate<<<(n + 127) / 128, 128, 0, st>>>(batch, scale, n, acc);
    return cudaGetLastError();
}

// Chunking of n_points points in molecules of mol_size for n_vec vectors:
// (points per chunk, slices per molecule, number of chunks).
static void direct_layout(int64_t n_points, int64_t mol_size, int64_t n_vec, int64_t *chunk,
                          int64_t *spm, int64_t *n_chunks) {
    const int64_t vblocks = (n_vec + PD_DIRECT_V * PD_DIRECT_THREADS - 1) /
                            (PD_DIRECT_V * PD_DIRECT_THREADS);
    for (int64_t len = PD_DIRECT_CHUNK_MAX;; len /= 2) {
        if (mol_size <= len) {
            *chunk = (len / mol_size) * mol_size;
            *spm = 1;
            *n_chunks = (n_points + *chunk - 1) / *chunk;
        } else {
            *chunk = len;
            *spm = (mol_size + len - 1) / len;
            *n_chunks = (n_points / mol_size) * *spm;
        }
        if (len <= PD_DIRECT_CHUNK_MIN || *n_chunks * vblocks >= PD_DIRECT_BLOCKS) return;
    }
}

int64_t direct_chunks(int64_t n_points, int64_t mol_size, int64_t n_vec) {
    int64_t chunk, spm, n;
    direct_layout(n_points, mol_size, n_vec, &chunk, &spm, &n);
    return n;
}

int64_t direct_blocks(int64_t n_points, int64_t mol_size, int64_t n_vec) {
    const int64_t vblocks = (n_vec + PD_DIRECT_V * PD_DIRECT_THREADS - 1) /
                            (PD_DIRECT_V * PD_DIRECT_THREADS);
    return direct_chunks(n_points, mol_size, n_vec) * vblocks;
}

cudaError_t launch_direct(const double *xyz, const uint32_t *kind, const double *weight,
                          const double *ff, int32_t n_kinds, const double *qvec, int64_t n_vec,
                          int64_t n_points, int64_t mol_size, double *part, int64_t part_chunks,
                          double *out, cudaStream_t st) {
    int64_t chunk, spm, n_chunks;
    direct_layout(n_points, mol_size, n_vec, &chunk, &spm, &n_chunks);
    constexpr int64_t per_block = PD_DIRECT_V * PD_DIRECT_THREADS;
    const int64_t vblocks = (n_vec + per_block - 1) / per_block;
    if (n_chunks > part_chunks || n_vec < 1 || n_chunks * vblocks > 0x7fffffffLL)
        return cudaErrorInvalidValue;
    pd_direct_chunks<<<static_cast<unsigned>(n_chunks * vblocks), PD_DIRECT_THREADS, 0, st>>>(
        xyz, kind, weight, ff, qvec, n_vec, vblocks, mol_size, chunk, spm, n_points, n_kinds,
        part);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    pd_direct_reduce<<<static_cast<unsigned>((n_vec + 31) / 32), 32 * PD_DIRECT_RED_WARPS, 0, st>>>(
        part, n_vec, n_chunks, spm, out);
    return cudaGetLastError();
}

// Stage length of the table kernel for indices up to nmax (0 when a single
// point's table does not fit).
int direct_table_points(int32_t nmax) {
    const int64_t per_point = 3LL * (nmax + 1) * static_cast<int64_t>(sizeof(double2));
    return static_cast<int>(std::min<int64_t>(PD_DTAB_MAX_POINTS, PD_DTAB_TABLE_BYTES / per_point));
}

cudaError_t launch_direct_table(const double *xyz, const uint32_t *kind, const double *weight,
                                const double *ff, const int32_t *hkl, int32_t nmax,
                                const double box[3], int64_t n_vec, int64_t n_points,
                                int64_t mol_size, double *part, int64_t part_chunks, double *out,
                                cudaStream_t st) {
    const int npts = direct_table_points(nmax);
    if (npts < 1 || n_vec < 1) return cudaErrorInvalidValue;
    const int stride = nmax + 1;
    const size_t smem = static_cast<size_t>(npts) * 3 * stride * sizeof(double2);
    // above 48 KB of dynamic shared memory needs the opt-in, set once per device
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = dev < 64 ? (uint64_t{1} << dev) : 0;
    if (!bit || !(done.load() & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(
            pd_direct_table, cudaFuncAttributeMaxDynamicSharedMemorySize, PD_DTAB_TABLE_BYTES);
        if (e != cudaSuccess) return e;
        if (bit) done.fetch_or(bit);
    }
    int64_t chunk, spm, n_chunks;
    direct_layout(n_points, mol_size, n_vec, &chunk, &spm, &n_chunks);
    constexpr int64_t per_block = PD_DTAB_V * PD_DTAB_THREADS;
    const int64_t vblocks = (n_vec + per_block - 1) / per_block;
    if (n_chunks > part_chunks || n_chunks * vblocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    pd_direct_table<<<static_cast<unsigned>(n_chunks * vblocks), PD_DTAB_THREADS, smem, st>>>(
        xyz, kind, weight, ff, hkl, box[0], box[1], box[2], stride, npts, n_vec, vblocks,
        mol_size, chunk, spm, n_points, part);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    pd_direct_reduce<<<static_cast<unsigned>((n_vec + 31) / 32), 32 * PD_DIRECT_RED_WARPS, 0, st>>>(
        part, n_vec, n_chunks, spm, out);
    return cudaGetLastError();
}

int direct_line_points(int32_t n_entries) {
    return std::min(PD_DLINE_MAX_POINTS, static_cast<int>(PD_DLINE_TABLE_BYTES /
                                                          (n_entries * sizeof(double2))));
}

// Slices of a molecule for the line kernel: up to 4 blocks per SM (three are resident
// at its registers) where the box allows that, slices of 128 to 2,048 points.
void direct_line_layout(int64_t n_points, int64_t mol_size, int32_t n_line, int64_t *chunk,
                        int64_t *spm) {
    const int64_t vblocks = (n_line + PD_DLINE_THREADS - 1) / PD_DLINE_THREADS;
    const int64_t units = n_points / mol_size * vblocks;
    *spm = std::clamp<int64_t>(148 * 4 / units, (mol_size + 2047) / 2048,
                               std::max<int64_t>((mol_size + 127) / 128, 1));
    *chunk = (mol_size + *spm - 1) / *spm;
    *spm = (mol_size + *chunk - 1) / *chunk;
}

cudaError_t launch_direct_sort(const double *xyz, const uint32_t *kind, const double *weight,
                               int64_t n_points, int64_t mol_size, int32_t n_kinds,
                               double *xyz_out, uint32_t *kind_out, double *weight_out,
                               cudaStream_t st) {
    const size_t smem = static_cast<size_t>(n_kinds) * PD_DSORT_THREADS * sizeof(uint32_t);
    const int64_t pieces = (mol_size + PD_DSORT_PIECE - 1) / PD_DSORT_PIECE;
    const int64_t blocks = n_points / mol_size * pieces;
    if (smem > 46 * 1024 || blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    pd_direct_sort<<<static_cast<unsigned>(blocks), PD_DSORT_THREADS, smem, st>>>(
        xyz, kind, weight, mol_size, static_cast<int32_t>(pieces), n_kinds, xyz_out, kind_out,
        weight_out);
    return cudaGetLastError();
}

cudaError_t launch_direct_lines(const double *xyz, const uint32_t *kind, const double *weight,
                                const double *ff, const PdLine *lines, const int32_t *index,
                                const int32_t n_index[3], const double box[3], int32_t n_line,
                                int64_t n_points, int64_t mol_size, int64_t chunk, int64_t spm,
                                double *part, double *out, cudaStream_t st) {
    const int n_ent = n_index[0] + n_index[1] + n_index[2];
    const int npts = direct_line_points(n_ent);
    if (npts < 1 || n_line < 1) return cudaErrorInvalidValue;
    const int threads = std::min(PD_DLINE_THREADS, (n_line + 31) / 32 * 32);
    const int vblocks = (n_line + threads - 1) / threads;
    const int64_t n_mol = n_points / mol_size, blocks = n_mol * spm * vblocks;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    const size_t smem = static_cast<size_t>(npts) * n_ent * sizeof(double2) +
                        2 * PD_DLINE_J * static_cast<size_t>(threads) * sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(
        pd_direct_lines, cudaFuncAttributeMaxDynamicSharedMemorySize,
        PD_DLINE_TABLE_BYTES + 2 * PD_DLINE_J * PD_DLINE_THREADS * static_cast<int>(sizeof(double)));
    if (e != cudaSuccess) return e;
    pd_direct_lines<<<static_cast<unsigned>(blocks), threads, smem, st>>>(
        xyz, kind, weight, ff, lines, index, make_int3(n_index[0], n_index[1], n_index[2]), box[0],
        box[1], box[2], npts, n_line, vblocks, mol_size, chunk, spm, part);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    pd_direct_lines_reduce<<<static_cast<unsigned>((PD_DLINE_J * static_cast<int64_t>(n_line) + 31) /
                                                   32),
                             1024, 0, st>>>(part, n_line, n_mol, spm, out);
    return cudaGetLastError();
}

cudaError_t launch_ff_eval(const int32_t *desc, const double *range, const double *params,
                           int32_t n_ff, double qmin, double qmax, int64_t nq, int *bad,
                           double *out, cudaStream_t st) {
    const int64_t total = static_cast<int64_t>(n_ff) * nq;
    pd_ff_eval<<<static_cast<unsigned>((total + 127) / 128), 128, 0, st>>>(
        desc, range, params, n_ff, qmin, qmax, nq, bad, out);
    return cudaGetLastError();
}

cudaError_t launch_ffma_probe(float *out, int iters, int grid, int block, bool packed,
                              cudaStream_t st) {
    if (packed)
        pd_ffma2_probe<<<grid, block, 0, st>>>(out, iters, 0.999999f, 1e-7f);
    else
        pd_ffma_probe<<<grid, block, 0, st>>>(out, iters, 0.999999f, 1e-7f);
    return cudaGetLastError();
}

}  // namespace pd
