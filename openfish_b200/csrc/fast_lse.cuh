// fast_lse.cuh -- fp32 evaluation of the reference's five-term log-sum-exp that knows when it
// is right.
//
// The value-exact routine in exact_math.cuh costs about 63 FP64 operations per state and
// timestep.  Most of the time that effort is not needed to know which float the reference
// arithmetic produces: the result max + log(sum) is rounded to a float whose spacing grows with
// the magnitude of the scores (2^-12 once they pass 2048), while log(sum) can be had in fp32
// to about 2^-20.  So: evaluate log(sum) in fp32, widen it by a bound on every error that
// separates it from the reference's own value, add both ends of that interval to the maximum
// with one correctly rounded float addition each, and accept when both ends land on the same
// float (rounding is monotone, so the reference's result is pinned between them).  Otherwise
// the caller falls back to the value-exact routine.  Nothing is approximated in what is
// accepted.
//
// Error budget of log(sum), all relative to sum >= 1 (so also absolute in the logarithm), in
// units of 1e-7:
//   ex2.approx: 2 ulp = 2^-22 documented (2^-22.7 measured), weights sum to one        2.38
//   rounding of (v-m)*log2(e) before ex2, weighted by the term's size
//     (max a*exp(-a) = 0.37, 4 terms)                                                   0.88
//   four float additions here, each relative to a partial sum                           2.38
//   the reference's five float roundings of its running sum (decode_cpu.c:47)           2.98
//   lg2.approx on [1,8): at most 2^-21.75 absolute in log2, its own rounding included
//     (measured over every float of the interval: 2^-21.78), times ln 2                 1.96
//   rounding of the product with ln 2 and of l -+ eps (l < 2)                           1.19
// Sum 11.8 = 2^-19.7; kLseEps = 13.5 = 2^-19.5.  openfish_b200_selfcheck_arith repeats the two
// measurements on the GPU at hand and compares them with the bounds used here.
#pragma once
#include <cuda_runtime.h>

#include "exact_math.cuh"

namespace ofd {

constexpr float kLseEps = 1.3487e-6f;  // 2^-19.5
// The same with the logarithm out of a table (lse5_guess_pairs) instead of lg2.approx: the table's
// error and the truncation after the third term, below 2^-26 each (tests/test_exact_math_host.py goes through
// the floats), take the place of the 1.96.  Sum 10.2; 11.2 = 2^-19.77.
constexpr float kGuessEps = 1.12e-6f;

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// maximum of three in one instruction (sm_100); a NaN operand loses against a number, as in fmaxf
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float max5(const float v[5]) { return max3(max3(v[0], v[1], v[2]), v[3], v[4]); }
__device__ __forceinline__ float lg2_approx(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// ln of s in [1, 8).
__device__ __forceinline__ float ln_1to8(float s) {
    const float kLn2 = 0.6931471805599453f;
    return lg2_approx(s) * kLn2;
}

// v: the five terms.  On success writes the reference-exact float to `out`.
__device__ __forceinline__ bool lse5_try_fast(const float v[5], float &out) {
    const float kLog2e = 1.4426950408889634f;
    const float m = max5(v);
    float s = ex2_approx((v[0] - m) * kLog2e);
    s += ex2_approx((v[1] - m) * kLog2e);
    s += ex2_approx((v[2] - m) * kLog2e);
    s += ex2_approx((v[3] - m) * kLog2e);
    s += ex2_approx((v[4] - m) * kLog2e);
    const float l = ln_1to8(s);
    const float lo = m + (l - kLseEps);
    const float hi = m + (l + kLseEps);
    out = lo;
    // A NaN or infinite term makes the sum NaN (an infinite maximum gives inf - inf in its own
    // term), the logarithm and both ends with it, and NaN compares unequal.
    return lo == hi;
}

}  // namespace ofd

namespace ofd {

// Two floats in a register pair, for the packed additions and multiplications of sm_100 (each half is
// an ordinary rounded operation; a pair costs one issue slot).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The logarithm of a guess: s = c * (1 + u) with 1/c a float out of a table of 64 intervals a binade
// and log(c) a multiple of 2^-11 to within 2^-26 (exact_math.cuh, fill_tables, chooses c so), so that
// adding log(c) to a float of the size the scores have is exact and log1p(u), |u| <= 2^-6, needs three
// terms.  (lg2.approx, with its 2^-22, makes the likelier candidate the wrong one four times as often.)
constexpr int kLogPairs = ofx::kLogTab;
struct LogPair { float rcp, log; };

// K (even) fast evaluations, two states in every packed operation.  out[k] is the certified result
// where bit k of the returned mask is clear, and otherwise the better of the two candidate floats
// (the one nearest to max + log(sum) as estimated), to be confirmed by the value-exact routine.  The
// sum takes the terms in the reference's order, which makes the guess right more often.
// TABLE: the logarithm out of the table (its look-up and two more terms of arithmetic take 60 cycles of a
// warp's timestep, which pays for rows of 256 states and not for rows of 64).
template <int K, bool TABLE>
__device__ __forceinline__ uint32_t lse5_guess_pairs(const float (*v)[5], float *out, const LogPair *tab) {
    const float kLog2e = 1.4426950408889634f;
    const f32x2 log2e = pack2(kLog2e, kLog2e), eps = pack2(TABLE ? kGuessEps : kLseEps, TABLE ? kGuessEps : kLseEps), one = pack2(1.f, 1.f);
    const f32x2 third = pack2(1.f / 3.f, 1.f / 3.f), half = pack2(0.5f, 0.5f), neg_one = pack2(-1.f, -1.f);
    f32x2 m[K / 2];
    float e[K][5];
    uint32_t bad = 0;
#pragma unroll
    for (int p = 0; p < K / 2; ++p) m[p] = pack2(max5(v[2 * p]), max5(v[2 * p + 1]));
#pragma unroll
    for (int p = 0; p < K / 2; ++p)
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            float a, b;
            unpack2(mul2(sub2(pack2(v[2 * p][i], v[2 * p + 1][i]), m[p]), log2e), a, b);
            e[2 * p][i] = ex2_approx(a);
            e[2 * p + 1][i] = ex2_approx(b);
        }
#pragma unroll
    for (int p = 0; p < K / 2; ++p) {
        f32x2 s = pack2(e[2 * p][0], e[2 * p + 1][0]);
#pragma unroll
        for (int i = 1; i < 5; ++i) s = add2(s, pack2(e[2 * p][i], e[2 * p + 1][i]));
        float s0, s1, g0, g1, lo0, lo1, hi0, hi1;
        unpack2(s, s0, s1);
        if constexpr (!TABLE) {
            const f32x2 ln2 = pack2(0.6931471805599453f, 0.6931471805599453f);
            const f32x2 l = mul2(pack2(lg2_approx(s0), lg2_approx(s1)), ln2);
            unpack2(add2(m[p], l), out[2 * p], out[2 * p + 1]);
            unpack2(add2(m[p], sub2(l, eps)), lo0, lo1);
            unpack2(add2(m[p], add2(l, eps)), hi0, hi1);
            bad |= lo0 == hi0 ? 0u : 1u << (2 * p);
            bad |= lo1 == hi1 ? 0u : 2u << (2 * p);
            continue;
        }
        // (anything but a number in [1, 8) can only come from terms that are not numbers: any entry will do)
        const uint32_t i0 = min((__float_as_uint(s0) >> 17) - (127u << 6), (uint32_t)(kLogPairs - 1));
        const uint32_t i1 = min((__float_as_uint(s1) >> 17) - (127u << 6), (uint32_t)(kLogPairs - 1));
        const LogPair c0 = tab[i0], c1 = tab[i1];
        const f32x2 logc = pack2(c0.log, c1.log);
        const f32x2 u = fma2(s, pack2(c0.rcp, c1.rcp), neg_one);
        const f32x2 w = fma2(sub2(mul2(u, third), half), u, one);  // log1p(u) = u * w
        const f32x2 b = mul2(u, w);
        const f32x2 l = add2(logc, b);
        unpack2(add2(add2(m[p], logc), b), g0, g1);
        unpack2(add2(m[p], sub2(l, eps)), lo0, lo1);
        unpack2(add2(m[p], add2(l, eps)), hi0, hi1);
        // (a NaN sum makes both ends NaN: never accepted.  Where the maximum plus log(c) is not exact, as
        // on the way across a power of two, the guess may lie outside the interval: a certified state
        // takes its end, not the guess.)
        const bool ok0 = lo0 == hi0, ok1 = lo1 == hi1;
        out[2 * p] = ok0 ? lo0 : g0;
        out[2 * p + 1] = ok1 ? lo1 : g1;
        bad |= ok0 ? 0u : 1u << (2 * p);
        bad |= ok1 ? 0u : 2u << (2 * p);
    }
    return bad;
}

}  // namespace ofd
