/*
 * Correctly rounded FP64 division, square root and reciprocal square root
 * on the integer and FP32 pipes.
 *
 * GB300 issues FP64 instructions at 1.7 lanes per clock and SM (measured: a
 * warp instruction every 19 clocks, 64 clocks on one scheduler); a / b costs
 * 7.2 of those slots, sqrt 7.5, 1 / sqrt 12, a comparison 1.  The integer
 * pipes are 40x wider and idle in the FP64 kernels.  The canonical
 * arithmetic (canon_math.h) needs the IEEE results, not a particular way to
 * them, so they are computed here from the operands' bits:
 *   - a 22-bit reciprocal (square root) from the FP32 unit;
 *   - one Newton step in 64-bit fixed point: about 44 bits;
 *   - the quotient (root) to 54 bits, corrected by its EXACT integer
 *     remainder, which fits 64 bits modulo 2^64 because the estimate is close;
 *   - round to nearest by adding the 54th bit: a quotient of 53-bit
 *     significands, a square root and a reciprocal never lie half way between
 *     two doubles (the odd 54-bit half-way point times the divisor, or
 *     squared, has more than 53 significant bits).
 * Newton's iteration and the remainder correction are the textbook methods
 * (Muller et al., Handbook of Floating-Point Arithmetic, 2018, ch. 4-5); the
 * error bounds are worked out at each step.  Operands outside the normal
 * range (zeros, subnormals, infinities, NaN) and results near its ends take
 * the FP64 instruction sequence of the compiler (fallback()).  Measured with
 * it and the comparisons below, per FIRE step of the grid kernel: 1 048 576
 * nodes 595 -> 412 us, 197 246-node Mikado 195 -> 136 us.  The same code
 * compiles for the host, where the tests compare it with the host's IEEE
 * operations, the FP32 estimate perturbed by its error bound.
 */
#ifndef NR_IEEE_INT_H
#define NR_IEEE_INT_H

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define NR_IHD __host__ __device__ __forceinline__
#else
#define NR_IHD inline
#endif

namespace nr {

/* On the device through the high / low word intrinsics: the compiler turns
 * tests and masks of a plain bit cast back into FP64 comparisons, negations
 * and absolute values, a slot each. */
NR_IHD uint64_t ii_bits(double v) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)(uint32_t)__double2hiint(v) << 32 | (uint32_t)__double2loint(v);
#else
    uint64_t u;
    memcpy(&u, &v, 8);
    return u;
#endif
}
NR_IHD double ii_double(uint64_t u) {
#if defined(__CUDA_ARCH__)
    return __hiloint2double((int)(uint32_t)(u >> 32), (int)(uint32_t)u);
#else
    double v;
    memcpy(&v, &u, 8);
    return v;
#endif
}
#if !defined(__CUDA_ARCH__)
/* Host: the FP32 estimate moved by this many units in the last place (the
 * tests sweep it over the device's error: one for rcp, two for rsqrt). */
inline int &ii_nudge() {
    static thread_local int n = 0;
    return n;
}
#endif

/* FP32 estimates of 1 / f, f in [1, 2], and 1 / sqrt(f), f in [1, 4], as
 * Q32 fixed point in [2^31, 2^32).  f is the significand rounded to 24 bits;
 * with it the relative error e0 is below 2^-22 (rcp.approx: 1 ulp;
 * rsqrt.approx: 2^-22.9, at most 2.1 units of 2^-24).  Over all f on GB300:
 * within one unit and two units of the rounded value.  (Estimates moved by three
 * units break the bound for values near 1/2, and quotients come out wrong.) */
NR_IHD uint32_t ii_q32(uint32_t fbits) {
    /* kept within [1/2, 1): the ends of the range by a step */
    fbits = fbits > 0x3f7fffffu ? 0x3f7fffffu : fbits < 0x3f000000u ? 0x3f000000u : fbits;
    return (fbits << 8) | 0x80000000u;
}
NR_IHD uint32_t ii_rcp_q32(uint32_t f) {
#if defined(__CUDA_ARCH__)
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(f)));
    return ii_q32(__float_as_uint(y));
#else
    float x, y;
    memcpy(&x, &f, 4);
    y = 1.0f / x;
    uint32_t u;
    memcpy(&u, &y, 4);
    return ii_q32(u + (uint32_t)ii_nudge());
#endif
}
NR_IHD uint32_t ii_rsqrt_q32(uint32_t f) {
#if defined(__CUDA_ARCH__)
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(f)));
    return ii_q32(__float_as_uint(y));
#else
    float x, y;
    memcpy(&x, &f, 4);
    y = (float)(1.0 / sqrt((double)x));
    uint32_t u;
    memcpy(&u, &y, 4);
    return ii_q32(u + (uint32_t)ii_nudge());
#endif
}

/* The compiler's FP64 sequences, out of line: one copy per kernel. */
#if defined(__CUDACC__)
static __host__ __device__ __noinline__ double ii_div_fallback(double a, double b) { return a / b; }
static __host__ __device__ __noinline__ double ii_sqrt_fallback(double q) { return sqrt(q); }
#else
static inline double ii_div_fallback(double a, double b) { return a / b; }
static inline double ii_sqrt_fallback(double q) { return sqrt(q); }
#endif

constexpr uint64_t kIiFrac = 0x000fffffffffffffULL, kIiOne = 0x0010000000000000ULL;

/* The pieces are 32-bit: a 64-bit multiply, shift or select is several
 * instructions.  ii_div takes about 50, ii_inv_sqrt about 75 (2 and 3 FP64
 * slots of issue time against 7.2 and 12 on the FP64 pipe). */
NR_IHD uint32_t ii_hi(uint64_t v) { return (uint32_t)(v >> 32); }
NR_IHD uint32_t ii_lo(uint64_t v) { return (uint32_t)v; }
NR_IHD uint64_t ii_join(uint32_t hi, uint32_t lo) { return (uint64_t)hi << 32 | lo; }
NR_IHD uint64_t ii_wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
NR_IHD int64_t ii_wides(int32_t a, int32_t b) { return (int64_t)a * b; }
/* High 64 bits of a b, low by at most 3 (the low partial product is left
 * out, the middle ones are truncated). */
NR_IHD uint64_t ii_mulhi_low3(uint64_t a, uint64_t b) {
    return ii_wide(ii_hi(a), ii_hi(b)) + (ii_wide(ii_hi(a), ii_lo(b)) >> 32) + (ii_wide(ii_lo(a), ii_hi(b)) >> 32);
}
/* Significand bits of f in [1, 2) from a 53-bit significand, rounded to
 * FP32 (a carry makes 2.0). */
NR_IHD uint32_t ii_f32(uint64_t m) { return (uint32_t)(((m & kIiFrac) + (1u << 28)) >> 29); }
/* y (1 - e), y Q32 (given as Q64), e = e1 / 2^63, |e| < 2^-21. */
NR_IHD uint64_t ii_newton(uint32_t y, int64_t e1) {
    return ii_join(y, 0) + (uint64_t)(ii_wides((int32_t)(e1 >> 11), (int32_t)(y >> 1)) >> 19);
}

/* Completes a 54-bit quotient: q is at most 2^11 below floor(2^s N / m),
 * rem = 2^s N - q m exactly (below 2^64), r32 = the Q32 reciprocal of
 * m / 2^52.  Returns the floor.  dq = rem_hi r32 / 2^52 estimates rem / m
 * within one (2^11 x 2^-22 + truncation), the remainder's sign says which. */
NR_IHD uint64_t ii_finish(uint64_t q, uint64_t rem, uint64_t m, uint32_t r32) {
    const uint32_t dq = ii_hi(ii_wide(ii_hi(rem), r32)) >> 20;
    const int64_t r2 = (int64_t)(rem - ii_wide(dq, ii_lo(m)) - ii_join(dq * ii_hi(m), 0));
    return q + dq + (r2 < 0 ? (uint64_t)-1 : (uint64_t)(r2 >= (int64_t)m));
}

/* a / b, round to nearest even. */
NR_IHD double ii_div(double a, double b) {
    const uint64_t ua = ii_bits(a), ub = ii_bits(b);
    const uint32_t ea = (ii_hi(ua) >> 20) & 0x7ffu, eb = (ii_hi(ub) >> 20) & 0x7ffu;
    const int32_t e = (int32_t)ea - (int32_t)eb + 1023;
    /* normal operands, and a result whose exponent cannot leave the normal
     * range by the adjustments below */
    if (ea - 1u >= 2046u || eb - 1u >= 2046u || (uint32_t)(e - 2) >= 2043u) {
        /* a zero over a normal number (straight triples at rest) is common */
        if ((ua << 1) == 0 && eb - 1u < 2046u) return ii_double((ua ^ ub) & 0x8000000000000000ULL);
        return ii_div_fallback(a, b);
    }
    const uint64_t ma = (ua & kIiFrac) | kIiOne, mb = (ub & kIiFrac) | kIiOne;
    /* f = mb / 2^52 in [1, 2); r0 = 2^32 / f (1 + e0), |e0| < 2^-22 */
    const uint32_t r0 = ii_rcp_q32(0x3f800000u + ii_f32(mb));
    const uint64_t B = mb << 11;
    /* p = B r0 / 2^32 = 2^63 (1 + e0); r1 = r0 (1 - e0): 2^64 / f (1 - e0^2),
     * truncations below 2^-51, always below 2^64 */
    const uint64_t p = ii_wide(ii_hi(B), r0) + (ii_wide(ii_lo(B), r0) >> 32);
    const uint64_t r1 = ii_newton(r0, (int64_t)(0x8000000000000000ULL - p));
    /* A / 2^62 = ma / 2^52, doubled when ma < mb, so that the quotient is in
     * [1, 2): to 54 bits, low by at most 2^-44 + 2^-51 relative; less one, as
     * the truncations of p may leave it a unit of 2^-63 high */
    const bool lt = ma < mb;
    uint64_t A = ma << 10;
    if (lt) A += A;
    const uint64_t q = (ii_mulhi_low3(A, r1) >> 9) - 1;
    /* A 2^43 - q mb modulo 2^64 */
    const uint64_t rem = ii_join((ii_lo(A) << 11) - ii_lo(q) * ii_hi(mb) - ii_hi(q) * ii_lo(mb), 0) -
                         ii_wide(ii_lo(q), ii_lo(mb));
    const uint64_t q54 = ii_finish(q, rem, mb, r0);
    const uint32_t top = ((ii_hi(ua) ^ ii_hi(ub)) & 0x80000000u) + ((uint32_t)(e - 1 - (lt ? 1 : 0)) << 20);
    return ii_double(((q54 + 1) >> 1) + ii_join(top, 0));
}

/* Root of the significand of a normal positive q: the 54-bit floor root, the
 * Q32 estimate y0 and its Newton refinement y1 (Q64) of 1 / sqrt, and the
 * result's biased exponent. */
NR_IHD uint64_t ii_root54(uint64_t uq, uint32_t &y0, uint64_t &y1, uint32_t &es) {
    const uint32_t eq = ii_hi(uq) >> 20;
    const uint32_t odd = (eq & 1u) ^ 1u; /* unbiased exponent odd: significand in [2, 4) */
    es = (eq + 1023u - odd) >> 1;
    const uint64_t mq = (uq & kIiFrac) | kIiOne;
    uint64_t X = mq << 10; /* Q62 in [1, 4) */
    if (odd) X += X;
    y0 = ii_rsqrt_q32((odd ? 0x40000000u : 0x3f800000u) + ii_f32(mq));
    /* x y0^2 = 1 + 2 e0 (Q62); y1 = y0 (1 - e0): 1 / sqrt(x) (1 - 1.5 e0^2) */
    const uint64_t p = ii_mulhi_low3(X, ii_wide(y0, y0));
    y1 = ii_newton(y0, (int64_t)(0x4000000000000000ULL - p));
    /* s1 = sqrt(x) (1 - 2^-43.4) in Q62, then one correction by x - s1^2
     * (Q60, below 2^20, off by a few units): within 2^5 of sqrt(x) in Q62 */
    const uint64_t s1 = ii_mulhi_low3(X, y1);
    const uint64_t sq = ii_wide(ii_hi(s1), ii_hi(s1)) + (ii_wide(ii_hi(s1), ii_lo(s1)) >> 31);
    const int32_t d = (int32_t)((X >> 2) - sq);
    const uint64_t s2 = s1 + (uint64_t)(ii_wides(d, (int32_t)(y0 >> 1)) >> 30);
    const uint64_t s = s2 >> 9; /* Q53: floor(sqrt(X 2^44)) within one */
    /* X 2^44 - s^2 modulo 2^64 */
    const int64_t rem = (int64_t)(ii_join((ii_lo(X) << 12) - 2u * (ii_lo(s) * ii_hi(s)), 0) - ii_wide(ii_lo(s), ii_lo(s)));
    return s + (rem < 0 ? (uint64_t)-1 : (uint64_t)(rem > (int64_t)(2 * s)));
}

NR_IHD bool ii_normal_positive(uint64_t uq) { return (ii_hi(uq) >> 20) - 1u < 2046u; }

/* sqrt(q), round to nearest even. */
NR_IHD double ii_sqrt(double q) {
    const uint64_t uq = ii_bits(q);
    if (!ii_normal_positive(uq)) return ii_sqrt_fallback(q);
    uint32_t y0, es;
    uint64_t y1;
    const uint64_t s = ii_root54(uq, y0, y1, es);
    return ii_double(((s + 1) >> 1) + ii_join((es - 1u) << 20, 0));
}

/* 1 / sqrt(q) as two roundings: the reciprocal, rounded to nearest, of the
 * square root rounded to nearest. */
NR_IHD double ii_inv_sqrt(double v) {
    const uint64_t uq = ii_bits(v);
    if (!ii_normal_positive(uq)) return ii_div_fallback(1.0, ii_sqrt_fallback(v));
    uint32_t y0, es;
    uint64_t y1;
    const uint64_t ms = (ii_root54(uq, y0, y1, es) + 1) >> 1; /* [2^52, 2^53] */
    /* rounded up to the next power of two: significand 1, exponent + 1 (the
     * estimates of 1 / 2 from below still fit 1 / 1) */
    if (ms >> 53) return ii_double(ii_join((2046u - es - 1u) << 20, 0));
    /* y1 / 2^64 = 1 / (ms / 2^52) (1 - 2^-43.4) up to the root's own rounding
     * (2^-53: two units of the 54-bit quotient, taken off): floor(2^106 / ms)
     * from its top 54 bits; ms = 2^52 gives 2^54 and the carry below */
    const uint64_t q = (y1 >> 10) - 4;
    const uint64_t rem = ii_join(0u - ii_lo(q) * ii_hi(ms) - ii_hi(q) * ii_lo(ms), 0) - ii_wide(ii_lo(q), ii_lo(ms));
    const uint64_t q54 = ii_finish(q, rem, ms, y0);
    return ii_double(((q54 + 1) >> 1) + ii_join((2045u - es - 1u) << 20, 0));
}

/* Comparisons without the FP64 pipe.  NaN: the callers' results are NaN
 * whichever way these answer. */
NR_IHD uint64_t ii_abs_bits(double v) { return ii_bits(v) & 0x7fffffffffffffffULL; }
NR_IHD bool ii_is_zero(double v) { return (ii_bits(v) << 1) == 0; }
NR_IHD bool ii_negative(double v) { return (ii_bits(v) >> 63) && !ii_is_zero(v); } /* v < 0 */
NR_IHD bool ii_positive(double v) { return !(ii_bits(v) >> 63) && !ii_is_zero(v); } /* v > 0 */
NR_IHD double ii_abs(double v) { return ii_double(ii_abs_bits(v)); }
NR_IHD double ii_flip(double v, bool neg) { return ii_double(ii_bits(v) ^ ((uint64_t)neg << 63)); }

}  // namespace nr

#endif
