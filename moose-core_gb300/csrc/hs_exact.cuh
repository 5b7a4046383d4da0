// hs_exact.cuh -- IEEE double operations with most of their work on the
// integer and FP32 pipes.
//
// GB300 issues one FP64 warp instruction per 76 cycles and SM sub-partition
// (measured; latency 64), an integer or FP32 one per cycle, and FP64 compares
// and conversions to and from integers run at the FP64 rate too.  A
// reference-order step is bound by that pipe, so the functions here give the
// IEEE result (every one is bit-identical to the plain operation) with as few
// FP64 instructions as the operation needs:
//   a / d                 2 instead of ~8 (a dependent division 564 -> 358 cycles;
//                         four warps a sub-partition, per division of a warp:
//                         563 -> 151 cycles)
//   a / d, d a constant   3 (Markstein's theorem)
//   compares              0
//   integer and fraction part of a non-negative value   0 instead of 3
#pragma once

#include <cstdint>

#ifdef __CUDACC__

namespace hsg {

// A double's bits, by a move that the compiler does not see through: it would
// turn integer tests on them (for a NaN, say) back into FP64 instructions.
__device__ __forceinline__ long long bitsOf(double x) {
    long long b;
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
    return b;
}
__device__ __forceinline__ uint32_t hiOf(double x) { return (uint32_t)((unsigned long long)bitsOf(x) >> 32); }
__device__ __forceinline__ uint32_t loOf(double x) { return (uint32_t)bitsOf(x); }
__device__ __forceinline__ double fromWords(uint32_t hi, uint32_t lo) { return __hiloint2double((int)hi, (int)lo); }

// a < b and a <= b as IEEE has them: false with a NaN, -0 equal to +0.
__device__ __forceinline__ bool compareKeys(double a, double b, long long& x, long long& y) {
    x = bitsOf(a);
    y = bitsOf(b);
    const long long top = 0x7FFFFFFFFFFFFFFFll;
    const bool ordered = (x & top) <= 0x7FF0000000000000ll && (y & top) <= 0x7FF0000000000000ll;
    if (x < 0) x = -(x & top);      // -0 and +0 both 0
    if (y < 0) y = -(y & top);
    return ordered;
}
__device__ __forceinline__ bool lessThan(double a, double b) {
    long long x, y;
    return compareKeys(a, b, x, y) && x < y;
}
__device__ __forceinline__ bool atMost(double a, double b) {
    long long x, y;
    return compareKeys(a, b, x, y) && x <= y;
}

__device__ __forceinline__ bool isOne(double x) { return hiOf(x) == 0x3FF00000u && loOf(x) == 0u; }
__device__ __forceinline__ bool isZero(double x) { return ((hiOf(x) << 1) | loOf(x)) == 0u; }

// The division as the compiler does it, out of line: the rare operands that
// quotient() does not take.
static __device__ __noinline__ double plainQuotient(double a, double d) { return a / d; }

// q if it is RN(a / d), else the plain division's result.  q is next to the
// quotient, so a - d q is exact, and q is right if that is less than |d| half
// a last place of q (a quarter on the lower side of a power of two, where
// places are half as large; never equal).
static __device__ __noinline__ double checkedQuotient(double a, double d, double q) {
    const double r = __fma_rn(-d, q, a);
    const unsigned long long top = 0x7FFFFFFFFFFFFFFFull, R = bitsOf(r) & top;
    const bool below = ((bitsOf(r) ^ bitsOf(a)) >> 63) && ((unsigned long long)bitsOf(q) << 12) == 0ull;
    const unsigned long long e = ((unsigned long long)bitsOf(q) & 0x7FF0000000000000ull) >> 52;
    const unsigned long long half = (bitsOf(d) & top) - ((1023ull + 53ull + (below ? 1ull : 0ull) - e) << 52);
    return R < half ? q : plainQuotient(a, d);
}

// RN(a / d).  With mantissas a', d' in [1, 2):
//   y0 + y1 ~ 1 / d', qh + ql ~ a' / d' as sums of two floats, from the FP32
//   reciprocal and the FP32 residual (relative error < 2^-43);
//   Q = qh + ql as a double (integer addition of the low part),
//   r = a - d Q, one fused operation: the remainder to 53 bits,
//   q = RN(Q + r y0): before rounding off by less than 2^-13 of q's last
//   place, so q is the correctly rounded quotient unless the sum lies within
//   that of a midpoint between two doubles.
// That case (the fraction of r / d in last places within 2^-10 of 1/2, about
// one division in 500) and a quotient next to a power of two (whose last place
// changes there; a saturated gate's is next to 1 at every step) are checked by
// their remainder.  A sum Q that leaves qh's binade, zeros, infinities, NaNs
// and exponents beyond +-383 take the plain division.  The remainder test needs no exact tie: a quotient of two
// doubles is never halfway between two doubles of normal range.
struct Recip {          // what a division needs of its divisor
    float y0, y1;
    uint32_t h;         // the divisor's high word
};

__device__ __forceinline__ float mantissa(uint32_t hi, uint32_t lo) {
    return __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x007FFFFFu) | 0x3F800000u);
}
// the 29 bits below the mantissa's 24, cut to 23, at their weight
__device__ __forceinline__ float mantissaTail(uint32_t lo) {
    return (__uint_as_float(((lo >> 6) & 0x007FFFFFu) | 0x3F800000u) - 1.0f) * 0x1p-23f;
}

__device__ __forceinline__ Recip recip(double d) {
    Recip R;
    R.h = hiOf(d);
    const uint32_t l = loOf(d);
    const float f = mantissa(R.h, l), t = mantissaTail(l);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(R.y0) : "f"(f));
    float e = fmaf(-f, R.y0, 1.0f);
    e = fmaf(-t, R.y0, e);
    R.y1 = R.y0 * fmaf(e, e, e);
    return R;
}

__device__ __forceinline__ double quotient(double a, double d, const Recip& R) {
    const uint32_t ha = hiOf(a), la = loOf(a), hd = R.h;
    const bool ok = (ha & 0x7FFFFFFFu) - 0x28000000u < 0x30000000u && (hd & 0x7FFFFFFFu) - 0x28000000u < 0x30000000u;
    const float fa = mantissa(ha, la), ta = mantissaTail(la);
    const float qh = fa * R.y0;
    float ql = fmaf(fa, R.y0, -qh);
    ql = fmaf(fa, R.y1, ql);
    ql = fmaf(ta, R.y0, ql);
    const uint32_t qb = __float_as_uint(qh);
    // ql (below 2^-21.2 of qh) in units of 2^9 last places of qh's double, that
    // is of 2^(exponent(qh) - 43): rounded to an integer by adding 1.5 * 2^23
    const float kf = fmaf(ql, __uint_as_float((297u << 23) - (qb & 0xFF800000u)), 12582912.0f);
    const int k = (__float_as_int(kf) - 0x4B400000) * 512;
    const uint32_t ea = ha & 0x7FF00000u, ed = hd & 0x7FF00000u, sgn = (ha ^ hd) & 0x80000000u;
    unsigned long long Qb = ((unsigned long long)((qb >> 3) + 0x38000000u) << 32) | (qb << 29);
    Qb += (long long)k;
    const uint32_t hQ = (uint32_t)(Qb >> 32) + ea - ed;
    const double Q = fromWords(hQ | sgn, (uint32_t)Qb);
    const double r = __fma_rn(-d, Q, a);
    const uint32_t yb = __float_as_uint(R.y0);
    const double y = fromWords(((yb >> 3) + 0x38000000u + 0x3FF00000u - ed) | (hd & 0x80000000u), yb << 29);
    const double q = __fma_rn(r, y, Q);
    // |r / d| in last places of Q, as a float
    const uint32_t hr = hiOf(r);
    const int s = (int)(hr & 0x7FFFFFFFu) - (int)(ed - 0x3FF00000u) - (int)((hQ & 0x7FF00000u) - 0x3FF00000u) -
                  (int)((1023u - 52u - 127u) << 20);
    const float t = __uint_as_float(((uint32_t)s << 3) | (loOf(r) >> 29)) * R.y0;
    const float n = (t + 12582912.0f) - 12582912.0f;
    const bool near = s >= (1 << 20) && fabsf(t - n) > 0.5f - 0x1p-10f;
    // q within 1,024 last places of a power of two
    const uint32_t lq = loOf(q) + 1024u;
    const bool edge = lq < 2048u && ((hiOf(q) + (lq < 1024u ? 1u : 0u)) & 0xFFFFFu) == 0u;
    // the integer sum crossed into another binade, whose last places differ
    const bool cross = (((uint32_t)(Qb >> 32) ^ ((qb >> 3) + 0x38000000u)) & 0x7FF00000u) != 0u;
    if (!ok || cross) return plainQuotient(a, d);
    if (near || edge) return checkedQuotient(a, d, q);
    return q;
}

__device__ __forceinline__ double quotient(double a, double d) { return quotient(a, d, recip(d)); }

// RN(a / d) for a divisor whose correctly rounded reciprocal y = RN(1 / d) is
// at hand: q0 = RN(a y), r = a - q0 d exactly, RN(q0 + r y) is the correctly
// rounded quotient (P. Markstein, Computation of elementary functions on the
// IBM RISC System/6000, 1990).  A non-zero a so small that the remainder
// could leave the normal range takes the plain division.
__device__ __forceinline__ double quotientBy(double a, double d, double y) {
    if ((hiOf(a) & 0x7FF00000u) < 0x10000000u && !isZero(a)) return plainQuotient(a, d);
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-q, d, a), y, q);
}

// Integer part of x >= 0 below 2^31, and the exact fraction x - integer part
// (a NaN: 0 and the NaN).
__device__ __forceinline__ uint32_t splitFraction(double x, double& frac) {
    const uint32_t h = hiOf(x);
    const int e = (int)(h >> 20) - 1023;
    if (e < 0 || e > 30) {
        frac = x;
        return 0u;
    }
    const unsigned long long m = ((unsigned long long)((h & 0xFFFFFu) | 0x100000u) << 32) | loOf(x);
    const uint32_t i = (uint32_t)(m >> (52 - e));
    const unsigned long long f = m << (12 + e);            // the fraction's bits, left-aligned
    const int lz = __clzll((long long)f);
    const unsigned long long g = f << lz;                  // top bit set, or 0
    const uint32_t hi = (uint32_t)(g >> 43);               // implicit bit at 20
    const uint32_t lo = (uint32_t)(g >> 11);
    frac = f ? fromWords(hi + ((uint32_t)(1021 - lz) << 20), lo) : 0.0;
    return i;
}

}  // namespace hsg

#endif  // __CUDACC__
