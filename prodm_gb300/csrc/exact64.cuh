// Products, quotients and square roots of doubles, correctly rounded, on the
// integer pipes. An SM of this chip does two FP64 operations a clock and a
// division or a root takes eight or more of them in a row, 128 clocks a warp;
// the same digits by integer arithmetic take about 55 instructions of pipes
// that are 32 times as wide. A product takes 45 instructions instead of one of
// 16 clocks: for where the FP64 pipe is full and the others are not. A
// correctly rounded result is one value, so these equal the operators bit for
// bit.
//
// Quotient and root are long division on 53-bit significands: a 23-bit
// reciprocal (root) from the special function unit gives a digit of 20 bits,
// the remainder is updated exactly (modulo 2^64; its true value is always below
// 2^55), and so on; the last digit is rounded to nearest, and the sign of the last remainder
// against half a unit decides the rounding. Neither a quotient nor a root of
// 53-bit numbers lies halfway between two 53-bit numbers. Operands or results
// that are zero, subnormal, infinite or NaN go to the operators.
#pragma once
#include <cstdint>

namespace prodm {

// the 24 bits of a float that is 1/2 .. 1 but for its error (below 1 in the end)
__device__ __forceinline__ uint32_t clamp24(float r) {
    return (min(max(__float_as_uint(r), 0x3f000000u), 0x3f7fffffu) & 0x7fffffu) | 0x800000u;
}

// 2^24 / f and 2^24 / sqrt(f), f a float in [1, 2) or [1, 4), within a few
// units
__device__ __forceinline__ uint32_t rcp24(float f) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
    return clamp24(r);
}
__device__ __forceinline__ uint32_t rsqrt24(float f) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
    return clamp24(r);
}

// rem + q * m modulo 2^64
__device__ __forceinline__ uint64_t mad64(uint32_t q, uint64_t m, uint64_t rem) {
    const uint64_t lo = (uint64_t)q * (uint32_t)m + rem;
    return lo + ((uint64_t)(q * (uint32_t)(m >> 32)) << 32);
}

__device__ __forceinline__ double div_exact(double a, double b) {
    const uint64_t ua = (uint64_t)__double_as_longlong(a), ub = (uint64_t)__double_as_longlong(b);
    const uint32_t ha = (uint32_t)(ua >> 32), hb = (uint32_t)(ub >> 32);
    const uint32_t ea = (ha >> 20) & 0x7ff, eb = (hb >> 20) & 0x7ff;
    const uint64_t ma = (uint64_t)((ha & 0xfffff) | 0x100000) << 32 | (uint32_t)ua;
    const uint64_t mb = (uint64_t)((hb & 0xfffff) | 0x100000) << 32 | (uint32_t)ub;
    const uint32_t lt = ma < mb;
    const uint32_t er = ea - eb + 1023 - lt;
    if (ea - 1 >= 2046u || eb - 1 >= 2046u || er - 1 >= 2045u) {
        if ((ua << 1) == 0 && eb - 1 < 2046u) return __longlong_as_double((long long)((ua ^ ub) & 1ull << 63));
        return a / b;
    }
    const uint32_t r = rcp24(__uint_as_float(0x3f800000u | ((uint32_t)(mb >> 29) & 0x7fffffu)));   // 2^76 / mb
    const uint64_t nb = 0 - mb;
    uint64_t rem = ma << lt;                                       // in [mb, 2 mb)
    const uint32_t q1 = __umulhi((uint32_t)(rem >> 24), r) - 1;    // below rem 2^20 / mb by 0.5 .. 2.6
    rem = mad64(q1, nb, rem << 20);
    const uint32_t q2 = __umulhi((uint32_t)(rem >> 24), r) - 1;    // by 0.3 .. 2.7
    rem = mad64(q2, nb, rem << 20);
    const uint32_t q3 = (__umulhi((uint32_t)(rem >> 24), r) + 128) >> 8;   // nearest, within 0.51
    rem = mad64(q3, nb, rem << 12);
    uint64_t q = ((uint64_t)q1 << 32) + ((uint64_t)q2 << 12) + q3;
    const int64_t two = (int64_t)(rem << 1);
    q += two > (int64_t)mb ? 1 : 0;
    q -= two < -(int64_t)mb ? 1 : 0;
    const uint64_t bits = q + ((uint64_t)(((er - 1) << 20) | ((ha ^ hb) & 0x80000000u)) << 32);
    return __longlong_as_double((long long)bits);
}

__device__ __forceinline__ double sqrt_exact(double x) {
    const uint64_t ux = (uint64_t)__double_as_longlong(x);
    const uint32_t hx = (uint32_t)(ux >> 32);
    const uint32_t e = hx >> 20;   // with the sign above it
    if (e - 1 >= 2046u) return ux == 0 ? x : sqrt(x);
    const uint32_t odd = ~e & 1;   // of the unbiased exponent
    const uint32_t er = (e + 1023 - odd) >> 1;
    const uint64_t m = ((uint64_t)((hx & 0xfffff) | 0x100000) << 32 | (uint32_t)ux) << odd;   // f 2^52, f in [1, 4)
    const uint32_t y =
        rsqrt24(__uint_as_float(((127 + odd) << 23) | ((hx & 0xfffff) << 3) | ((uint32_t)ux >> 29)));   // 2^24 / sqrt(f)
    // root S = s1 2^31 + d2 2^10 + d3 of f 2^104, remainder f 2^104 - S^2 in
    // units of 2^42 after s1 and of 2^20 after d2
    const uint32_t s1 = (__umulhi((uint32_t)(m >> 22), y) >> 1) - 2;   // below by 1.2 .. 3.6
    uint64_t rem = (m << 10) - ((uint64_t)s1 * s1 << 20);
    const uint32_t d2 = __umulhi((uint32_t)(rem >> 14), y << 1) - 3;   // below by 1.5 .. 11.3 (16 would be too far)
    rem = ((rem - (uint64_t)s1 * d2) << 22) - (uint64_t)d2 * d2;
    const uint32_t d3 = (__umulhi((uint32_t)(rem >> 16), y) + 256) >> 9;   // nearest, within 0.51
    uint64_t s = ((uint64_t)s1 << 31) + ((uint64_t)d2 << 10);
    rem = mad64(d3, 0 - (2 * s + d3), rem << 20);
    s += d3;
    const int64_t left = (int64_t)rem, half = (int64_t)s;
    s += left > half ? 1 : 0;
    s -= left <= -half ? 1 : 0;
    return __longlong_as_double((long long)(s + ((uint64_t)((er - 1) << 20) << 32)));
}

// a * b by the operator, in a call: as a single instruction the compiler puts it
// under a predicate, and the FP64 pipe is as busy with it as if it ran
static __device__ __noinline__ double mul_fp64(double a, double b) { return __dmul_rn(a, b); }

// a * b, rounded to nearest even: the 128-bit product of the significands
__device__ __forceinline__ double mul_exact(double a, double b) {
    const uint64_t ua = (uint64_t)__double_as_longlong(a), ub = (uint64_t)__double_as_longlong(b);
    const uint32_t ha = (uint32_t)(ua >> 32), hb = (uint32_t)(ub >> 32);
    const uint32_t ea = (ha >> 20) & 0x7ff, eb = (hb >> 20) & 0x7ff;
    const uint32_t sum = ea + eb;
    if (ea - 1 >= 2046u || eb - 1 >= 2046u || sum - 1025 >= 2043u) return mul_fp64(a, b);
    // significands as 1.63 fixed point
    const uint32_t a0 = (uint32_t)ua << 11, a1 = __funnelshift_l((uint32_t)ua, ha, 11) | 0x80000000u;
    const uint32_t b0 = (uint32_t)ub << 11, b1 = __funnelshift_l((uint32_t)ub, hb, 11) | 0x80000000u;
    const uint64_t t0 = (uint64_t)a0 * b0, t1 = (uint64_t)a1 * b0 + (t0 >> 32), t2 = (uint64_t)a0 * b1 + (uint32_t)t1;
    uint64_t hi = (uint64_t)a1 * b1 + (t1 >> 32) + (t2 >> 32);   // in [2^62, 2^64)
    const uint32_t below = (uint32_t)t2 | (uint32_t)t0;
    const uint32_t big = (uint32_t)(hi >> 63);
    hi <<= 1 - big;
    const uint32_t rest = ((uint32_t)hi & 0x7ffu) | (below ? 1u : 0u);   // (a bit shifted in from below is below's)
    uint64_t q = hi >> 11;
    q += rest + ((uint32_t)q & 1u) > 0x400u ? 1 : 0;
    return __longlong_as_double((long long)(q + ((uint64_t)(((sum - 1024 + big) << 20) | ((ha ^ hb) & 0x80000000u)) << 32)));
}

constexpr uint64_t kInfBits = 0x7ff0000000000000ull;
__device__ __forceinline__ unsigned long long bits64(double x) { return (unsigned long long)__double_as_longlong(x); }
// a > b for a, b that are +0, positive or NaN (a comparison of doubles is an
// FP64 operation too)
__device__ __forceinline__ bool above(double a, double b) { return bits64(a) > bits64(b) && bits64(a) <= kInfBits; }
// 2 |x|
__device__ __forceinline__ double twice_abs(double x) {
    const uint64_t u = bits64(x) & ~(1ull << 63);
    if ((uint32_t)(u >> 52) - 1 < 2045u) return __longlong_as_double((long long)(u + (1ull << 52)));
    return mul_fp64(2.0, __longlong_as_double((long long)u));
}

}  // namespace prodm
