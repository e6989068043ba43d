// lg_exact_div.cuh -- correctly rounded FP64 division and square root on the integer and FP32 pipes.
//
// GB300 issues one FP64 warp instruction per SM sub-partition about every 64 cycles, and one 32-bit
// integer instruction every cycle or two, so an FP64 division (about ten FP64 instructions) costs as
// much issue time as several hundred integer instructions. Here both operations run in fixed point:
//   reciprocal  a 22-bit estimate (MUFU), two Newton steps y <- y + y (1 - b y) on the 64-bit
//               significand: y = 2^64 / b' to a few units, never above it;
//   quotient    the high half of a' y: the quotient to about 60 bits, never above it, cut to 53 bits;
//               the sign of the exact remainder a - m b of the midpoint m above it decides the rounding
//               (the remainder is smaller than b, so 64-bit wrap-around arithmetic holds it; a quotient
//               of two 53-bit significands is never a midpoint itself);
//   root        the same with an inverse-root estimate, one Newton step, s = z y, one correction
//               s + (z - s^2) y / 2, and the sign of z - m^2.
// No step branches on the values, so independent quotients overlap.
// So results are RN(a / b) and RN(sqrt(z)), bit for bit what IEEE arithmetic gives. Long division
// with a quotient estimate and an exact remainder test is Knuth's (The Art of Computer Programming,
// vol. 2, 4.3.1); Newton iterations with a final remainder test are described in Muller et al.,
// Handbook of Floating-Point Arithmetic, ch. 4. Operands or results outside the normal range
// (subnormals, infinities, NaN, overflow, negative radicands) take the hardware's operation.
//
// The header also compiles as host code (the estimate from a host division), which the CPU tests use.
#pragma once
#include <cstdint>
#include <cstring>
#include <cmath>

#ifdef __CUDACC__
#define LG_XD __device__ __forceinline__
#define LG_XD_SLOW static __device__ __noinline__
#else
#define LG_XD static inline
#define LG_XD_SLOW static
#endif

namespace lg {
namespace xd {

LG_XD uint64_t bits_of(double v) {
#ifdef __CUDACC__
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t u;
    std::memcpy(&u, &v, 8);
    return u;
#endif
}
LG_XD double of_bits(uint64_t u) {
#ifdef __CUDACC__
    return __longlong_as_double((long long)u);
#else
    double v;
    std::memcpy(&v, &u, 8);
    return v;
#endif
}
LG_XD float float_of(uint32_t u) {
#ifdef __CUDACC__
    return __uint_as_float(u);
#else
    float v;
    std::memcpy(&v, &u, 4);
    return v;
#endif
}
LG_XD uint64_t mul_hi(uint64_t a, uint64_t b) {
#ifdef __CUDACC__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
LG_XD uint64_t mul_wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
#ifndef LG_XD_ESTIMATE  // (a test may pass its own, poorer estimates)
LG_XD float rcp_estimate(float f) {
#ifdef __CUDACC__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
    return r;
#else
    return 1.0f / f;
#endif
}
LG_XD float rsqrt_estimate(float f) {
#ifdef __CUDACC__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
    return r;
#else
    return 1.0f / std::sqrt(f);
#endif
}
#else
float rcp_estimate(float f);
float rsqrt_estimate(float f);
#endif

// 2^32 f for an estimate f of about [0.5, 1], kept within [2^31, 2^32 - 2^8]: from the float's bits, since
// a conversion instruction would go through the same slow path as the FP64 operations
LG_XD uint32_t fixed32(float f) {
#ifdef __CUDACC__
    int32_t u = __float_as_int(f);
#else
    int32_t u;
    std::memcpy(&u, &f, 4);
#endif
    u = u < 0x3f000000 ? 0x3f000000 : u > 0x3f7fffff ? 0x3f7fffff : u;
    return ((uint32_t)u << 8) | 0x80000000u;
}

constexpr uint64_t kFrac = 0xfffffffffffffull;  // 52 fraction bits
constexpr uint64_t kOne = 0x10000000000000ull;  // the implicit bit
LG_XD_SLOW double slow_div(double a, double b) { return a / b; }
LG_XD_SLOW double slow_sqrt(double z) { return ::sqrt(z); }

// A divisor: its significand and y = 2^64 / b' (b' in [1, 2)) from below.
struct Divisor {
    uint64_t y, m;  // reciprocal, 53-bit significand
    uint32_t top;   // sign and exponent field (bits 52..63 of b)
};

LG_XD Divisor divisor(double b) {
    const uint64_t u = bits_of(b);
    Divisor d;
    d.top = (uint32_t)(u >> 52);
    d.m = (u & kFrac) | kOne;
    const uint64_t bn = d.m << 11;  // b' 2^63
    const float r = rcp_estimate(float_of(0x3f800000u | ((uint32_t)(u >> 29) & 0x7fffffu)));
    const uint32_t y0 = fixed32(r);
    // e = 1 - b' y0 (2^63 units, |e| < 2^-20), y1 = y0 + y0 e
    const uint64_t t0 = mul_wide((uint32_t)(bn >> 32), y0) + (mul_wide((uint32_t)bn, y0) >> 32);
    const int32_t e0 = (int32_t)((int64_t)(0x8000000000000000ull - t0) >> 12);
    const uint64_t y1 = ((uint64_t)y0 << 32) + (uint64_t)(((int64_t)e0 * (int64_t)(uint64_t)y0) >> 19);
    // the same from y1 (|e| < 2^-40); e one unit low, so that y stays at or below 2^64 / b'
    const int32_t e1 = (int32_t)(int64_t)(0x8000000000000000ull - 2u - mul_hi(bn, y1));
    d.y = y1 + (uint64_t)(((int64_t)e1 * (int64_t)(y1 >> 32)) >> 31);
    return d;
}

// RN(a / b) for the divisor b where `ok` stays true: a zero or normal, b and the quotient normal
LG_XD double quotient(double a, const Divisor &d, bool &ok) {
    const uint64_t u = bits_of(a);
    const uint32_t top = (uint32_t)(u >> 52), ea = top & 0x7ffu, eb = d.top & 0x7ffu;
    const uint64_t sign = (uint64_t)((top ^ d.top) & 0x800u) << 52;
    const uint64_t m = (u & kFrac) | kOne;
    uint64_t q = mul_hi(m << 11, d.y);  // a' / b' 2^63, in (2^62, 2^64)
    const bool ge1 = (int64_t)q < 0;
    const int32_t er = (int32_t)ea - (int32_t)eb + (ge1 ? 1022 : 1021);  // exponent field of the quotient, less 1
    if (!ge1) q += q;
    const uint64_t s = q >> 11;  // the quotient's 53-bit significand, truncated
    // (a' 2^53 or 2^54) - (2 s + 1) b': the sign of quotient - midpoint
    const uint64_t rem = (m << (ge1 ? 53 : 54)) - (2u * s + 1u) * d.m;
    const double r = of_bits(sign | (((uint64_t)(uint32_t)er << 52) + s + ((int64_t)rem > 0 ? 1u : 0u)));
    const bool zero = (u << 1) == 0;
    ok = ok && (eb - 1u) < 0x7feu && (zero || ((ea - 1u) < 0x7feu && (uint32_t)er < 0x7fdu));
    return zero ? of_bits(sign) : r;
}

LG_XD double div(double a, double b) {
    bool ok = true;
    const double r = quotient(a, divisor(b), ok);
    return ok ? r : slow_div(a, b);
}

// RN(sqrt(z))
LG_XD double root(double z) {
    const uint64_t u = bits_of(z);
    const uint32_t top = (uint32_t)(u >> 52);  // exponent field (a sign bit fails the range test)
    const uint32_t odd = (top & 1u) ^ 1u;      // of the unbiased exponent
    const uint64_t m = (u & kFrac) | kOne;
    const uint64_t zn = m << (10 + odd);  // z' 2^62, z' in [1, 4)
    const float r = rsqrt_estimate(float_of(((127u + odd) << 23) | ((uint32_t)(u >> 29) & 0x7fffffu)));
    const uint32_t y0 = fixed32(r);
    // e = 1 - z' y0^2 (2^62 units, |e| < 2^-19), y1 = y0 + y0 e / 2
    const int32_t e0 = (int32_t)((int64_t)(0x4000000000000000ull - mul_hi(zn, mul_wide(y0, y0))) >> 12);
    const uint64_t y1 = ((uint64_t)y0 << 32) + (uint64_t)(((int64_t)e0 * (int64_t)(uint64_t)y0) >> 19);
    // s1 = z' y1 (2^62 units, |error| < 2^-38), s = s1 + (z' - s1^2) y1 / 2, a unit of the difference low
    const uint64_t s1 = mul_hi(zn, y1);
    const int32_t e1 = (int32_t)(int64_t)((zn >> 2) - 1u - mul_hi(s1, s1));
    const uint64_t s = s1 + (uint64_t)(((int64_t)e1 * (int64_t)(y1 >> 32)) >> 31);
    const uint64_t t = s >> 10;  // 53-bit significand, truncated
    const uint64_t mid = 2u * t + 1u;
    const bool up = (int64_t)((m << (54 + odd)) - mid * mid) > 0;
    const uint32_t er = (top + 1023u - 1u + (odd ^ 1u)) >> 1;  // exponent field of the root
    const double v = of_bits(((uint64_t)(er - 1u) << 52) + t + (up ? 1u : 0u));
    if ((top - 1u) >= 0x7feu) return (u << 1) == 0 ? z : slow_sqrt(z);
    return v;
}

}  // namespace xd
}  // namespace lg
