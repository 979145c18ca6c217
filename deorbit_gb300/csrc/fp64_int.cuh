// fp64_int.cuh -- IEEE double-precision operations on the integer pipes.
//
// GB300 issues an FP64 instruction on an SM sub-partition every 64 cycles, an
// integer one every one or two, so a kernel of FP64 arithmetic leaves nine
// tenths of its issue slots empty (the grid solver's FP64 face pass before it
// used these: FP64 pipe 87 % busy, issue slots 8 %).  A division or a square
// root is a chain of eight or more FP64 instructions; here it is about sixty
// 32-bit integer ones.  Measured, full SMs, cycles at 1.92 GHz per warp
// operation and sub-partition: division 556 -> 115, by a prepared divisor 84,
// square root 556 -> 136; an FP64 add, product or fused multiply-add takes 74.
// Every function returns the IEEE round-to-nearest result, bit for bit;
// operands or results outside the normal range (zeros apart) take the hardware
// operation.
//
// Methods: schoolbook division in a large radix with a reciprocal estimate
// (Knuth, The Art of Computer Programming 2, 4.3.1; Moeller & Granlund, Improved
// division by invariant integers), the digit-by-digit square root with its
// exact remainder.  Both round on the exact remainder.  (A product takes 149
// cycles this way and 74 on the FP64 pipe; it stays there.)
#pragma once

#include <cstdint>
#include <cstring>
#ifdef __CUDACC__
#include <cuda_runtime.h>
#define FI_FN __host__ __device__ __forceinline__
#else
#include <cmath>
#define FI_FN inline
#endif

namespace fi {

FI_FN uint64_t bits(double x) {
#ifdef __CUDA_ARCH__
    // opaque to the compiler, which turns integer tests of a double's bits
    // (zero, NaN) back into comparisons on the FP64 pipe
    uint32_t lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(x));
    return (uint64_t)hi << 32 | lo;
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}
FI_FN double from_bits(uint64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}
FI_FN uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }
FI_FN uint32_t lo32(uint64_t x) { return (uint32_t)x; }
FI_FN uint64_t mul32(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
FI_FN uint32_t mulhi(uint32_t a, uint32_t b) { return hi32(mul32(a, b)); }

// Hardware estimates: the callers allow for two units in the last place.  On
// the host a test can move its stand-ins by FI_ESTIMATE_ULP units.
#ifndef FI_ESTIMATE_ULP
#define FI_ESTIMATE_ULP 0
#endif
FI_FN float bits_f(uint32_t b) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float f;
    std::memcpy(&f, &b, 4);
    return f;
#endif
}
FI_FN uint32_t f_bits(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    uint32_t b;
    std::memcpy(&b, &f, 4);
    return b;
#endif
}
FI_FN float rcp_est(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return bits_f(f_bits(1.0f / x) + (uint32_t)(FI_ESTIMATE_ULP));
#endif
}
FI_FN float rsqrt_est(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return bits_f(f_bits((float)(1.0 / std::sqrt((double)x))) + (uint32_t)(FI_ESTIMATE_ULP));
#endif
}

// A divisor prepared for any number of divisions: significand, exponent and
// y, an underestimate of 2^84 / m by at most 2^-30 of it.
struct Divisor {
    uint64_t m;    // significand with its leading bit, 2^52 <= m < 2^53
    uint32_t y;
    uint32_t e;    // biased exponent
    uint32_t sign; // bit 31
    bool normal;
    double b;
};

FI_FN Divisor divisor(double b) {
    Divisor d;
    const uint64_t u = bits(b);
    d.b = b;
    d.e = (hi32(u) >> 20) & 0x7ffu;
    d.sign = hi32(u) & 0x80000000u;
    d.normal = d.e - 1u < 0x7feu;
    d.m = (u & 0xfffffffffffffull) | 0x10000000000000ull;
    const uint32_t t = (uint32_t)(d.m >> 21);  // leading 32 bits
    // estimate of 1 / t rounded up to 24 bits, less three units: below 2^63 / t
    // whatever the estimate's last two units are
    const uint32_t f = f_bits(rcp_est(bits_f((0x3f800000u | ((t << 1) >> 9)) + 1u))) - 3u;
    const uint32_t y0 = (f < 0x3f000000u ? 0x3f000000u : f) << 8 | 0x80000000u;
    // one Newton step y0 (2 - t y0), whose error term e is in [0, 2^43); y <= 2^63 / t
    // is above 2^84 / m by 2 units at most, which the last 3 take off
    const uint64_t e = (1ull << 63) - mul32(t, y0);
    d.y = y0 + (mulhi(y0, (uint32_t)(e >> 11)) >> 20) - 3u;
    return d;
}

// The hardware's operations for what the integer ones leave out.  Calls, not
// inline code: the compiler would otherwise issue the FP64 instruction in every
// case and select.
#ifdef __CUDACC__
#define FI_RARE static __host__ __device__ __noinline__
#else
#define FI_RARE static
#endif
FI_RARE double div_general(double a, double b) { return a / b; }
FI_RARE double sqrt_general(double a) {
#ifdef __CUDA_ARCH__
    return __dsqrt_rn(a);
#else
    return std::sqrt(a);
#endif
}
FI_RARE double half_general(double x) { return 0.5 * x; }
FI_RARE float to_float_general(double x) { return (float)x; }
FI_RARE double to_double_general(float y) { return (double)y; }
FI_RARE bool product_le0(double a, double b) { return a * b <= 0; }

// a / d, rounded to nearest even (a tie cannot occur: it would need a divisor
// significand with a factor 2^53).
FI_FN double div(double a, const Divisor& d) {
    const uint64_t u = bits(a);
    const uint32_t ea = (hi32(u) >> 20) & 0x7ffu;
    const uint64_t ma = (u & 0xfffffffffffffull) | 0x10000000000000ull;
    const bool less = ma < d.m;
    const uint64_t A = less ? ma << 1 : ma;              // d.m <= A < 2 d.m: quotient in [1, 2)
    const uint32_t e = ea - d.e + (less ? 1021u : 1022u); // biased exponent of the quotient less one
    const uint32_t s = (hi32(u) ^ d.sign) & 0x80000000u;
    // first digit: 2^30 A / m, underestimated by less than 8 (y by 6 units of 2^31
    // at most, A >> 22 and the product by their last places): r1 < 2^56
    const uint32_t q1 = mulhi((uint32_t)(A >> 22), d.y);
    const uint64_t r1 = (A << 30) - (uint64_t)q1 * d.m;
    // second digit: 2^22 r1 / m, underestimated by less than 1.1
    const uint32_t q2 = mulhi((uint32_t)(r1 >> 24), d.y) >> 6;
    const uint64_t r2 = (r1 << 22) - (uint64_t)q2 * d.m;
    const uint64_t q = ((uint64_t)q1 << 22) + q2 + (2 * r2 > d.m ? 1u : 0u);
    double v = from_bits(q + ((uint64_t)(s | (e << 20)) << 32));
    const bool zero = (u << 1) == 0;
    if (zero) v = from_bits((uint64_t)s << 32);
    if (!(d.normal && (zero || (ea - 1u < 0x7feu && e - 1u < 0x7fcu)))) v = div_general(a, d.b);
    return v;
}
FI_FN double div(double a, double b) { return div(a, divisor(b)); }

// Square root, rounded to nearest (no ties: the root of a 53-bit significand
// is never halfway between two of them).
FI_FN double sqrt(double x) {
    const uint64_t u = bits(x);
    const uint32_t e = hi32(u) >> 20;  // with the sign: 0 and >= 0x7ff take the general route
    const uint64_t m = (u & 0xfffffffffffffull) | 0x10000000000000ull;
    const bool odd = (e & 1u) == 0;    // 1023 is odd: an even biased exponent is an odd power
    const uint64_t M = odd ? m << 1 : m;           // radicand t = M / 2^52 in [1, 4)
    const uint32_t t = (uint32_t)(M >> 22);         // t 2^30
    // y ~ 2^32 / sqrt(t): estimate and one Newton step
    float f = rsqrt_est(bits_f(((odd ? 0x40000000u : 0x3f800000u) | ((uint32_t)(m >> 29) & 0x7fffffu))));
    f = f >= 1.0f ? 0x1.fffffep-1f : (f < 0.5f ? 0.5f : f);
    const uint32_t y0 = (f_bits(f) << 8) | 0x80000000u;
    const uint64_t y2 = mul32(y0, y0);              // 2^64 / t
    // g = 2^62 - t y^2 (t 2^30 * y2 2^-32), |g| < 2^41
    const int64_t g = (int64_t)((1ull << 62) - mul32(t, hi32(y2)));
    const int32_t g32 = (int32_t)(g >> 11);         // 2^51 (1 - t y^2)
    const int64_t corr = (int64_t)y0 * g32;         // y 2^51 (1 - t y^2)
    uint32_t y = y0 + (uint32_t)(int32_t)(corr >> 52);
    if (y < 0x80000000u) y = (y0 >= 0xc0000000u) ? 0xffffffffu : 0x80000000u;  // wrapped at 1 or fell below 1/2
    // first part: sqrt(t) 2^30, underestimated by 1 .. 16
    const uint32_t s1 = mulhi(t, y) - 8u;
    const uint64_t r1 = (M << 8) - mul32(s1, s1);   // t 2^60 - s1^2, below 2^38
    // the remaining 22 bits: r1 2^22 / (2 s1), underestimated by 0 .. 2.4 units
    const uint32_t s2 = (uint32_t)(((uint64_t)(uint32_t)(r1 >> 6) * y) >> 35) - 1u;
    uint64_t s = ((uint64_t)s1 << 22) + s2;
    const uint64_t r2 = (M << 52) - s * s;          // exact remainder mod 2^64
    const int64_t r = (int64_t)r2;
    s += (r > (int64_t)s ? 1u : 0u) + (r > (int64_t)(3 * s + 2) ? 1u : 0u) + (r > (int64_t)(5 * s + 6) ? 1u : 0u);
    double v = from_bits(s + ((uint64_t)(((e + 1023u) >> 1) - 1u) << 52));
    if (e - 1u >= 0x7feu) v = (u << 1) == 0 ? x : sqrt_general(x);
    return v;
}

// Comparisons and scalings without the FP64 pipe.  NaN compares false, zeros of
// either sign are equal.
FI_FN bool lt0(double x) { return bits(x) - 0x8000000000000001ull < 0x7ff0000000000000ull; }
FI_FN bool gt0(double x) { return bits(x) - 1u < 0x7ff0000000000000ull; }
FI_FN bool ge0(double x) { return bits(x) <= 0x7ff0000000000000ull || bits(x) == 0x8000000000000000ull; }
FI_FN bool le0(double x) { return bits(x) == 0 || bits(x) - 0x8000000000000000ull <= 0x7ff0000000000000ull; }
// the value's place among the doubles as a signed integer
FI_FN int64_t order(double x) {
    const uint64_t u = bits(x);
    return (int64_t)(u >> 63 ? 0x8000000000000000ull - u : u);
}
FI_FN bool is_nan(double x) { return (bits(x) << 1) > 0xffe0000000000000ull; }
FI_FN bool lt(double a, double b) { return order(a) < order(b) && !is_nan(a) && !is_nan(b); }
FI_FN bool le(double a, double b) { return order(a) <= order(b) && !is_nan(a) && !is_nan(b); }
// |a| < |b|
FI_FN bool abs_lt(double a, double b) { return (bits(a) << 1) < (bits(b) << 1) && !is_nan(b); }

// x / 2 (below the normal range: the hardware product).
FI_FN double half(double x) {
    const uint32_t e = (hi32(bits(x)) >> 20) & 0x7ffu;
    if (e - 2u < 0x7fdu) return from_bits(bits(x) - 0x10000000000000ull);
    return (bits(x) << 1) == 0 || e == 0x7ffu ? x : half_general(x);
}

// Conversions (FP64-pipe instructions in hardware): to nearest even, and exact.
// Results or operands below FP32's normal range, infinities and NaN take the
// hardware's.
FI_FN float to_float(double x) {
    const uint64_t u = bits(x);
    const uint32_t e = (hi32(u) >> 20) & 0x7ffu, rest = lo32(u) << 3;
    uint32_t f = (uint32_t)((u & 0x7fffffffffffffffull) >> 29) - (896u << 23);
    f += rest + (f & 1u) > 0x80000000u ? 1u : 0u;
    const bool zero = (u << 1) == 0;
    if (zero) f = 0;
    if (!zero && !(e - 897u < 254u)) return to_float_general(x);
    return bits_f(f | (hi32(u) & 0x80000000u));
}
FI_FN double to_double(float y) {
    const uint32_t f = f_bits(y), a = f & 0x7fffffffu;
    const bool zero = a == 0;
    if (!zero && !(a - 0x800000u < 0x7f000000u)) return to_double_general(y);
    const uint32_t h = zero ? 0u : (a >> 3) + (896u << 20);
    return from_bits(((uint64_t)(h | (f & 0x80000000u)) << 32) | (uint64_t)(f << 29));
}

// minmod: 0 where a b <= 0, else the smaller of the two in magnitude (b where
// the product or the comparison has a NaN); the product's own underflow to
// zero counts as 0.
FI_FN double minmod(double a, double b) {
    const uint32_t ea = (hi32(bits(a)) >> 20) & 0x7ffu, eb = (hi32(bits(b)) >> 20) & 0x7ffu;
    const bool zero = (bits(a) << 1) == 0 || (bits(b) << 1) == 0;
    if (ea == 0x7ffu || eb == 0x7ffu || (!zero && ea + eb < 1023u)) {
        if (product_le0(a, b)) return 0.0;
    } else if (zero || ((hi32(bits(a)) ^ hi32(bits(b))) >> 31)) {
        return 0.0;
    }
    return abs_lt(a, b) ? a : b;
}

}  // namespace fi
