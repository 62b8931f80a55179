// fp64_int.cuh -- parts of the exact FP64 collision on the integer pipes, with the FP64 pipe's bits.
//
// GB300 issues fewer than two FP64 operations per clock and SM (a warp instruction holds its scheduler's FP64 pipe for
// some 80 cycles), but 64 integer ALU operations and 64 integer multiply-adds.  Where the range of the operands is known,
// a correctly rounded FP64 add is an integer add and a rounding to a fixed bit position, about a dozen integer
// instructions, and runs beside the FP64 work of the other warps.  Everything here is integer arithmetic from the
// definition of round-to-nearest-even; the results are the IEEE ones, bit for bit.
#pragma once

#include <cstdint>

namespace erlbm {
namespace fp64int {

#ifdef __CUDA_ARCH__
__device__ __forceinline__ uint64_t bits(double x) { return (uint64_t)__double_as_longlong(x); }
__device__ __forceinline__ double from_bits(uint64_t b) { return __longlong_as_double((long long)b); }
#else
inline uint64_t bits(double x)
{
    uint64_t b;
    __builtin_memcpy(&b, &x, 8);
    return b;
}
inline double from_bits(uint64_t b)
{
    double x;
    __builtin_memcpy(&x, &b, 8);
    return x;
}
#endif

__host__ __device__ __forceinline__ uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }
__host__ __device__ __forceinline__ uint64_t mantissa(uint64_t b) { return (b & 0xfffffffffffffull) | 0x10000000000000ull; }
__host__ __device__ __forceinline__ int exponent(uint64_t b) { return (int)(hi32(b) >> 20) & 0x7ff; }

// x rounded to a multiple of 2^K, ties to even.
template <int K>
__host__ __device__ __forceinline__ uint64_t round_at(uint64_t x)
{
    const uint64_t r = x + ((1u << (K - 1)) - 1) + ((uint32_t)x >> K & 1u);
    return r & ~(uint64_t)((1u << K) - 1);
}
// The same at bit k (k < 32).
__host__ __device__ __forceinline__ uint64_t round_at(uint64_t x, int k)
{
    const uint32_t low = 1u << k;
    const uint64_t r = x + ((low >> 1) - 1) + ((uint32_t)x >> k & 1u);
    return r & ~(uint64_t)(low - 1);
}

// x >> sh (0 <= sh <= 63) with a 1 in the last place if a bit was lost: enough for any later rounding at a
// higher place to go the way the exact value would.
__host__ __device__ __forceinline__ uint64_t shift_sticky(uint64_t x, int sh)
{
    const uint64_t t = x >> sh;
    return t | (uint64_t)((t << sh) != x);
}

constexpr uint64_t ONE62 = 1ull << 62;

// A double 0 <= x < 1 in units of 2^-62, lost bits sticky (0 gives 0 or 1: see eq_pair).
__host__ __device__ __forceinline__ uint64_t fixed62(double x)
{
    const uint64_t b = bits(x);
    const int sh = 1022 - exponent(b);
    return shift_sticky(mantissa(b) << 9, sh < 63 ? sh : 63);
}

// The velocity components and their sums eq_pair takes are below this in modulus.
constexpr double EQ_MAX = 0.16;
constexpr uint32_t EQ_MAX_HI = 0x3fc47ae1u;  // upper word of 0.16

// ((1 + t) + B) - C and ((1 - t) + B) - C with t = RN(3 cv), B = RN(3 RN(1.5 cv2)), every sum rounded, for |cv| <
// EQ_MAX, cv2 = RN(cv cv) and C = RN(1.5 u^2) in the form of fixed62, C < 0.12.  In units of 2^-62, sums below
// 1 are rounded at bit 9 and sums in [1, 2) at bit 10.  With a = |t| <= 0.48, 1 + a and (1 + a) + B lie in [1, 2);
// 1 - a, (1 - a) + B (B <= 0.24 |t|) and that less C lie in [1/2, 1]; only (1 + a) + B less C can lie on either
// side of 1.  A sum that rounds up to 1 at bit 9 is 1.  Zero operands come out of the shifts as 0 or sticky 1, and
// one unit more or less beside a multiple of 2^9 does not change a rounding.  Nine FP64 operations.
__host__ __device__ __forceinline__ void eq_pair(double cv, double cv2, uint64_t C62, double &plus, double &minus)
{
    const uint64_t bc = bits(cv), bp = bits(cv2);
    // t: 3 m has 54 or 55 bits, rounded to 53; 2^7 (3 m) 2^(E - 1020) is t in units of 2^-62
    const uint64_t m3 = mantissa(bc) * 3u;
    const uint64_t v = round_at(m3, 1 + (int)(hi32(m3) >> 22));
    const int st = 1020 - exponent(bc);
    const uint64_t t = shift_sticky(v << 7, st < 63 ? st : 63);
    // B: the same twice; 3 times the first has 56 or 57 bits
    const uint64_t n3 = mantissa(bp) * 3u;
    const uint64_t n9 = round_at(n3, 1 + (int)(hi32(n3) >> 22)) * 3u;
    const uint64_t w = round_at(n9, 3 + (int)(hi32(n9) >> 24));
    const int sb = 1019 - exponent(bp);
    const uint64_t B = shift_sticky(w << 5, sb < 63 ? sb : 63);

    uint64_t p = round_at<10>(ONE62 + t), q = round_at<9>(ONE62 - t);
    p = round_at<10>(p + B);
    q = round_at<9>(q + B);
    p = p - C62;
    const int k = 9 + (int)(hi32(p) >> 30);
    p = round_at(p, k);
    q = round_at<9>(q - C62);
    // units of 2^-62 to a double: the leading bit adds 1 to the exponent field
    const uint64_t up = (p >> k) + ((uint64_t)(1012 + k) << 52), uq = (q >> 9) + (1021ull << 52);
    const bool neg = (int64_t)bc < 0;
    plus = from_bits(neg ? uq : up);
    minus = from_bits(neg ? up : uq);
}

// ---- quotients by a constant ------------------------------------------------------------------------------------
// a / y rounded to nearest from z = RN(1 / y): a quotient within an ulp corrected by one fused step on its exact
// residual (Markstein's theorem, which asks for a correctly rounded reciprocal), after one step that brings the
// product a z within an ulp.  For |a| and |y| well inside the exponent range.  5 operations.
__host__ __device__ __forceinline__ double fused(double a, double b, double c)
{
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return __builtin_fma(a, b, c);
#endif
}
__host__ __device__ __forceinline__ bool quotient_range(double a)
{
    return (hi32(bits(a)) & 0x7fffffffu) - 0x20000000u < 0x3ff00000u;  // 2^-511 <= |a| < 2^512
}
__host__ __device__ __forceinline__ double quotient(double a, double y, double z)
{
    double q = a * z;
    q = fused(fused(-y, q, a), z, q);
    return fused(fused(-y, q, a), z, q);
}
// a / 3: RN(1/3) is a quarter ulp off, so that a z is within an ulp at once.  3 operations.
__host__ __device__ __forceinline__ double quotient3(double a)
{
    const double z = 1.0 / 3.0, q = a * z;
    return fused(fused(-3.0, q, a), z, q);
}

// ---- reciprocal --------------------------------------------------------------------------------------------------
__host__ __device__ __forceinline__ uint64_t mul_hi64(uint64_t a, uint64_t b)
{
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)((unsigned __int128)a * b >> 64);
#endif
}

// 1 / r rounded to nearest for a positive r in quotient_range, from y0, a 32-bit fraction (units of 2^-32) within
// 2^-20 of 1 / m, where m in [1, 2) is r's mantissa.  Two Newton steps y (2 - m y) in fixed point give y to some units
// of 2^-62; the quotient q = 2^105 / M of the integer mantissa M, rounded from it, is then within one of the correctly
// rounded one, which the exact remainder 2^105 - q M, taken modulo 2^64, tells (no ties: M divides no such power
// unless it is one itself, and then the remainder is 0).  Some 50 integer instructions for the FP64 division's
// dependent FP64 operations.  512^2 D2Q9: 49.2 -> 47.3 us a step; D3Q19 lattices (64^3 109 us), the FP64 maps and
// four lanes a node (7.1 -> 7.2 us) gain nothing, and keep the division.
__host__ __device__ __forceinline__ double reciprocal_from(double r, uint32_t y0)
{
    const uint64_t b = bits(r), M = mantissa(b), m = M << 11;  // m in units of 2^-63
    // e = 1 - m y0, |e| < 2^-20, in units of 2^-50; y1 in units of 2^-63
    const uint64_t p = (uint64_t)hi32(m) * y0 + ((uint64_t)(uint32_t)m * y0 >> 32);
    const int32_t e0 = (int32_t)((int64_t)((1ull << 63) - p) >> 13);
    const uint64_t y1 = ((uint64_t)y0 << 31) + (uint64_t)((int64_t)e0 * (int64_t)(uint64_t)(y0 >> 1) >> 18);
    // e1 = 1 - m y1, |e1| < 2^-38, in units of 2^-62
    const int32_t e1 = (int32_t)((1ull << 62) - mul_hi64(m, y1));
    const uint64_t y2 = y1 + (uint64_t)((int64_t)e1 * (int64_t)(uint64_t)(hi32(y1)) >> 30);
    uint64_t q = (y2 + 512) >> 10;
    const int64_t rem = (int64_t)(0 - q * M) * 2;  // 2^105 is 0 modulo 2^64
    q = rem > (int64_t)M ? q + 1 : (rem < -(int64_t)M ? q - 1 : q);
    return from_bits(q + ((uint64_t)(uint32_t)(2044 - exponent(b)) << 52));
}

#ifdef __CUDACC__
__device__ __forceinline__ double reciprocal(double r)
{
    const uint64_t b = bits(r);
    float y;  // the hardware's approximation, within 2^-22, of the mantissa's leading 24 bits
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(0x3f800000u | (uint32_t)(b >> 29 & 0x7fffffu))));
    // y in [1/2, 1]: its mantissa is a fraction; 1 itself becomes the greatest fraction
    const uint32_t f = max(__float_as_uint(y), 0x3f000000u);
    return reciprocal_from(r, f >= 0x3f800000u ? 0xffffffffu : (f | 0x800000u) << 8);
}
#endif

// ---- populations in fixed point --------------------------------------------------------------------------------
// A population 2^-7 <= f < 1 is a whole number of units of 2^-59 below 2^59.

constexpr int FIX_E0 = 1016;  // exponent field of 2^-7

// max over values of fix_range is below this when all of them are in range (negative ones and NaN are not): up to 1
// for nine populations, up to 1/2 for nineteen, so that their sum stays below 2^63 units
constexpr uint32_t FIX_SPAN = 7u << 20, FIX_SPAN_HALF = 6u << 20;
__host__ __device__ __forceinline__ uint32_t fix_range(double f) { return hi32(bits(f)) - ((uint32_t)FIX_E0 << 20); }

__host__ __device__ __forceinline__ int64_t to_fixed(double f)
{
    const uint64_t b = bits(f);
    return (int64_t)(mantissa(b) << (((hi32(b) >> 20) - FIX_E0) & 7u));
}

__host__ __device__ __forceinline__ int clz32(uint32_t x)
{
#ifdef __CUDA_ARCH__
    return __clz((int)x);
#else
    return x ? __builtin_clz(x) : 32;
#endif
}
__host__ __device__ __forceinline__ int clz64(uint64_t x)
{
#ifdef __CUDA_ARCH__
    return __clzll((long long)x);
#else
    return x ? __builtin_clzll(x) : 64;
#endif
}

// x rounded to 53 significant bits, ties to even (|x| < 2^63).  Rounding by the floor of x + half works on
// two's complement as it is; the magnitude's leading bit is found on x or its complement.
__host__ __device__ __forceinline__ int64_t round53(int64_t x)
{
    const int32_t h = (int32_t)hi32((uint64_t)x);
    const int k0 = 11 - clz32((uint32_t)(h ^ (h >> 31)));
    const int k = k0 > 0 ? k0 : 0;
    const uint32_t mask = (1u << k) - 1;
    const uint64_t r = (uint64_t)x + (mask >> 1) + (((uint32_t)x >> k) & mask & 1u);
    return (int64_t)(r & ~(uint64_t)mask);
}

// A fixed-point number of at most 53 significant bits as a double.
__host__ __device__ __forceinline__ double to_double(int64_t x)
{
    const uint64_t a = x < 0 ? 0 - (uint64_t)x : (uint64_t)x;
    const int lz = clz64(a) & 63;
    const uint64_t m = (a << lz) >> 11;  // leading bit at 52: it adds 1 to the exponent field
    const uint64_t b = m + ((uint64_t)(uint32_t)(1026 - lz) << 52);
    return from_bits(a == 0 ? 0 : b | ((uint64_t)x & 0x8000000000000000ull));
}

}  // namespace fp64int
}  // namespace erlbm
