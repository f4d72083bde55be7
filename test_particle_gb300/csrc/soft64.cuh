// soft64.cuh -- FP64 division, square root, sine and cosine in integers.
//
// An FP64 instruction holds its SM sub-partition's FP64 pipe for 64 cycles on
// this part (0.5 lanes a clock); an integer multiply-add takes about 2 and an
// add 1, on pipes the FP64 kernels leave idle (7.7 % of issue slots used).  A
// division or square root is eight to ten dependent FP64 instructions, so the
// same correctly rounded result is made here from the operands' bits in 60 to
// 75 integer instructions.
//
// Method: an approximate reciprocal (or reciprocal square root) of 23 bits
// from the FP32 unit, one Newton step in 32-bit fixed point, two digits of
// the result from it (an underestimate by a few units of its 59th bit), and
// the exact remainder of the truncated 53-bit result modulo 2^64, whose sign
// against half a unit decides the rounding.  Neither operation has ties.
// Operands outside the exponent window (zero, subnormal, huge, infinite, NaN)
// take the FP64 instructions.
#pragma once
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

namespace tp {
namespace sd {

#ifdef __CUDA_ARCH__
__device__ __forceinline__ uint64_t bits(double v) { return (uint64_t)__double_as_longlong(v); }
__device__ __forceinline__ double value(uint64_t b) { return __longlong_as_double((long long)b); }
__device__ __forceinline__ float fvalue(uint32_t b) { return __uint_as_float(b); }
__device__ __forceinline__ uint32_t fbits(float v) { return __float_as_uint(v); }
__device__ __forceinline__ uint32_t mulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_approx(float x)
{
    float r;
    asm("rsqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
#else
inline uint64_t bits(double v) { uint64_t b; memcpy(&b, &v, 8); return b; }
inline double value(uint64_t b) { double v; memcpy(&v, &b, 8); return v; }
inline float fvalue(uint32_t b) { float v; memcpy(&v, &b, 4); return v; }
inline uint32_t fbits(float v) { uint32_t b; memcpy(&b, &v, 4); return b; }
inline uint32_t mulhi(uint32_t a, uint32_t b) { return (uint32_t)((uint64_t)a * b >> 32); }
#ifndef TP_SOFT64_HOST_APPROX  // a host test may bring approximations of its own
inline float rcp_approx(float x) { return 1.0f / x; }
inline float rsqrt_approx(float x) { return (float)(1.0 / sqrt((double)x)); }
#endif
#endif

// exponents within 2^-447 .. 2^448: quotients and roots of such operands are normal
__host__ __device__ __forceinline__ bool in_window(uint32_t hi)
{
    return (hi & 0x7ff00000u) - (576u << 20) < (896u << 20);
}

// A divisor prepared for any number of quotients: its 53-bit significand and
// x = 2^92 / (significand 2^8) from below, good to about 2^-30.
struct Divisor {
    double v;
    uint32_t mh, ml;   // significand, high 21 and low 32 bits
    uint32_t x;
    uint32_t hi;       // high word of v (sign, exponent)
};

__host__ __device__ __forceinline__ Divisor divisor(double b)
{
    Divisor d;
    const uint64_t B = bits(b);
    d.v = b;
    d.hi = (uint32_t)(B >> 32);
    d.ml = (uint32_t)B;
    d.mh = (d.hi & 0xfffffu) | 0x100000u;
    // the significand as a float in [1, 2), its reciprocal in (0.5, 1) as 2^32
    // units: the float is rounded up, so that a reciprocal of 1 does not occur
    const uint32_t top = (uint32_t)((((uint64_t)d.mh << 32) | d.ml) >> 21);  // 2^31 .. 2^32
    const float f = fvalue(0x3f800001u + ((top << 1) >> 9));
    const uint32_t x0 = (fbits(fmaxf(rcp_approx(f), 0.5f)) << 8) | 0x80000000u;
    // Newton: x1 = x0 + x0 (1 - x0 b), the bracket from the high product
    const int32_t e = (int32_t)(0x80000000u - mulhi(x0, top));
    // (e is within +-1024; it is overestimated by the truncations, in all by
    // less than 5 units of x)
    d.x = x0 + (uint32_t)((uint64_t)x0 * (uint32_t)(e + 1024) >> 31) - (x0 >> 21) - 6u;
    return d;
}

// a / d, round to nearest even
__host__ __device__ __forceinline__ double div(double a, const Divisor& d)
{
    const uint64_t A = bits(a);
    const uint32_t ahi = (uint32_t)(A >> 32), al = (uint32_t)A;
    if (!(in_window(ahi) && in_window(d.hi))) {
        if (A << 1 == 0 && in_window(d.hi)) return value((A ^ (uint64_t)d.hi << 32) & 0x8000000000000000ull);
        return a / d.v;
    }
    const uint32_t ah = (ahi & 0xfffffu) | 0x100000u;
    const uint64_t a6 = (((uint64_t)ah << 32) | al) << 6;          // [2^58, 2^59)
    const uint64_t b7 = (((uint64_t)d.mh << 32) | d.ml) << 7;      // [2^59, 2^60)
    // q1 ~ a 2^32 / b from below by at most 12, remainder below 13 b < 2^64
    const uint32_t q1 = mulhi((uint32_t)(a6 >> 27), d.x);
    const uint64_t rem = ((uint64_t)(uint32_t)a6 << 32) - (uint64_t)q1 * (uint32_t)b7 -
                         ((uint64_t)(q1 * (uint32_t)(b7 >> 32)) << 32);
    const uint32_t q2 = (uint32_t)((uint64_t)(uint32_t)(rem >> 32) * d.x >> 31);
    const uint64_t q = ((uint64_t)q1 << 28) + q2;                  // a 2^60 / b, from below
    const uint32_t big = (uint32_t)(q >> 59);                      // the significand of a is not below b's
    const uint64_t t = q >> (6 + big);                             // 53 bits
    // 2 (a 2^s - t b) - b modulo 2^64: positive where the rest passes half a unit
    const uint64_t t2 = 2 * t + 1;
    const uint32_t tl = (uint32_t)t2, th = (uint32_t)(t2 >> 32);
    const uint64_t p = (uint64_t)tl * d.ml + ((uint64_t)(tl * d.mh + th * d.ml) << 32);
    const int64_t w = (int64_t)(((uint64_t)(al << (22 - big)) << 32) - p);
    uint64_t r = t + (uint64_t)(w > 0);
    const uint32_t e = (ahi & 0x7ff00000u) - (d.hi & 0x7ff00000u) + ((1021u + big) << 20);
    r += (uint64_t)(e | ((ahi ^ d.hi) & 0x80000000u)) << 32;
    return value(r);
}

__host__ __device__ __forceinline__ double div(double a, double b) { return div(a, divisor(b)); }

// square root, round to nearest even
__host__ __device__ __forceinline__ double sqrt_rn(double v)
{
    const uint64_t V = bits(v);
    const uint32_t hi = (uint32_t)(V >> 32), lo = (uint32_t)V;
    if ((hi >> 31) || !in_window(hi)) return sqrt(v);
    // m = significand at an even exponent, [2^62, 2^64)
    const uint32_t odd = ~(hi >> 20) & 1u;  // exponent - 1023 odd
    const uint64_t m = (((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | lo) << (10 + odd);
    const uint32_t mh = (uint32_t)(m >> 32);
    // y ~ 2^32 2^31 / sqrt(m) from below: FP32, then one Newton step
    const float f = fvalue(0x3f800000u + (odd << 23) + ((((hi << 12) | (lo >> 20))) >> 9));
    const float y0f = fminf(fmaxf(rsqrt_approx(f), 0.5f), 0.99999994f);
    const uint32_t y0 = (fbits(y0f) << 8) | 0x80000000u;
    // g = m y^2: 2^30 (1 + 2 e) from which y (1 - e)
    const uint32_t g = mulhi(mulhi(y0, y0), mh);                   // ~ 2^30
    const int32_t e = (int32_t)(0x40000000u - g);                  // -2 e 2^30
    const uint32_t y = y0 + (uint32_t)((int64_t)((uint64_t)y0 * (uint32_t)(e + 1024) >> 31)) - (y0 >> 21) - 6u;
    // s1 ~ sqrt(m) from below (32 bits), remainder, next digit of 27 bits
    const uint32_t s1 = (uint32_t)((uint64_t)mh * y >> 31);
    const uint64_t rem = m - (uint64_t)s1 * s1;
    const uint32_t r32 = (uint32_t)(rem >> 6);
    const uint32_t s2 = (uint32_t)((uint64_t)r32 * y >> 31);
    const uint64_t s = ((uint64_t)s1 << 27) + s2;                  // 59 bits, from below
    const uint64_t t = (s - 6) >> 6;                               // 53 bits
    // m 2^42 - t^2 - t modulo 2^64: positive where the root passes t + 1/2
    const uint32_t tl = (uint32_t)t, th = (uint32_t)(t >> 32);
    const uint64_t p = (uint64_t)tl * tl + ((uint64_t)(2u * tl * th) << 32) + t;
    const int64_t w = (int64_t)(((uint64_t)((uint32_t)m << 10) << 32) - p);
    uint64_t r = t + (uint64_t)(w > 0);
    // exponent: (e - 1023 - odd) / 2 + 1023, less the significand's own bit
    r += (uint64_t)((((hi >> 20) - odd + 1023u) >> 1) - 1u) << 52;
    return value(r);
}

// (z a) >> 64, less at most 2
__host__ __device__ __forceinline__ uint64_t mul64(uint64_t z, uint64_t a)
{
    const uint32_t zh = (uint32_t)(z >> 32), zl = (uint32_t)z, ah = (uint32_t)(a >> 32), al = (uint32_t)a;
    return (uint64_t)zh * ah + (uint32_t)((uint64_t)zh * al >> 32) + (uint32_t)((uint64_t)zl * ah >> 32);
}

// sin x and cos x within 0.513 units of the last place (0.5122 the most in 40
// million arguments).  x = M 2^(E - 52) is
// reduced by its product with 2 / pi in 96 bits (Payne and Hanek, for the
// exponents taken here the leading words are enough): k quarter turns and
// f in [-1/2, 1/2] of one, kept both in fixed point and normalised.  The two
// Taylor polynomials in z = f^2 run in 64-bit fixed point (their last four
// terms in 32 bits), and sin = f P(z) is multiplied from the normalised f, so
// that its relative precision does not depend on f.
// Outside 2^-12 <= |x| < 2^10, and within 2^-20 quarter turns of a multiple of
// pi / 2, the CUDA functions.
__host__ __device__ __forceinline__ void sin_cos(double x, double& sn, double& cs)
{
    const uint64_t X = bits(x);
    const uint32_t hi = (uint32_t)(X >> 32), ml = (uint32_t)X;
    const uint32_t ex = (hi >> 20) & 0x7ffu;
    if (ex - 1011u < 22u) {
        const uint32_t mh = (hi & 0xfffffu) | 0x100000u;
        const uint32_t c2 = 0xa2f9836eu, c1 = 0x4e441529u, c0 = 0xfc2757d1u;  // 2 / pi
        const uint64_t t0 = (uint64_t)ml * c0;
        const uint64_t t1 = (uint64_t)ml * c1 + (t0 >> 32);
        const uint64_t t2 = (uint64_t)ml * c2 + (t1 >> 32);
        const uint64_t u0 = (uint64_t)mh * c0 + (uint32_t)t1;
        const uint64_t u1 = (uint64_t)mh * c1 + (uint32_t)t2 + (u0 >> 32);
        const uint64_t u2 = (uint64_t)mh * c2 + (t2 >> 32) + (u1 >> 32);
        // the binary point to the top of the third word
        const uint32_t sh = ex - 1011u;
        const uint32_t p1 = (uint32_t)u0, p2 = (uint32_t)u1, p3 = (uint32_t)u2, p4 = (uint32_t)(u2 >> 32);
        uint32_t k = (uint32_t)(((uint64_t)p4 << sh) >> 32);
        uint32_t f2 = (uint32_t)((((uint64_t)p4 << 32 | p3) << sh) >> 32);
        uint32_t f1 = (uint32_t)((((uint64_t)p3 << 32 | p2) << sh) >> 32);
        uint32_t f0 = (uint32_t)((((uint64_t)p2 << 32 | p1) << sh) >> 32);
        k += f2 >> 31;
        const uint32_t neg = (uint32_t)((int32_t)f2 >> 31);  // f < 0
        f2 ^= neg; f1 ^= neg; f0 ^= neg;
#ifdef __CUDA_ARCH__
        const uint32_t lz = (uint32_t)__clz((int)f2);
#else
        const uint32_t lz = f2 ? (uint32_t)__builtin_clz(f2) : 32u;
#endif
        if (lz <= 20u) {
            const uint32_t F1 = (uint32_t)((((uint64_t)f2 << 32 | f1) << lz) >> 32);
            const uint32_t F0 = (uint32_t)((((uint64_t)f1 << 32 | f0) << lz) >> 32);
            const uint64_t z = (uint64_t)f2 * f2 + ((uint64_t)f2 * f1 >> 31);
            const uint32_t zh = (uint32_t)(z >> 32);
            // (pi/2)^(2n+1) / (2n+1)! and (pi/2)^(2n) / (2n)!, in 2^-61 (the last in 2^-55 and 2^-52)
            const uint32_t s6 = 0x7a3d0d34u - mulhi(zh, 0x16fadbau - mulhi(zh, 0x355d8u));
            uint64_t s = 0x78c1d3f7a22ull - ((uint64_t)zh * s6 >> 26);
            s = 0x150783487ee78ull - mul64(z, s);
            s = 0x265a599cc57b0bull - mul64(z, s);
            s = 0x28cd78ceeb55c3aull - mul64(z, s);
            s = 0x14abbce625be52bfull - mul64(z, s);
            s = 0x3243f6a8885a308dull - mul64(z, s);
            const uint32_t c6 = 0x7e74e28eu - mulhi(zh, 0x1b6e24fu - mulhi(zh, 0x48319u - mulhi(zh, 0x950u)));
            uint64_t c = 0x34da3e544095ull - ((uint64_t)zh * c6 >> 23);
            c = 0x787d41a246eafull - mul64(z, c);
            c = 0xaae9e3f1e5ffd0ull - mul64(z, c);
            c = 0x81e0f840dad61daull - mul64(z, c);
            c = 0x277a79937c8bbcb5ull - mul64(z, c);
            c = 0x2000000000000000ull - mul64(z, c);
            s = mul64((uint64_t)F1 << 32 | F0, s);
            const uint32_t b = (uint32_t)(s >> 61);
            uint64_t S = ((s + (128u << b)) >> (8 + b)) + ((uint64_t)(1021u + b - lz) << 52);
            uint64_t Cv = ((c + 128u) >> 8) + ((uint64_t)1021u << 52);
            // signs: sin of the reduced angle is odd in f
            S ^= (uint64_t)(neg & 0x80000000u) << 32;
            const uint64_t a = k & 1u ? Cv : S, d = k & 1u ? S : Cv;
            sn = value(a ^ (uint64_t)((hi ^ (k << 30)) & 0x80000000u) << 32);
            cs = value(d ^ (uint64_t)(((k + 1u) << 30) & 0x80000000u) << 32);
            return;
        }
    }
    sn = sin(x);
    cs = cos(x);
}

}  // namespace sd
}  // namespace tp
