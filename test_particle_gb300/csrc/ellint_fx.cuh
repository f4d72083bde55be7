// ellint_fx.cuh -- the elliptic integrals of the loop's field in fixed point.
//
// K(m) and E(m) by the same piecewise series as ellint64 (fields_fp64.cuh), the
// polynomials in 64-bit integers: at 64 cycles an FP64 instruction the 37 terms
// of an interval cost 6000 cycles there and about 700 here.  The argument is
// u = 16 |m - m0| < 0.8 and the coefficients are scaled to it; even and odd
// powers run as two chains in z = u^2, in units of 2^-61.  Above m = 0.9 the
// same two polynomials, with other rows of the table, are the parts of K and E
// of the reference's formula, and a third series gives the nome.
// Against quadruple precision, corrected coefficients, 3,000,000 values of m: up to
// 0.9 K and E are off by at most 4.7e-16 and 4.2e-16 of their value, the FP64
// series by 1.04e-15 and 1.08e-15; above, K by 6.5e-16 (9.4e-16) and E, which
// cancels towards m = 1, by 4.1e-15 (4.3e-15).  Only within 1e-13 of m = 1 is the
// worst K the larger one, 6.1e-16 against 4.5e-16.  4,096 particles x 200 steps, two wires and
// loops: 8.9 -> 4.5 ms; 20,000 x 50: 9.8 -> 4.6 ms.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "soft64.cuh"

namespace tp {
namespace ellfx {

// Rows of the table: K of intervals 0..9 and interval 9 with the reference's
// coefficient (20 terms each); E of intervals 0..9, then the series of its
// branch above 0.9 (17 each); the nome's 14 terms; the intervals' centres.
constexpr int kRows = 11, kK = 20, kE = 17, kQ = 14;
constexpr int kOffE = kRows * kK, kOffQ = kOffE + kRows * kE, kOffC = kOffQ + kQ, kSize = kOffC + kRows;

#ifdef __CUDA_ARCH__
__device__ __forceinline__ uint64_t at(const uint64_t* t, int i)
{
    return __ldg(reinterpret_cast<const unsigned long long*>(t) + i);
}
#else
inline uint64_t at(const uint64_t* t, int i) { return t[i]; }
#endif

// m in [2^-900, 1) to 2^-63
__host__ __device__ __forceinline__ uint64_t fixed63(double m)
{
    const uint64_t b = sd::bits(m);
    const uint32_t sh = 1023u - (uint32_t)(b >> 52);
    const uint64_t v = (b << 11) | 0x8000000000000000ull;
    return sh < 64u ? v >> sh : 0ull;
}

__host__ __device__ __forceinline__ double unit61(uint64_t v) { return (double)v * 4.336808689942018e-19; }

// K, E by the reference's formulas (src/wlcs.c:460-809); false where m is not
// inside (0, 1): take ellint64
__host__ __device__ __forceinline__ bool integrals(const uint64_t* tab, double m, int corrected, double& elle, double& ellf)
{
    const uint32_t ex = (uint32_t)(sd::bits(m) >> 52);
    if (ex - 123u >= 900u) return false;  // zero, tiny, negative, one and above, NaN
    const uint64_t M = fixed63(m);
    const bool high = !(m < 0.9);
    const int i = m < 0.8 ? (int)(((M >> 32) * 10) >> 31) : m < 0.85 ? 8 : 9;
    const int rk = high ? 0 : i == 9 && !corrected ? 10 : i, re = high ? 10 : i;
    // distances from the centres (0.95 above 0.9), signed
    const int64_t d = (int64_t)(M - at(tab, kOffC + (high ? 10 : i)));
    const bool below = d < 0;
    const uint64_t u = (uint64_t)(below ? -d : d) << 5;  // 16 |d| in 2^-64
    const uint64_t z = sd::mul64(u, u);
    const uint64_t *ck = tab + rk * kK, *ce = tab + kOffE + re * kE;
    uint64_t k0 = at(ck, 18), k1 = at(ck, 19), e0 = at(ce, 16), e1 = at(ce, 15);
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int j = 16; j >= 2; j -= 2) {
        k0 = at(ck, j) + sd::mul64(z, k0);
        k1 = at(ck, j + 1) + sd::mul64(z, k1);
        if (j <= 14) {
            e0 = at(ce, j) + sd::mul64(z, e0);
            e1 = at(ce, j - 1) + sd::mul64(z, e1);
        }
    }
    k0 = at(ck, 0) + sd::mul64(z, k0);
    k1 = at(ck, 1) + sd::mul64(z, k1);
    e0 = sd::mul64(z, e0);  // without its constant
    k1 = sd::mul64(u, k1);
    e1 = sd::mul64(u, e1);
    if (!high) {
        ellf = unit61(below ? k0 - k1 : k0 + k1);
        // E's coefficients past the constant are negative
        elle = unit61(at(ce, 0) - e0 - (below ? 0 - e1 : e1));
        return true;
    }
    // the first series runs in m - 0.95 (the reference) or 0.95 - m (corrected),
    // the last in 0.95 - m
    const bool neg = corrected ? !below : below;
    const double ellf1 = unit61(neg ? k0 - k1 : k0 + k1);
    const double hm = unit61(at(ce, 0) + e0 + (below ? e1 : 0 - e1));
    const uint64_t v = (0x8000000000000000ull - M) << 4;  // 8 (1 - m) in 2^-64
    uint64_t s = at(tab, kOffQ + kQ - 1);
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int j = kQ - 2; j >= 0; j--) s = at(tab, kOffQ + j) + sd::mul64(v, s);
    const double q1 = (1.0 - m) * unit61(s);
    ellf = -log(q1) * sd::div(ellf1, 3.14159265358979323846);
    elle = sd::div(1.0, ellf1) * (3.14159265358979323846 / 2.0 + ellf * hm);
    return true;
}

}  // namespace ellfx
}  // namespace tp
