// modesum_fx.cuh -- the plane-wave mode sum in fixed-point integers.
//
// An FP64 instruction holds its SM sub-partition's FP64 pipe for 64 cycles on
// this part (0.5 lanes a clock), an integer multiply-add 32 x 32 + 64 -> 64
// bits a little over 2.  The sum needs no floating point: a phase is already
// an exact 64-bit fraction of a revolution, its cosine and the amplitudes lie
// in known ranges.  So each term is evaluated and summed in integers and one
// conversion per component makes the double.  The FP64 cosine and sums took
// about 2900 cycles a warp and mode; a run of 65,536 particles over 10 steps in
// a 512-mode field (host buffers in and out) went from 49.8 to 4.8 ms, and a
// training run on 131,072 samples of such a field from 9.64 to 6.60 ms.  It is
// bound by the issue of 126 instructions a mode (43 multiply-adds, 65 on the
// half-rate integer pipe) and by four warps on one sub-partition where others
// have three.
//
// Accuracy, against quadruple precision: the cosine is off by 2^-53.9 rms and
// 2^-51.4 at most, the FP64 form (whose phase rounds before its cosine) by
// 2^-53.2 and 2^-50.9; the sums carry 2^-61 of the sum of the |amplitudes|.
// Whole sums of 1, 512, 4096 and 16384 modes of one size are off by 0.97e-16,
// 1.4e-16, 7.3e-16 and 2.5e-15 of their rms, the FP64 form's by 1.5e-16,
// 7.6e-16, 2.1e-15 and 4.1e-15; the share grows with the number of modes, and
// past kMaxModes the sums stay in FP64.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace tp {
namespace fx {

constexpr int kChunk = 8;           // modes between two carries of the low sums; tables are padded to it
constexpr int kMaxModes = 16384;
constexpr int kTab = 1024;          // cosine table intervals per quarter revolution

// One mode: lattice vector, phase offset (32-bit revolutions) and six
// amplitudes a = ah 2^31 + al 2 (|al| <= 2^29) in units of the component's scale.
struct alignas(16) Mode {
    int n[3];
    uint32_t ph;
    int ah[6];
    int al[6];
};

// Table entry i of the angle phi = i (pi/2) / kTab: C = cos phi in Q62 as
// (C >> 31, C & (2^31 - 1)), and 2 pi sin phi in Q60 as (>> 32, low word >> 1).
// int4: x, y the cosine, z, w the sine.

// acc + a b, 32 x 32 + 64 bits, signed.  Spelled out on the device: where the
// compiler knows a factor not to be negative it widens the two factors
// differently and multiplies in 64 bits, four instructions for one.
__host__ __device__ __forceinline__ int64_t mad(int32_t a, int32_t b, int64_t acc)
{
#ifdef __CUDA_ARCH__
    int64_t r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(acc));
    return r;
#else
    return acc + (int64_t)a * b;
#endif
}

// High and low parts of cos(2 pi ph / 2^64) = (ch 2^32 + cl 4) / 2^62.
// The revolution is folded into its first quarter, p = angle * 2^64 / 2 pi in
// [0, 2^62]; the nearest table point is within d = 2 pi 2^-13, and
// cos(phi + d) = C - S d - C d^2/2 + S d^3/6 + C d^4/24 (the next term is
// below 2^-58): S d in 52 x 63 bits, the quadratic term (below 2^-21) in
// 32 x 32 bits, the last two (below 2^-33) in FP32.
__host__ __device__ __forceinline__ void cosine(uint64_t ph, const int4* tab, int& ch, int& cl)
{
    const int64_t m1 = (int64_t)ph >> 63;
    uint64_t p = ph ^ (uint64_t)m1;                      // cos is even: [0, 2^63)
    const int64_t m2 = (int64_t)(p << 1) >> 63;          // past a quarter: cos(pi - a) = -cos(a)
    p = (p ^ (uint64_t)m2) & 0x7fffffffffffffffull;
    const uint32_t idx = (uint32_t)((p + (1ull << 51)) >> 52);
    const int64_t t = (int64_t)(p - ((uint64_t)idx << 52));  // [-2^51, 2^51)
    const int4 e = tab[idx];
    const int32_t th = (int32_t)(t >> 20);
    const int32_t tl = (int32_t)((uint32_t)t << 12 >> 1);    // low 20 bits, scaled to 31
    // S d in Q62: (sh 2^32 + sl 2) (th 2^20 + tl 2^-11) 2^-62
    const int64_t a1 = mad(e.z, th, 0);
    const int64_t a2 = mad(e.z, tl, mad(e.w, th, 0));
    // C d^2 / 2 in Q62: z = t^2 2^-71 with the dropped bits of t at their middle
    const int64_t t2 = mad(th, th, th);
    const uint32_t z = (uint32_t)((uint64_t)(t2 + (1ll << 30)) >> 31);
    const uint32_t zz = (uint32_t)(((uint64_t)z * 2649351758u + (1ull << 30)) >> 31);  // (2 pi)^2 / 2 * 2^27
    const uint64_t quad = (uint64_t)(uint32_t)e.x * zz;
    // S d^3 / 6 + C d^4 / 24 in Q62
    const float tf = (float)th * 4.656612873077393e-10f;     // 2^-31
    const float zf = tf * tf;
    const float r = zf * ((float)e.z * tf * 2.0561676e-1f + (float)(uint32_t)e.x * zf * 3.0965516e-5f);
    const int32_t corr = (int32_t)r;
    int64_t c = ((int64_t)(uint32_t)e.x << 31) + (uint32_t)e.y;
    c -= (a1 + (a2 >> 31)) >> 10;
    c -= (int64_t)(quad >> 22);
    c += corr;
    c ^= m2;
    ch = (int32_t)(c >> 32);
    cl = (int32_t)((uint32_t)c >> 2);
}

// The six components at the point with box fractions u (64-bit fixed point),
// as integers to be multiplied with the components' scales.  nm is a multiple
// of kChunk (tables are padded with zero amplitudes).  Chunks first, first +
// step, ... only: the sums of all of them add up exactly.  U modes are unrolled:
// a whole chunk where a thread has a particle of its own (65,536 particles x 10
// steps, 512 modes: 5.10 ms with four, 4.83 with eight; 30,000: 2.95 and 2.71;
// only 30,000 with 2,000 modes, whose table leaves L1, loses 1.3 %), four where
// four lanes share one and the warps are many (19,000: 1.70 and 1.72 ms).
template <int U>
__host__ __device__ __forceinline__ void mode_sum(const Mode* modes, int nm, const int4* tab, const uint64_t u[3],
                                                  int64_t out[6], int first = 0, int step = 1)
{
    // u = uh 2^32 + ul with signed ul, so that n u mod 2^64 takes signed products
    int32_t ul[3];
    uint32_t uh[3];
    for (int k = 0; k < 3; k++) {
        ul[k] = (int32_t)(uint32_t)u[k];
        uh[k] = (uint32_t)(u[k] >> 32) + (uint32_t)(ul[k] < 0);
    }
    int64_t hh[6] = {0, 0, 0, 0, 0, 0}, mid[6] = {0, 0, 0, 0, 0, 0};
    for (int m0 = first * kChunk; m0 < nm; m0 += step * kChunk) {
#ifdef __CUDA_ARCH__
#pragma unroll U
#endif
        for (int m = m0; m < m0 + kChunk; m++) {
            int4 r[4];
#ifdef __CUDA_ARCH__
#pragma unroll
            for (int q = 0; q < 4; q++) r[q] = __ldg(reinterpret_cast<const int4*>(modes + m) + q);
#else
            for (int q = 0; q < 4; q++) r[q] = reinterpret_cast<const int4*>(modes + m)[q];
#endif
            uint64_t ph = (uint64_t)mad(r[0].z, ul[2], mad(r[0].y, ul[1], mad(r[0].x, ul[0], 0)));
            const uint32_t hi = (uint32_t)r[0].x * uh[0] + (uint32_t)r[0].y * uh[1] + (uint32_t)r[0].z * uh[2] +
                                (uint32_t)r[0].w;
            ph += (uint64_t)hi << 32;
            int ch, cl;
            cosine(ph, tab, ch, cl);
            const int ah[6] = {r[1].x, r[1].y, r[1].z, r[1].w, r[2].x, r[2].y};
            const int al[6] = {r[2].z, r[2].w, r[3].x, r[3].y, r[3].z, r[3].w};
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
            for (int k = 0; k < 6; k++) {
                hh[k] = mad(ah[k], ch, hh[k]);
                mid[k] = mad(al[k], ch, mad(ah[k], cl, mid[k]));
            }
        }
        // |mid| < 2^63 over a chunk: carry it up
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int k = 0; k < 6; k++) {
            hh[k] += (mid[k] + (1ll << 29)) >> 30;
            mid[k] = 0;
        }
    }
    for (int k = 0; k < 6; k++) out[k] = hh[k];
}

}  // namespace fx
}  // namespace tp
