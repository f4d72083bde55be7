// fields_fp64.cuh -- FP64 field evaluation on the device.
//
// Each function follows the reference function named in its comment.  In the
// parity build (-fmad=false: no multiply-add is fused) a field differs from the
// reference's by:
//   gridded fields   nothing: the same roundings, in FP32 with carried errors
//                    where those are certain (interp_filtered), else in double;
//   analytic ABC     sine and cosine in fixed point (soft64.cuh, 0.513 units of
//                    the last place), the sums in the reference's order;
//   wires            the same sine and cosine, CUDA's arc cosine and Bessel terms;
//   loops            K and E in fixed point (ellint_fx.cuh, 6.5e-16 and 4.1e-15 of
//                    their value at most), CUDA's logarithm, the rest in order;
//                    the adaptive stepper keeps the FP64 series;
//   mode sum         the whole sum in fixed point (modesum_fx.cuh; its header has
//                    the errors by number of modes), in FP64 outside its range.
// Divisions and square roots are correctly rounded throughout.
#pragma once
#include "ellint_fx.cuh"
#include "tp_common.cuh"

// In global memory, read through L1: the lanes of a warp index different
// intervals, and constant-cache reads of different addresses serialise.
#define TP_ELL_QUAL __device__ static const
#include "ellint_coeffs.h"
#undef TP_ELL_QUAL

namespace tp {

#ifndef TP_PI
#define TP_PI 3.14159265358979323846
#endif

// get_trilinar_parameters + grid_indices, src/interpolation.c:36-181
struct Tri64 {
    long c[8];
    double w[8];
    double dt;
};

__device__ __forceinline__ long idx3(int nx, int ny, int ix, int iy, int iz)
{
    long index = ix;          // index_transfer, src/interpolation.c:119-128
    int shift = nx;
    index += shift * iy;
    shift *= ny;
    index += shift * iz;
    return index;
}

// SOFT: the index quotients in integers (soft64.cuh, one an axis: the same doubles),
// where every sample takes this form; in the push, where one in ten thousand does,
// the FP64 instructions, whose code is the shorter (ABC with either, 65,536
// particles: 1.9 % slower with integers, gridded 0.7 %).
template <bool SOFT = false>
__device__ __forceinline__ void trilinear64(const DevField& f, double x, double y, double z,
                                            double t, Tri64& r)
{
    int nx = f.nx, ny = f.ny, nz = f.nz;
    int ix1, iy1, iz1, ix2, iy2, iz2;
    double dx, dy, dz;
    if (SOFT) {
        const bool ox = x > f.xmax || x < f.xmin, oy = y > f.ymax || y < f.ymin, oz = z > f.zmax || z < f.zmin;
        const double qx = sd::div(ox ? x : x - f.xmin, f.d_gdx), qy = sd::div(oy ? y : y - f.ymin, f.d_gdy),
                     qz = sd::div(oz ? z : z - f.zmin, f.d_gdz);
        ix1 = (int)floor(qx); iy1 = (int)floor(qy); iz1 = (int)floor(qz);
        ix2 = ix1 + 1; iy2 = iy1 + 1; iz2 = iz1 + 1;
        dx = qx - ix1; dy = qy - iy1; dz = qz - iz1;
        if (ox) { ix1 = nx - 1; ix2 = 0; dx = x < f.xmin ? qx + 1.0 : qx - (nx - 1); }
        if (oy) { iy1 = ny - 1; iy2 = 0; dy = y < f.ymin ? qy + 1.0 : qy - (ny - 1); }
        if (oz) { iz1 = nz - 1; iz2 = 0; dz = z < f.zmin ? qz + 1.0 : qz - (nz - 1); }
    } else {
        ix1 = (int)floor((x - f.xmin) / f.gdx);
        iy1 = (int)floor((y - f.ymin) / f.gdy);
        iz1 = (int)floor((z - f.zmin) / f.gdz);
        ix2 = ix1 + 1; iy2 = iy1 + 1; iz2 = iz1 + 1;
        dx = (x - f.xmin) / f.gdx - ix1;
        dy = (y - f.ymin) / f.gdy - iy1;
        dz = (z - f.zmin) / f.gdz - iz1;
        if (x > f.xmax) { ix1 = nx - 1; ix2 = 0; dx = x / f.gdx - (nx - 1); }
        if (y > f.ymax) { iy1 = ny - 1; iy2 = 0; dy = y / f.gdy - (ny - 1); }
        if (z > f.zmax) { iz1 = nz - 1; iz2 = 0; dz = z / f.gdz - (nz - 1); }
        if (x < f.xmin) { ix1 = nx - 1; ix2 = 0; dx = x / f.gdx + 1.0; }
        if (y < f.ymin) { iy1 = ny - 1; iy2 = 0; dy = y / f.gdy + 1.0; }
        if (z < f.zmin) { iz1 = nz - 1; iz2 = 0; dz = z / f.gdz + 1.0; }
    }
    if (f.multi_tframe == 0) {
        r.dt = 0.0;
    } else {
        int it1 = (int)floor(t / f.gdt);
        r.dt = t / f.gdt - it1;
    }
    r.c[0] = idx3(nx, ny, ix1, iy1, iz1);
    r.c[1] = idx3(nx, ny, ix1, iy1, iz2);
    r.c[2] = idx3(nx, ny, ix1, iy2, iz1);
    r.c[3] = idx3(nx, ny, ix2, iy1, iz1);
    r.c[4] = idx3(nx, ny, ix2, iy2, iz1);
    r.c[5] = idx3(nx, ny, ix2, iy1, iz2);
    r.c[6] = idx3(nx, ny, ix1, iy2, iz2);
    r.c[7] = idx3(nx, ny, ix2, iy2, iz2);
    double ax = 1.0 - dx, ay = 1.0 - dy, az = 1.0 - dz;
    if (!f.interp_corrected) {
        // the reference's weights (src/interpolation.c:173-180): corners
        // 1, 3, 4, 6 carry the weight of their x<->z mirror
        r.w[0] = ax * ay * az;
        r.w[1] = dx * ay * az;
        r.w[2] = ax * dy * az;
        r.w[3] = ax * ay * dz;
        r.w[4] = ax * dy * dz;
        r.w[5] = dx * ay * dz;
        r.w[6] = dx * dy * az;
        r.w[7] = dx * dy * dz;
    } else {
        r.w[0] = ax * ay * az;
        r.w[1] = ax * ay * dz;
        r.w[2] = ax * dy * az;
        r.w[3] = dx * ay * az;
        r.w[4] = dx * dy * az;
        r.w[5] = dx * ay * dz;
        r.w[6] = ax * dy * dz;
        r.w[7] = dx * dy * dz;
    }
}

__device__ __forceinline__ bool corner_ok(const DevField& f, long c, int* status)
{
    long ncell = (long)f.nx * f.ny * f.nz;
    if (c < 0 || c >= ncell) {
        if (status) atomicOr(status, ST_BAD_INDEX);
        return false;
    }
    return true;
}

// get_double_velocity_at_point, src/velocity_field.c:555-584
__device__ __forceinline__ void interp_d3(const DevField& f, const Tri64& r, const double* c,
                                          const double* a, const double* b, double out[3],
                                          int* status)
{
    if (f.multi_tframe == 0) {
        double v0 = 0.0, v1 = 0.0, v2 = 0.0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if (!corner_ok(f, r.c[i], status)) continue;
            const double* p = c + 3 * r.c[i];
            v0 += p[0] * r.w[i];
            v1 += p[1] * r.w[i];
            v2 += p[2] * r.w[i];
        }
        out[0] = v0; out[1] = v1; out[2] = v2;
    } else {
        double p[3] = {0.0, 0.0, 0.0}, q[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if (!corner_ok(f, r.c[i], status)) continue;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                p[k] += a[3 * r.c[i] + k] * r.w[i];
                q[k] += b[3 * r.c[i] + k] * r.w[i];
            }
        }
#pragma unroll
        for (int k = 0; k < 3; k++) out[k] = r.dt * p[k] + (1.0 - r.dt) * q[k];
    }
}

// get_float_{b,e}field_at_point / get_float_velocity_at_point,
// src/magnetic_field.c:593-622: float results accumulated through double
__device__ __forceinline__ void interp_f3(const DevField& f, const Tri64& r, const float* c,
                                          const float* a, const float* b, float out[3],
                                          int* status)
{
    if (f.multi_tframe == 0) {
        float v0 = 0.0f, v1 = 0.0f, v2 = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if (!corner_ok(f, r.c[i], status)) continue;
            const float* p = c + 3 * r.c[i];
            v0 = (float)((double)v0 + (double)__ldg(p + 0) * r.w[i]);
            v1 = (float)((double)v1 + (double)__ldg(p + 1) * r.w[i]);
            v2 = (float)((double)v2 + (double)__ldg(p + 2) * r.w[i]);
        }
        out[0] = v0; out[1] = v1; out[2] = v2;
    } else {
        double p[3] = {0.0, 0.0, 0.0}, q[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if (!corner_ok(f, r.c[i], status)) continue;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                p[k] += (double)__ldg(a + 3 * r.c[i] + k) * r.w[i];
                q[k] += (double)__ldg(b + 3 * r.c[i] + k) * r.w[i];
            }
        }
#pragma unroll
        for (int k = 0; k < 3; k++) out[k] = (float)(r.dt * p[k] + (1.0 - r.dt) * q[k]);
    }
}

// ---------------------------------------------------------------- float grids, filtered
// The reference's float-grid interpolation rounds v + p w, formed in double
// from a float v, a float node value p and a double weight w, to a float after
// every corner.  Those roundings are reproduced in FP32: the weight in two
// floats (48 of its 53 bits), the product and the sum with their rounding
// errors (two-product by FMA, two-sum), and a bound d on what is left out.
// Where v + p w - d and v + p w + d round to the same float, so does the
// double sum, whatever its own rounding.  Where they do not (about one
// evaluation in ten thousand), or where an exponent could make an error term
// inexact, the caller takes the double form.  16 FP32 instructions a term
// instead of two FP64 ones (64 pipe cycles each) and three conversions.

// v <- RN32(v + p w); bad: the rounding is not certain
__device__ __forceinline__ void add_term(float& v, float p, float wh, float wl, bool& bad)
{
    const float ph = __fmul_rn(p, wh);
    const float pl = __fmaf_rn(p, wl, __fmaf_rn(p, wh, -ph));
    const float s = __fadd_rn(v, ph), t = __fsub_rn(s, v);
    const float e = __fadd_rn(__fsub_rn(v, __fsub_rn(s, t)), __fsub_rn(ph, t));
    const float rest = __fadd_rn(e, pl);
    // left out: 2^-45.7 |ph| of the product, 2^-24 |rest| in forming rest,
    // |rest| <= 2^-24 |s| + 2^-22.4 |ph|, and the double roundings; in all
    // below 2^-44.9 |ph| + 2^-47.9 |s|
    const float d = __fadd_rn(fabsf(ph), fabsf(s));
    const float r = __fadd_rn(s, __fmaf_rn(d, 5.6843418860808015e-14f, rest));   // 2^-44
    const float q = __fadd_rn(s, __fmaf_rn(d, -5.6843418860808015e-14f, rest));
    // a node value of 2^-60 or less (not zero) could lose bits of its product
    bad |= r != q || (__float_as_uint(p) << 1) - 1u < (0x21800000u << 1) - 1u;
    v = r;
}

// A weight in [2^-36, 1], or 0, as two floats: its leading 24 bits, and the
// other 29 rounded to 24.  bad: outside that range.
__device__ __forceinline__ void split_weight(double w, float& wh, float& wl, bool& bad)
{
    const uint32_t hi = (uint32_t)__double2hiint(w), lo = (uint32_t)__double2loint(w);
    const bool zero = (hi | lo) == 0u;
    bad |= !zero && hi - (987u << 20) > (36u << 20);
    const uint32_t b = ((hi - (896u << 20)) << 3) | (lo >> 29);
    const float scale = __uint_as_float((b & 0x7f800000u) - (52u << 23));
    wh = zero ? 0.0f : __uint_as_float(b);
    wl = zero ? 0.0f : __fmul_rn(__uint2float_rn(lo & 0x1fffffffu), scale);
}

// Index and fraction along one axis inside the box (src/interpolation.c:36-105);
// false where the reference's wrap branches or the array's end would apply.
__device__ __forceinline__ bool cell64(double x, double lo, double hi, const sd::Divisor& d, int n, int& i, double& fr)
{
    const double q = sd::div(x - lo, d), fl = floor(q);
    i = (int)fl;
    fr = q - fl;
    return !(x > hi) && !(x < lo) && (unsigned)i < (unsigned)(n - 1);
}

// NF fields on the same float grid at one point, single time frame, filtered.
// False: not certain, take interp_f3.
template <int NF>
__device__ __forceinline__ bool interp_filtered(const DevField& f, double x, double y, double z, const float* const g[NF],
                                                float out[NF][3])
{
    int ix, iy, iz;
    double dx, dy, dz;
    const bool in = cell64(x, f.xmin, f.xmax, f.d_gdx, f.nx, ix, dx) &
                    cell64(y, f.ymin, f.ymax, f.d_gdy, f.ny, iy, dy) &
                    cell64(z, f.zmin, f.zmax, f.d_gdz, f.nz, iz, dz);
    if (!in) return false;
    const size_t base = ((size_t)((size_t)iz * f.ny + iy) * f.nx + ix) * 3;
    const size_t sy = 3 * (size_t)f.nx, sz = sy * f.ny;
    const size_t off[8] = {0, sz, sy, 3, 3 + sy, 3 + sz, sy + sz, 3 + sy + sz};  // trilinear64's corner order
    float p[NF][8][3];
#pragma unroll
    for (int a = 0; a < NF; a++)
#pragma unroll
        for (int c = 0; c < 8; c++)
#pragma unroll
            for (int k = 0; k < 3; k++) p[a][c][k] = __ldg(g[a] + base + off[c] + k);
    const double ax = 1.0 - dx, ay = 1.0 - dy, az = 1.0 - dz;
    const double w00 = ax * ay, w10 = dx * ay, w01 = ax * dy, w11 = dx * dy;
    double w[8] = {w00 * az, w10 * az, w01 * az, w00 * dz, w01 * dz, w10 * dz, w11 * az, w11 * dz};
    if (f.interp_corrected) {
        double t = w[1]; w[1] = w[3]; w[3] = t;
        t = w[4]; w[4] = w[6]; w[6] = t;
    }
    bool bad = false;
#pragma unroll
    for (int a = 0; a < NF; a++)
#pragma unroll
        for (int k = 0; k < 3; k++) out[a][k] = 0.0f;
#pragma unroll
    for (int c = 0; c < 8; c++) {
        float wh, wl;
        split_weight(w[c], wh, wl, bad);
#pragma unroll
        for (int a = 0; a < NF; a++)
#pragma unroll
            for (int k = 0; k < 3; k++) add_term(out[a][k], p[a][c][k], wh, wl, bad);
    }
    return !bad;
}

// NF fields on float grids in the reference's own arithmetic (any time frames): a
// call in the loops of the push, whose instruction cache it would fill, inline
// (INL below) in the diffusion terms of a batch, which evaluate it twice and where
// the call made a pair in two time frames 71 us instead of 59.
template <int NF>
__device__ __forceinline__ void interp_exact_inline(const DevField& f, double x, double y, double z, double t,
                                                    const float* const g[NF], const float* const ga[NF],
                                                    const float* const gb[NF], float out[NF][3], int* status)
{
    Tri64 r;
    trilinear64(f, x, y, z, t, r);
    for (int a = 0; a < NF; a++) interp_f3(f, r, g[a], ga[a], gb[a], out[a], status);
}

template <int NF>
__device__ __noinline__ void interp_exact(const DevField& f, double x, double y, double z, double t, const float* const g[NF],
                                          const float* const ga[NF], const float* const gb[NF], float out[NF][3],
                                          int* status)
{
    interp_exact_inline<NF>(f, x, y, z, t, g, ga, gb, out, status);
}

// The same for component c alone of each field.
template <int NF>
__device__ __noinline__ void interp_exact_lane(const DevField& f, double x, double y, double z, double t,
                                               const float* const g[NF], const float* const ga[NF],
                                               const float* const gb[NF], int c, float out[NF], int* status)
{
    Tri64 r;
    trilinear64<true>(f, x, y, z, t, r);
#pragma unroll
    for (int a = 0; a < NF; a++) {
        if (f.multi_tframe == 0) {
            float v = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (corner_ok(f, r.c[i], status))
                    v = (float)((double)v + (double)__ldg(g[a] + 3 * r.c[i] + c) * r.w[i]);
            out[a] = v;
        } else {
            double p = 0.0, q = 0.0;
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (corner_ok(f, r.c[i], status)) {
                    p += (double)__ldg(ga[a] + 3 * r.c[i] + c) * r.w[i];
                    q += (double)__ldg(gb[a] + 3 * r.c[i] + c) * r.w[i];
                }
            out[a] = (float)(r.dt * p + (1.0 - r.dt) * q);
        }
    }
}

template <int NF, bool INL = false>
__device__ __forceinline__ void interp_grids(const DevField& f, double x, double y, double z, double t,
                                             const float* const g[NF], const float* const ga[NF],
                                             const float* const gb[NF], float out[NF][3], int* status)
{
    if (f.multi_tframe != 0 || !interp_filtered<NF>(f, x, y, z, g, out)) {
        if (INL) interp_exact_inline<NF>(f, x, y, z, t, g, ga, gb, out, status);
        else interp_exact<NF>(f, x, y, z, t, g, ga, gb, out, status);
    }
}

// ---------------------------------------------------------------- WLCS
// transform / reverse_tran, src/wlcs.c:871-903
__device__ __forceinline__ void wl_transform(double& ax, double& ay, double& az, double c1,
                                             double s1, double c2, double s2)
{
    double ax1 = c2 * ax + s2 * ay;
    double ay1 = -s2 * ax + c2 * ay;
    double az1 = az;
    ax = c1 * ax1 - s1 * az1;
    ay = ay1;
    az = s1 * ax1 + c1 * az1;
}

__device__ __forceinline__ void wl_reverse(double& ax, double& ay, double& az, double c1,
                                           double s1, double c2, double s2)
{
    double ax1 = c1 * ax + s1 * az;
    double ay1 = ay;
    double az1 = -s1 * ax + c1 * az;
    ax = c2 * ax1 - s2 * ay1;
    ay = s2 * ax1 + c2 * ay1;
    az = az1;
}

// ellint, src/wlcs.c:460-809 (Fukushima 2009), coefficient tables recomputed
// from the mathematics (gen_ellint_coeffs.py)
// The division and square root of the loop's field as calls and its series
// rolled (TP_SOFT_CALLS), or all inline.  The adaptive stepper, whose warps sit
// at different points of a long loop body, calls them: inlined it waited for
// code 38 % of the time (65,536 particles: 433 -> 389 ms).  The fixed-step
// kernels, whose warps run in step, are 3 % faster inline.
#ifdef TP_SOFT_CALLS
constexpr int kEllUnroll = 4;
static __device__ __noinline__ double soft_div(double a, double b) { return sd::div(a, b); }
static __device__ __noinline__ double soft_sqrt(double x) { return sd::sqrt_rn(x); }
#else
constexpr int kEllUnroll = 20;
__device__ __forceinline__ double soft_div(double a, double b) { return sd::div(a, b); }
__device__ __forceinline__ double soft_sqrt(double x) { return sd::sqrt_rn(x); }
#endif

__device__ __forceinline__ void ellint64(const DevField& f, double k, int corrected, double& elle, double& ellf)
{
    double m = k * k;
    int i;
    elle = 0.0;
    ellf = 0.0;
    // (with contraction on, which product the compiler fuses into m - m0 below
    // depends on the instructions that read m: the adaptive stepper, whose step
    // counts follow the last bit, keeps the FP64 quotient)
#ifdef TP_ELL_FP64_QUOTIENT
    if (m < 0.8) i = (int)(m / 0.1);
#else
    if (m < 0.8) i = (int)sd::div(m, f.d_tenth);
#endif
    else if (m >= 0.8 && m < 0.85) i = 8;
    else if (m >= 0.85 && m < 0.9) i = 9;
    else i = 10;
    if (i >= 0 && i <= 9) {
        // every lane runs the longest series of the table: past an interval's
        // own length its coefficients are zero and add +0 exactly, so the
        // sums are those of the interval's own length while the lanes of a
        // warp, whatever their intervals, take the same loop
        double m1 = m - __ldg(&tp_ell_m0[i]), powj = 1.0;
#pragma unroll kEllUnroll
        for (int j = 0; j < TP_ELL_NK_MAX; j++) {
            double kc = __ldg(&tp_ell_k[i][j]);
            if (!corrected && i == 9 && j == 19) kc = TP_ELL_K9_19_REF;
            ellf += kc * powj;
            if (j < TP_ELL_NE_MAX) elle += __ldg(&tp_ell_e[i][j]) * powj;
            powj *= m1;
        }
        return;
    }
    // the powers of the third series, in 0.95 - m, are those of the first up to
    // sign (the reference's first series runs in m - 0.95): one chain for both,
    // the sign on the coefficient's bits
    double ellf1 = 0.0, q1 = 0.0, hm = 0.0, powj = 1.0;
    const double m1 = corrected ? (0.95 - m) : (m - 0.95), mq = 1.0 - m;
    double powq = mq;
    const uint64_t flip = corrected ? 0ull : 0x8000000000000000ull;
#pragma unroll kEllUnroll
    for (int j = 0; j <= 10; j++) {
        const uint64_t h = (uint64_t)__double_as_longlong(__ldg(&tp_ell_h[j])) ^ (j & 1 ? flip : 0ull);
        ellf1 += __ldg(&tp_ell_k[0][j]) * powj;
        hm += __longlong_as_double((long long)h) * powj;
        powj *= m1;
    }
#pragma unroll kEllUnroll
    for (int j = 1; j <= 14; j++) {
        q1 += __ldg(&tp_ell_q[j]) * powq;
        powq *= mq;
    }
    ellf = -log(q1) * soft_div(ellf1, TP_PI);
    elle = soft_div(1.0, ellf1) * (TP_PI / 2.0 + ellf * hm);
}

// getWireB, src/wlcs.c:361-401
__device__ __forceinline__ void wl_wire_static(const wlcs& c, double x, double y, double z,
                                               double B[3])
{
    double xp = x - c.x_wr, yp = y - c.y_wr, zp = z - c.z_wr;
    wl_transform(xp, yp, zp, c.costheta_wr, c.sintheta_wr, c.cosphi_wr, c.sinphi_wr);
    double rho = sd::sqrt_rn(xp * xp + yp * yp);
    if (rho < 0.1) rho = 0.1;
    double cos_phi0 = sd::div(xp, rho), phi0;
    if (yp >= 0.0) phi0 = acos(cos_phi0);
    else phi0 = 2.0 * TP_PI - acos(cos_phi0);
    double bphi = sd::div(1.0 / 5.0 * (c.cur_wr * TP_I0), rho * TP_L0);
    double sn, cs;
    sd::sin_cos(phi0 + TP_PI / 2.0, sn, cs);
    B[0] = bphi * cs;
    B[1] = bphi * sn;
    B[2] = 0.0;
    wl_reverse(B[0], B[1], B[2], c.costheta_wr, c.sintheta_wr, c.cosphi_wr, c.sinphi_wr);
}

// getWire_Bessel, src/wlcs.c:281-355 (single-precision Bessel functions)
__device__ __forceinline__ void wl_wire_bessel(const wlcs& c, double x, double y, double z,
                                               double t, double B[3], double E[3])
{
    double xp = x - c.x_wr, yp = y - c.y_wr, zp = z - c.z_wr;
    double t1 = c.t0 + t, curI = c.cur_wr, omega = c.omega, phi1;
    wl_transform(xp, yp, zp, c.costheta_wr, c.sintheta_wr, c.cosphi_wr, c.sinphi_wr);
    double rho = sqrt(xp * xp + yp * yp);
    double x0 = omega * rho * TP_L0 / TP_C0;
    double bj0 = j0f((float)x0), bj1 = j1f((float)x0);
    double by0 = y0f((float)x0), by1 = y1f((float)x0);
    double const0 = (curI * TP_I0) / (5.0 * rho * TP_L0) * TP_PI / 2.0;
    double wireB = const0 * x0 * (-by1 * cos(omega * t1) + bj1 * sin(omega * t1));
    if (rho == 0.0) phi1 = TP_PI / 2.0;
    else if (yp >= 0.0) phi1 = acos(xp / rho) + TP_PI / 2.0;
    else phi1 = 2.0 * TP_PI - acos(xp / rho) + TP_PI / 2.0;
    B[0] = wireB * cos(phi1);
    B[1] = wireB * sin(phi1);
    B[2] = 0.0;
    wl_reverse(B[0], B[1], B[2], c.costheta_wr, c.sintheta_wr, c.cosphi_wr, c.sinphi_wr);
    double wireE = -const0 * x0 * (by0 * sin(omega * t1) + bj0 * cos(omega * t1));
    E[0] = 0.0; E[1] = 0.0; E[2] = wireE;
    wl_reverse(E[0], E[1], E[2], c.costheta_wr, c.sintheta_wr, c.cosphi_wr, c.sinphi_wr);
}

// getLoopB, src/wlcs.c:406-449 (NaN Bx, By on the loop axis, as there)
__device__ __forceinline__ void wl_loop(const DevField& f, const wlcs& c, const LoopPre& pre, int ell_corr, double x,
                                        double y, double z, double B[3])
{
    double xp = (x - c.x_lp) * TP_L0, yp = (y - c.y_lp) * TP_L0, zp = (z - c.z_lp) * TP_L0;
    const double al = pre.al, al2 = pre.al2, Irho = pre.Irho;
    if (!pre.flat) wl_transform(xp, yp, zp, c.cosbeta_lp, c.sinbeta_lp, c.cosalpha_lp, c.sinalpha_lp);
    double rho_xy = soft_sqrt(xp * xp + yp * yp);
    double r2 = rho_xy * rho_xy + zp * zp;
    double irho1 = soft_div(1.0, soft_sqrt((al + rho_xy) * (al + rho_xy) + zp * zp));
    double irho2 = soft_div(1.0, (al - rho_xy) * (al - rho_xy) + zp * zp);
    double k = soft_sqrt(pre.al4 * rho_xy) * irho1, elle, ellk;
#ifndef TP_SOFT_CALLS
    // (the adaptive stepper, whose step counts follow the last bit, keeps the
    // FP64 series; its calls are those of this macro)
    if (!ellfx::integrals(f.ell, k * k, ell_corr, elle, ellk))
#endif
        ellint64(f, k, ell_corr, elle, ellk);
    double Brho = soft_div(Irho * zp * irho1 * (-ellk + (al2 + r2) * elle * irho2), rho_xy);
    if (rho_xy == 0.0) Brho = 0.0;
    double Bz = Irho * irho1 * (ellk - (r2 - al2) * elle * irho2);
    if (ell_corr && rho_xy == 0.0) {
        B[0] = 0.0; B[1] = 0.0;
    } else {
        Brho = soft_div(Brho, rho_xy);
        B[0] = __dmul_rn(Brho, xp);
        B[1] = __dmul_rn(Brho, yp);
    }
    B[2] = Bz;
    // (a component that is not finite, as on the axis, spreads through the rotation)
    const uint32_t e0 = (uint32_t)__double2hiint(B[0]) & 0x7ff00000u, e1 = (uint32_t)__double2hiint(B[1]) & 0x7ff00000u;
    if (!pre.flat || e0 == 0x7ff00000u || e1 == 0x7ff00000u) wl_reverse(B[0], B[1], B[2], c.cosbeta_lp, c.sinbeta_lp, c.cosalpha_lp, c.sinalpha_lp);
}

// ---------------------------------------------------------------- mode sum
// Exact phase in 64-bit fixed point: u = (x - min)/L per axis, U = frac(u)*2^64.
__device__ __forceinline__ uint64_t fixed_frac64(double u)
{
    double fr = u - floor(u);
    return __double2ull_rz(fr * 18446744073709551616.0);
}

// The six sums in fixed point (modesum_fx.cuh) as doubles.
__device__ __forceinline__ void mode_sum_fixed(const DevField& f, const int4* tab, const uint64_t u[3], double e[6])
{
    int64_t s[6];
    fx::mode_sum<fx::kChunk>(f.fxm, f.nfx, tab, u, s);
#pragma unroll
    for (int k = 0; k < 6; k++) e[k] = (double)s[k] * f.fxs[k];
}

// get_emf, src/emfields.c:32-60, specialised per system type (0..5).  TAB: the
// cosine table of the mode sum lies at the start of the block's dynamic shared
// memory, else it is read from global memory.
template <int SYS, bool TAB = false, bool INL = false>
__device__ __forceinline__ void emf64(const DevField& f, double x, double y, double z, double t,
                                      double e[6], int* status)
{
    e[0] = 0.0; e[1] = 0.0; e[2] = 0.0; e[3] = 0.0; e[4] = 0.0; e[5] = 0.0;
    if (SYS == TP_SYS_TEST) {
        e[2] = 1.0E0;  // getemf_test, src/emfields.c:210-218
    } else if (SYS == TP_SYS_FORCEFREE) {
        // getb_ff / gete_ff, src/force_free.c:78-86,138-150
        double l = f.lambda0;
        double sx, cx, sy, cy, sz, cz;
        sd::sin_cos(l * x, sx, cx);
        sd::sin_cos(l * y, sy, cy);
        sd::sin_cos(l * z, sz, cz);
        double bx = f.ffA * sz + f.ffC * cy;
        double by = f.ffB * sx + f.ffA * cz;
        double bz = f.ffC * sy + f.ffB * cx;
        bx *= f.B0;
        by *= f.B0;
        bz *= f.B0;
        e[0] = bx; e[1] = by; e[2] = bz;
        if (f.vc_d || f.va_d) {
            Tri64 r;
            trilinear64(f, x, y, z, t, r);
            double v[3];
            interp_d3(f, r, f.vc_d, f.va_d, f.vb_d, v, status);
            e[3] = by * v[2] - bz * v[1];
            e[4] = bz * v[0] - bx * v[2];
            e[5] = bx * v[1] - by * v[0];
        }
    } else if (SYS == TP_SYS_WLCS) {
        // getemf_wlcs, src/wlcs.c:814-865
        double Bx = 0.0, By = 0.0, Bz = 0.0, Ex = 0.0, Ey = 0.0, Ez = 0.0;
        for (int i = 0; i < f.nwlcs; i++) {
            double B[3], E[3];
            wlcs c = f.cfg[i];
            if (f.iBessel == 0) {
                // A wire without current adds exact zeros (its B is the
                // current times finite factors, the radius clamped at 0.1),
                // which leave the sums bit for bit as they are: skip its
                // square root, arc cosine, sine and cosine.
                if (c.cur_wr != 0.0) {
                    wl_wire_static(c, x, y, z, B);
                    Bx += B[0]; By += B[1]; Bz += B[2];
                }
            } else {
                wl_wire_bessel(c, x, y, z, t, B, E);
                Bx += B[0]; Ex += E[0];
                By += B[1]; Ey += E[1];
                Bz += B[2]; Ez += E[2];
            }
            wl_loop(f, c, f.pre[i], f.ellint_corrected, x, y, z, B);
            Bx += B[0]; By += B[1]; Bz += B[2];
        }
        e[0] = Bx; e[1] = By; e[2] = Bz + 0.0;
        e[3] = Ex; e[4] = Ey; e[5] = Ez;
    } else if (SYS == TP_SYS_MHD) {
        // getemf_mhd_test_particle, src/emfields.c:107-120
        const float *g[2] = {f.vc_f, f.bc_f}, *ga[2] = {f.va_f, f.ba_f}, *gb[2] = {f.vb_f, f.bb_f};
        float vb[2][3];
        interp_grids<2, INL>(f, x, y, z, t, g, ga, gb, vb, status);
        const float *v = vb[0], *b = vb[1];
        e[0] = b[0]; e[1] = b[1]; e[2] = b[2];
        e[3] = e[1] * v[2] - e[2] * v[1];
        e[4] = e[2] * v[0] - e[0] * v[2];
        e[5] = e[0] * v[1] - e[1] * v[0];
    } else if (SYS == TP_SYS_PIC) {
        // getemf_pic_test_particle, src/emfields.c:153-166; the reference
        // computes the same corners and weights twice, once is enough
        const float *g[2] = {f.ec_f, f.bc_f}, *ga[2] = {f.ea_f, f.ba_f}, *gb[2] = {f.eb_f, f.bb_f};
        float eb[2][3];
        interp_grids<2, INL>(f, x, y, z, t, g, ga, gb, eb, status);
        const float *ev = eb[0], *b = eb[1];
        e[3] = ev[0]; e[4] = ev[1]; e[5] = ev[2];
        e[0] = b[0]; e[1] = b[1]; e[2] = b[2];
    } else if (SYS == TP_SYS_MODESUM) {
        uint64_t ux = fixed_frac64((x - f.xmin) / (f.xmax - f.xmin));
        uint64_t uy = fixed_frac64((y - f.ymin) / (f.ymax - f.ymin));
        uint64_t uz = fixed_frac64((z - f.zmin) / (f.zmax - f.zmin));
        if (f.fxm) {
            extern __shared__ int4 s_ctab[];
            const uint64_t u[3] = {ux, uy, uz};
            mode_sum_fixed(f, TAB ? s_ctab : f.ctab, u, e);
            e[2] = f.B0 + e[2];
            return;
        }
        double b0 = 0.0, b1 = 0.0, b2 = 0.0, e0 = 0.0, e1 = 0.0, e2 = 0.0;
        for (int m = 0; m < f.nmodes; m++) {
            const tp_mode& md = f.modes[m];
            // md.pad holds the 32-bit fixed-point phase offset (host-filled)
            uint64_t ph = (uint64_t)(int64_t)md.n[0] * ux + (uint64_t)(int64_t)md.n[1] * uy +
                          (uint64_t)(int64_t)md.n[2] * uz +
                          ((uint64_t)(uint32_t)md.pad << 32);
            double th = (double)(int64_t)ph * (2.0 * TP_PI / 18446744073709551616.0);
            double c = cos(th);
            b0 += md.amp_b[0] * c; b1 += md.amp_b[1] * c; b2 += md.amp_b[2] * c;
            e0 += md.amp_e[0] * c; e1 += md.amp_e[1] * c; e2 += md.amp_e[2] * c;
        }
        e[0] = b0; e[1] = b1; e[2] = f.B0 + b2;
        e[3] = e0; e[4] = e1; e[5] = e2;
    }
}

// Same, dispatched at run time (batch utilities; the tracking kernels are
// instantiated per system type).
__device__ __forceinline__ void emf64_dispatch(const DevField& f, double x, double y, double z,
                                               double t, double e[6], int* status)
{
    switch (f.system_type) {
    case TP_SYS_TEST: emf64<TP_SYS_TEST>(f, x, y, z, t, e, status); break;
    case TP_SYS_WLCS: emf64<TP_SYS_WLCS>(f, x, y, z, t, e, status); break;
    case TP_SYS_FORCEFREE: emf64<TP_SYS_FORCEFREE>(f, x, y, z, t, e, status); break;
    case TP_SYS_MHD: emf64<TP_SYS_MHD>(f, x, y, z, t, e, status); break;
    case TP_SYS_PIC: emf64<TP_SYS_PIC>(f, x, y, z, t, e, status); break;
    case TP_SYS_MODESUM: emf64<TP_SYS_MODESUM>(f, x, y, z, t, e, status); break;
    default:
        e[0] = e[1] = e[2] = e[3] = e[4] = e[5] = 0.0;
        break;
    }
}

}  // namespace tp
