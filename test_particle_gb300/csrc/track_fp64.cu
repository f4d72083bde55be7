// track_fp64.cu -- FP64 tracking path: the Wirz push, boundary conditions,
// energy binning and diffusion coefficients in the reference's arithmetic,
// and the persistent fixed-step tracking kernel with fused diagnostics.
//
// Built twice: with -fmad=false as the parity path (TP_FP64_NS = fp64) and
// with -fmad=true as the fast FP64 path (TP_FP64_NS = fp64fast, -DTP_FAST).
#include <algorithm>

#include "fields_fp64.cuh"
#include "tp_kernels.h"

#ifndef TP_FP64_NS
#define TP_FP64_NS fp64
#endif

namespace tp {
namespace TP_FP64_NS {

struct P64 {
    double x, y, z, ux, uy, uz, t, xs, ys, zs;
};

// tracking_wirz, src/tracking.c:749-892 (c0_norm = 1).  Both field evaluations
// of a push, at its start and at its midpoint, are followed by the same work
// (the frame about B, the gyration angle, its sine and cosine): one loop body
// run twice, in the reference's operations and order.  Inlined twice, the body
// spills the instruction cache.
template <int SYS, bool TAB = false>
__device__ __forceinline__ void wirz(const DevField& f, P64& p, double dt, int* status)
{
    const double cm = f.charge_mass;
    const double dth = dt * 0.5;
    double e[6];
    double gama = 1.0, igama = 1.0, vm0 = 0.0, vm1 = 0.0, vm2 = 0.0;
    double iBtot, h0, h1, h2, vdothp, vperp, hp0, hp1, hp2, hr0, hr1, hr2, sind, cosd;
    double px = p.x, py = p.y, pz = p.z;
#pragma unroll 1
    for (int half = 0;; half++) {
        emf64<SYS, TAB>(f, px, py, pz, half ? p.t + dth : p.t, e, status);
        const double Btot = sd::sqrt_rn(e[0] * e[0] + e[1] * e[1] + e[2] * e[2]);
        iBtot = sd::div(1.0, Btot);
        if (half == 0) {
            const double dm0 = p.ux + cm * dth * e[3];
            const double dm1 = p.uy + cm * dth * e[4];
            const double dm2 = p.uz + cm * dth * e[5];
            gama = sd::sqrt_rn(1.0 + dm0 * dm0 + dm1 * dm1 + dm2 * dm2);
            igama = sd::div(1.0, gama);
            vm0 = dm0 * igama; vm1 = dm1 * igama; vm2 = dm2 * igama;
        }
        h0 = e[0] * iBtot; h1 = e[1] * iBtot; h2 = e[2] * iBtot;
        vdothp = 0.0;
        vdothp += vm0 * h0;
        vdothp += vm1 * h1;
        vdothp += vm2 * h2;
        const double q0 = vm0 - vdothp * h0, q1 = vm1 - vdothp * h1, q2 = vm2 - vdothp * h2;
        vperp = sd::sqrt_rn(q0 * q0 + q1 * q1 + q2 * q2);
        const sd::Divisor d_vperp = sd::divisor(vperp);
        hp0 = sd::div(q0, d_vperp);
        hp1 = sd::div(q1, d_vperp);
        hp2 = sd::div(q2, d_vperp);
        hr0 = h1 * hp2 - h2 * hp1;
        hr1 = h2 * hp0 - h0 * hp2;
        hr2 = h0 * hp1 - h1 * hp0;
        const double omegac = cm * Btot * igama;
        const double dtheta = omegac * dt;
        const double ang = half ? dtheta : dtheta * 0.5;
        if (SYS == TP_SYS_MHD || SYS == TP_SYS_PIC) {
            // the float grids' roundings turn a last-place difference of the
            // orbit into one of 2^-24 of a field: these systems keep CUDA's
            sind = sin(ang);
            cosd = cos(ang);
        } else {
            sd::sin_cos(ang, sind, cosd);
        }
        if (half) break;
        const double gyroR = sd::div(vperp * gama * 1.0 * iBtot, f.d_cm);
        const double tmp1 = dth * vdothp * 1.0, tmp2 = gyroR * sind, tmp3 = -gyroR * (1.0 - cosd);
        px = p.x + h0 * tmp1 + hp0 * tmp2 + hr0 * tmp3;
        py = p.y + h1 * tmp1 + hp1 * tmp2 + hr1 * tmp3;
        pz = p.z + h2 * tmp1 + hp2 * tmp2 + hr2 * tmp3;
    }
    const double vp0 = h0 * vdothp + vperp * (cosd * hp0 - sind * hr0);
    const double vp1 = h1 * vdothp + vperp * (cosd * hp1 - sind * hr1);
    const double vp2 = h2 * vdothp + vperp * (cosd * hp2 - sind * hr2);
    double bm = 0.0;  // get_delta_vec, src/tracking.c:1066-1078
    bm += vp0 * vp0;
    bm += vp1 * vp1;
    bm += vp2 * vp2;
    const double g2 = sd::div(1.0, sd::sqrt_rn(1.0 - bm));
    p.ux = g2 * vp0 + cm * dth * e[3];
    p.uy = g2 * vp1 + cm * dth * e[4];
    p.uz = g2 * vp2 + cm * dth * e[5];
    vdothp = 0.0;
    vdothp += vp0 * h0;
    vdothp += vp1 * h1;
    vdothp += vp2 * h2;
    const double q0 = vp0 - vdothp * h0, q1 = vp1 - vdothp * h1, q2 = vp2 - vdothp * h2;
    vperp = sd::sqrt_rn(q0 * q0 + q1 * q1 + q2 * q2);
    const double gyroR = sd::div(vperp * gama * 1.0 * iBtot, f.d_cm);
    const double tmp1 = dt * vdothp * 1.0;
    const double tmp2 = gyroR * sind;
    const double tmp3 = -gyroR * (1.0 - cosd);
    p.x += h0 * tmp1 + hp0 * tmp2 + hr0 * tmp3;
    p.y += h1 * tmp1 + hp1 * tmp2 + hr1 * tmp3;
    p.z += h2 * tmp1 + hp2 * tmp2 + hr2 * tmp3;
    p.t += dt;
}

// particle_bc, src/tracking.c:1172-1221
__device__ __forceinline__ void particle_bc(const DevField& f, P64& p, int& iescape)
{
    double xdim = f.xmax - f.xmin, ydim = f.ymax - f.ymin, zdim = f.zmax - f.zmin;
    if (f.bc_flag == 0) {
        if (p.x > f.xmax) { p.x -= xdim; p.xs += xdim; }
        if (p.y > f.ymax) { p.y -= ydim; p.ys += ydim; }
        if (p.z > f.zmax) { p.z -= zdim; p.zs += zdim; }
        if (p.x < f.xmin) { p.x += xdim; p.xs -= xdim; }
        if (p.y < f.ymin) { p.y += ydim; p.ys -= ydim; }
        if (p.z < f.zmin) { p.z += zdim; p.zs -= zdim; }
    } else if (f.bc_flag == 1) {
        if ((p.x > f.xmax) || (p.y > f.ymax) || (p.z > f.zmax) || (p.x < f.xmin) ||
            (p.y < f.ymin) || (p.z < f.zmin))
            iescape = 1;
    } else if (f.bc_flag == 2) {
        iescape = 0;
    }
}

// ptl_energy_fixed binning, src/diagnostics.c:187-205, done exactly by
// comparing against thresholds the host derived from the reference formula:
// the bin is the number of thresholds <= e.  NaN, e <= 0 and e = +inf give
// bin 0 as the reference does on x86.
__device__ __forceinline__ int energy_bin(const double* thr, int nbins, double ux, double uy,
                                          double uz)
{
    double gama = sqrt(1.0 + ux * ux + uy * uy + uz * uz);
    double e = gama - 1.0;
    if (!(e < INFINITY)) return 0;
    int lo = 0, hi = nbins - 1;  // answer in [0, nbins-1]
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;  // is thr[mid-1] <= e ?
        if (__ldg(thr + mid - 1) <= e) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// calc_diff_coeff, src/diagnostics.c:659-705 (pow(v, 2) taken as v * v).
// Output order: drr, dxx, dyy, dzz, dpp, duu, daa, dee.
template <int SYS, bool TAB = false, bool INL = false>
__device__ __forceinline__ void calc_diff(const DevField& f, const P64& p0, const P64& p,
                                          double dt, double o[8], int* status)
{
    double t = p.t * 2 + dt;
    double a = p0.x - (p.x + p.xs), b = p0.y - (p.y + p.ys), c = p0.z - (p.z + p.zs);
    double dxx = a * a / t, dyy = b * b / t, dzz = c * c / t;
    double drr = dxx + dyy + dzz;
    double d0 = p0.ux - p.ux, d1 = p0.uy - p.uy, d2 = p0.uz - p.uz;
    double dpp = (d0 * d0 + d1 * d1 + d2 * d2) / t;
    double gamma = sqrt(1.0 + p.ux * p.ux + p.uy * p.uy + p.uz * p.uz);
    double gamma0 = sqrt(1.0 + p0.ux * p0.ux + p0.uy * p0.uy + p0.uz * p0.uz);
    double dg = gamma - gamma0;
    double dee = dg * dg / t;
    double e[6], e0[6];
    emf64<SYS, TAB, INL>(f, p.x, p.y, p.z, p.t, e, status);
    emf64<SYS, TAB, INL>(f, p0.x, p0.y, p0.z, p0.t, e0, status);
    double abs_b = sqrt(e[0] * e[0] + e[1] * e[1] + e[2] * e[2]);
    double abs_u = sqrt(p.ux * p.ux + p.uy * p.uy + p.uz * p.uz);
    double mu = (e[0] * p.ux + e[1] * p.uy + e[2] * p.uz) / (abs_b * abs_u);
    abs_b = sqrt(e0[0] * e0[0] + e0[1] * e0[1] + e0[2] * e0[2]);
    abs_u = sqrt(p0.ux * p0.ux + p0.uy * p0.uy + p0.uz * p0.uz);
    double mu0 = (e0[0] * p0.ux + e0[1] * p0.uy + e0[2] * p0.uz) / (abs_b * abs_u);
    double dmu = mu - mu0;
    double duu = dmu * dmu / t;
    double theta = acos(mu) * 180 / TP_PI;
    double theta0 = acos(mu0) * 180 / TP_PI;
    double dth = theta - theta0;
    double daa = dth * dth / t;
    o[0] = drr; o[1] = dxx; o[2] = dyy; o[3] = dzz;
    o[4] = dpp; o[5] = duu; o[6] = daa; o[7] = dee;
}

__device__ __forceinline__ void load(const TrackBufs& b, int i, P64& p)
{
    p.x = b.x[i]; p.y = b.y[i]; p.z = b.z[i];
    p.ux = b.ux[i]; p.uy = b.uy[i]; p.uz = b.uz[i];
    p.t = b.t[i]; p.xs = b.xs[i]; p.ys = b.ys[i]; p.zs = b.zs[i];
}

__device__ __forceinline__ void store(const TrackBufs& b, int i, const P64& p)
{
    b.x[i] = p.x; b.y[i] = p.y; b.z[i] = p.z;
    b.ux[i] = p.ux; b.uy[i] = p.uy; b.uz[i] = p.uz;
    b.t[i] = p.t; b.xs[i] = p.xs; b.ys[i] = p.ys; b.zs[i] = p.zs;
}

// Deterministic block sum of the eight per-particle diffusion values into this
// block's slice of the partial-sum scratch: warp tree, then warps in order.
__device__ __forceinline__ void block_diff_sum(const double sg[8], double* red, double* slot)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
#pragma unroll
    for (int c = 0; c < 8; c++) {
        double v = sg[c];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane == 0) red[warp * 8 + c] = v;
    }
    __syncthreads();
    if (threadIdx.x < 8) {
        double s = 0.0;
        for (int w = 0; w < nwarps; w++) s += red[w * 8 + threadIdx.x];
        slot[threadIdx.x] += s;
    }
    __syncthreads();
}

// Resident blocks per SM the kernel is compiled for (3: at most 168 registers,
// no spills).  Two blocks (up to 228 registers) left the gridded run of 131,072
// particles 8 % slower, four (128, 120-316 bytes of spills) 4 %.
// The mode sum: four blocks, with some 100 bytes of spills (kernel time of 10 steps,
// 512 modes, 65,536 particles 4.63 ms against 4.91 with three and none; 262,144
// 16.0 and 15.7; in between it depends on the last wave: 131,072 9.25 and 7.97).
constexpr int track_min_blocks(int sys) { return sys == TP_SYS_MODESUM ? 4 : 3; }

// Persistent fixed-step tracking, restating particle_tracking_multi_steps_openmp
// and _single_step_openmp (src/tracking.c:297-462): one thread owns one
// particle for all estep steps; blocks walk tiles of kBlock particles.  All
// threads of a block run the same step sequence, so the diagnostic steps
// (every einterval steps for the spectrum, every 100 for the diffusion sums)
// are block-uniform and reduce through shared memory.
template <int SYS>
__global__ void __launch_bounds__(kBlock, track_min_blocks(SYS)) track_kernel(DevField f, TrackBufs b, TrackParams q)
{
    __shared__ double red[(kBlock / 32) * 8];
    __shared__ unsigned int hist[kMaxSmemBins];
    constexpr bool kTab = SYS == TP_SYS_MODESUM;
    if (kTab && f.fxm) {  // the cosine table of the mode sum, once per block
        extern __shared__ int4 s_ctab[];
        for (int k = threadIdx.x; k <= fx::kTab; k += blockDim.x) s_ctab[k] = f.ctab[k];
        __syncthreads();
    }
    const bool smem_hist = q.nbins <= kMaxSmemBins;
    for (int tile = blockIdx.x; tile < q.ntiles; tile += gridDim.x) {
        const int slot = tile * kBlock + threadIdx.x;
        const bool active = slot < q.n;
        const int i = active && q.idx ? q.idx[slot] : slot;  // the particle of this lane
        P64 p = {}, p0 = {};
        int nst = 1;
        if (active) {
            load(b, i, p);
            p0.x = b.x0[i]; p0.y = b.y0[i]; p0.z = b.z0[i];
            p0.ux = b.ux0[i]; p0.uy = b.uy0[i]; p0.uz = b.uz0[i]; p0.t = b.t0[i];
            nst = b.nsteps_ptl[i];
        }
        int esc_pre = 0;
        if (active) particle_bc(f, p, esc_pre);
        int esc_after = esc_pre;
        int ntp = q.ntp0, tstep = 1 + q.row0;
        double sg[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (active && q.resumed && b.sg_carry) {
#pragma unroll
            for (int c = 0; c < 8; c++) sg[c] = b.sg_carry[(size_t)i * kSegCarry + c];
        }
        // (remain has two entries at least; a test of q.nsdc here costs the mode
        // sum 0.6 %, its registers being full)
        if (active && esc_pre && !q.resumed) atomicSub(&b.remain[1], 1);
        double* slot_base = b.dpart + (size_t)blockIdx.x * q.nsdc * 8;
        int npts = 1;
        long toff = 0;
        if (active && q.traj_every > 0) {
            npts = b.ntraj_points[i];
            toff = i > 0 ? (long)b.ntraj_accum[i - 1] : 0;
        }
        for (int j = q.sstep; j <= q.estep; j++) {
            sg[0] = 0.0; sg[4] = 0.0; sg[5] = 0.0;  // src/tracking.c:334-336
            if (active && (esc_pre == 0 || f.bc_flag == 0)) {
                wirz<SYS, kTab>(f, p, q.dt, b.status);
                particle_bc(f, p, esc_after);
                nst += 1;
                if (esc_after == 0 && j % kDiffInterval == 0)
                    calc_diff<SYS, kTab>(f, p0, p, q.dt, sg, b.status);
                if (q.traj_every > 0 && j % q.traj_every == 0) {
                    // trajectory point, src/tracking.c:440-447
                    long off = toff + npts;
                    if (off >= 0 && off < b.ntraj_total) {
                        double* r = b.ptl_time + 11 * off;
                        r[0] = p.x; r[1] = p.y; r[2] = p.z; r[3] = b.qm[i];
                        r[4] = p.ux; r[5] = p.uy; r[6] = p.uz; r[7] = p.t;
                        r[8] = p.xs; r[9] = p.ys; r[10] = p.zs;
                    } else {
                        atomicOr(b.status, ST_BAD_INDEX);
                    }
                    npts++;
                }
            }
            if (active && esc_pre == 0 && esc_after == 1 && f.bc_flag == 1 && ntp < q.nt_out)
                atomicAdd(&b.espect_esc[ntp * q.nbins +
                                        energy_bin(b.ebin_thr, q.nbins, p.ux, p.uy, p.uz)], 1u);
            if (j % q.einterval == 0) {  // block-uniform
                if (ntp < q.nt_out) {
                    bool take = active && esc_after == 0;
                    if (smem_hist) {
                        __syncthreads();
                        for (int k = threadIdx.x; k < q.nbins; k += blockDim.x) hist[k] = 0u;
                        __syncthreads();
                        if (take) atomicAdd(&hist[energy_bin(b.ebin_thr, q.nbins, p.ux, p.uy, p.uz)], 1u);
                        __syncthreads();
                        for (int k = threadIdx.x; k < q.nbins; k += blockDim.x)
                            if (hist[k]) atomicAdd(&b.espect[ntp * q.nbins + k], hist[k]);
                    } else if (take) {
                        atomicAdd(&b.espect[ntp * q.nbins +
                                            energy_bin(b.ebin_thr, q.nbins, p.ux, p.uy, p.uz)], 1u);
                    }
                }
                ntp++;
            }
            if (j % kDiffInterval == 0) {  // block-uniform
                block_diff_sum(sg, red, slot_base + (size_t)tstep * 8);
                tstep++;
            }
            if (active && esc_after && j % kDiffInterval == 0 && tstep < q.nsdc)
                atomicSub(&b.remain[tstep], 1);
            esc_pre = esc_after;
        }
        if (active) {
            // the index again from the list rather than held through the loop
            const int ie = q.idx ? q.idx[tile * kBlock + threadIdx.x] : tile * kBlock + threadIdx.x;
            store(b, ie, p);
            b.nsteps_ptl[ie] = nst;
            if (q.traj_every > 0) b.ntraj_points[ie] = npts;
            if (b.sg_carry) {
#pragma unroll
                for (int c = 0; c < 8; c++) b.sg_carry[(size_t)ie * kSegCarry + c] = sg[c];
            }
            if (b.esc_out) b.esc_out[ie] = esc_after;
        }
    }
}

// Fixed-order sum of the per-block partials: dsum[c * nsdc + s] (component-major).
// A block takes 32 outputs; each of its rows sums every kReduceRows-th tracking
// block, then the rows are added in order.
constexpr int kReduceRows = 16;
__global__ void __launch_bounds__(32 * kReduceRows) reduce_dpart_kernel(const double* dpart, int nblocks, int nsdc,
                                                                        double* dsum)
{
    __shared__ double part[kReduceRows][32];
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    const int k = blockIdx.x * 32 + lane;  // k = s * 8 + c
    double s = 0.0;
    if (k < nsdc * 8) {
#pragma unroll 4
        for (int b = row; b < nblocks; b += kReduceRows) s += dpart[(size_t)b * nsdc * 8 + k];
    }
    part[row][lane] = s;
    __syncthreads();
    if (row == 0 && k < nsdc * 8) {
        double t = 0.0;
#pragma unroll
        for (int r = 0; r < kReduceRows; r++) t += part[r][lane];
        dsum[(k & 7) * nsdc + (k >> 3)] = t;
    }
}

#include "track_small.cuh"

// ---------------------------------------------------------------- batch utilities
// Points and fields pass through shared memory, so that a block reads and writes
// whole lines: in host memory (read and written in place) the 48-byte rows of
// one thread each cost more than staged copies above some 100,000 points (256
// against 221 us a call of the ABC field).  In lines, calls of 64, 10,000 and
// 200,000 points take 17, 27 and 240 us; with staged copies 23, 52 and 289.
__global__ void __launch_bounds__(128) emf_batch_kernel(DevField f, int n, const double* xyzt, double* out, int* status)
{
    __shared__ double buf[128 * 6];
    const int first = blockIdx.x * 128, cnt = min(128, n - first), t = threadIdx.x;
    for (int k = t; k < 4 * cnt; k += 128) buf[k] = xyzt[4 * (size_t)first + k];
    __syncthreads();
    const int r = min(t, cnt - 1);
    const double x = buf[4 * r], y = buf[4 * r + 1], z = buf[4 * r + 2], w = buf[4 * r + 3];
    __syncthreads();
    double e[6];
    if (t < cnt) {
        emf64_dispatch(f, x, y, z, w, e, status);
        for (int k = 0; k < 6; k++) buf[6 * t + k] = e[k];
    }
    __syncthreads();
    for (int k = t; k < 6 * cnt; k += 128) out[6 * (size_t)first + k] = buf[k];
}

template <int SYS>
__global__ void wirz_steps_kernel(DevField f, int n, double* st, int nsteps, double dt,
                                  int* iescape, int* status)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double* r = st + (size_t)11 * i;  // particles record, include/particle_info.h:6-12
    P64 p = {r[0], r[1], r[2], r[4], r[5], r[6], r[7], r[8], r[9], r[10]};
    int esc = iescape ? iescape[i] : 0;
    for (int s = 0; s < nsteps; s++) {
        wirz<SYS>(f, p, dt, status);
        if (iescape) particle_bc(f, p, esc);  // no iescape: tracking_wirz alone
    }
    r[0] = p.x; r[1] = p.y; r[2] = p.z; r[4] = p.ux; r[5] = p.uy; r[6] = p.uz;
    r[7] = p.t; r[8] = p.xs; r[9] = p.ys; r[10] = p.zs;
    if (iescape) iescape[i] = esc;
}

__global__ void ebin_kernel(const double* thr, int nbins, int n, const double* st, int* bins)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* r = st + (size_t)11 * i;
    bins[i] = energy_bin(thr, nbins, r[4], r[5], r[6]);
}

template <int SYS>
__global__ void diffc_kernel(DevField f, int n, const double* st0, const double* st, double dt,
                             double* out, int* status)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* r = st + (size_t)11 * i;
    const double* r0 = st0 + (size_t)11 * i;
    P64 p = {r[0], r[1], r[2], r[4], r[5], r[6], r[7], r[8], r[9], r[10]};
    P64 p0 = {r0[0], r0[1], r0[2], r0[4], r0[5], r0[6], r0[7], r0[8], r0[9], r0[10]};
    double o[8];
    calc_diff<SYS, false, true>(f, p0, p, dt, o, status);
    for (int k = 0; k < 8; k++) out[8 * i + k] = o[k];
}

__global__ void trilinear_kernel(DevField f, int n, const double* xyzt, long* corners,
                                 double* weights)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Tri64 r;
    trilinear64(f, xyzt[4 * i], xyzt[4 * i + 1], xyzt[4 * i + 2], xyzt[4 * i + 3], r);
    for (int k = 0; k < 8; k++) {
        corners[8 * i + k] = r.c[k];
        weights[8 * i + k] = r.w[k];
    }
}

// particle_bc on a batch of particles records
__global__ void bc_kernel(DevField f, int n, double* st, int* iescape)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double* r = st + (size_t)11 * i;
    P64 p = {r[0], r[1], r[2], r[4], r[5], r[6], r[7], r[8], r[9], r[10]};
    int esc = iescape[i];
    particle_bc(f, p, esc);
    r[0] = p.x; r[1] = p.y; r[2] = p.z; r[8] = p.xs; r[9] = p.ys; r[10] = p.zs;
    iescape[i] = esc;
}

// get_{float,double}_{b,e,velocity}_at_point (src/magnetic_field.c:555-622,
// src/electric_field.c:370-437, src/velocity_field.c:555-622).  which:
// 0 B float, 1 E float, 2 v float, 3 B double, 4 E double, 5 v double.
__global__ void point_interp_kernel(DevField f, int which, int n, const double* xyzt,
                                    double* out, int* status)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Tri64 r;
    trilinear64(f, xyzt[4 * i], xyzt[4 * i + 1], xyzt[4 * i + 2], xyzt[4 * i + 3], r);
    if (which <= 2) {
        const float *c = which == 0 ? f.bc_f : which == 1 ? f.ec_f : f.vc_f;
        const float *a = which == 0 ? f.ba_f : which == 1 ? f.ea_f : f.va_f;
        const float *b = which == 0 ? f.bb_f : which == 1 ? f.eb_f : f.vb_f;
        float v[3] = {0.f, 0.f, 0.f};
        if ((f.multi_tframe == 0 && c) || (f.multi_tframe != 0 && a && b))
            interp_f3(f, r, c, a, b, v, status);
        else
            atomicOr(status, ST_BAD_INDEX);
        out[3 * i] = v[0]; out[3 * i + 1] = v[1]; out[3 * i + 2] = v[2];
    } else {
        const double *c = which == 3 ? f.bc_d : which == 4 ? f.ec_d : f.vc_d;
        const double *a = which == 3 ? f.ba_d : which == 4 ? f.ea_d : f.va_d;
        const double *b = which == 3 ? f.bb_d : which == 4 ? f.eb_d : f.vb_d;
        double v[3] = {0.0, 0.0, 0.0};
        if ((f.multi_tframe == 0 && c) || (f.multi_tframe != 0 && a && b))
            interp_d3(f, r, c, a, b, v, status);
        else
            atomicOr(status, ST_BAD_INDEX);
        out[3 * i] = v[0]; out[3 * i + 1] = v[1]; out[3 * i + 2] = v[2];
    }
}

// ---------------------------------------------------------------- Poincare map
// Field lines of the gridded B (get_magnetic_field, src/emfields.c:76-96:
// the float B grid for systems 3 and 4) traced with the fixed-step RK4 of
// next_location (src/poincare_map.c:243-290) on the unit vector of B, the
// stage points wrapped into the box (field_boundary, :296-321), and the
// crossings of the plane pos[face] = seed[face] recorded as the first point
// after a sign change (:158-181).  One thread per seed.
__device__ __forceinline__ void pm_boundary(const DevField& f, double& x, double& y, double& z)
{
    double xdim = f.xmax - f.xmin, ydim = f.ymax - f.ymin, zdim = f.zmax - f.zmin;
    if (x > f.xmax) x -= xdim;
    if (y > f.ymax) y -= ydim;
    if (z > f.zmax) z -= zdim;
    if (x < f.xmin) x += xdim;
    if (y < f.ymin) y += ydim;
    if (z < f.zmin) z += zdim;
}

__device__ __forceinline__ void pm_unit_b(const DevField& f, double x, double y, double z, double b[3],
                                          int* status)
{
    const float *g[1] = {f.bc_f}, *ga[1] = {f.ba_f}, *gb[1] = {f.bb_f};
    float v[1][3];
    interp_grids<1>(f, x, y, z, 0.0, g, ga, gb, v, status);
    double bx = v[0][0], by = v[0][1], bz = v[0][2];
    double ib = sd::div(1.0, sd::sqrt_rn(bx * bx + by * by + bz * bz));
    b[0] = bx * ib;
    b[1] = by * ib;
    b[2] = bz * ib;
}

// One RK4 step.  The four stages are one loop body (four inlined copies of the
// field evaluation do not fit the instruction cache: 6.5 of 13 cycles an
// instruction waited for code), the sum b1 + 2 b2 + 2 b3 + b4 taken in order.
__device__ __forceinline__ void pm_next(const DevField& f, double& px, double& py, double& pz, double h,
                                        int* status)
{
    pm_boundary(f, px, py, pz);
    double xt = px, yt = py, zt = pz, s0 = 0.0, s1 = 0.0, s2 = 0.0;
#pragma unroll 1
    for (int stage = 0; stage < 4; stage++) {
        double b[3];
        pm_unit_b(f, xt, yt, zt, b, status);
        if (stage == 0) {
            s0 = b[0]; s1 = b[1]; s2 = b[2];
        } else {
            const double w = stage < 3 ? 2.0 : 1.0;
            s0 = s0 + w * b[0];
            s1 = s1 + w * b[1];
            s2 = s2 + w * b[2];
        }
        if (stage == 3) break;
        const double hs = stage < 2 ? 0.5 * h : h;
        xt = px + hs * b[0];
        yt = py + hs * b[1];
        zt = pz + hs * b[2];
        pm_boundary(f, xt, yt, zt);
    }
    px += (h / 6) * s0;
    py += (h / 6) * s1;
    pz += (h / 6) * s2;
}

// outputs [n][ncross + 1] per coordinate; entries a seed does not reach keep
// the reference's fill value 2 * max of the axis
__global__ void poincare_kernel(DevField f, int n, const double* __restrict__ seeds, int face, double h,
                                double lmax, int ncross, double* xo, double* yo, double* zo, int* found,
                                int* status)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t row = (size_t)i * (ncross + 1);
    for (int k = 0; k <= ncross; k++) {
        xo[row + k] = f.xmax * 2;
        yo[row + k] = f.ymax * 2;
        zo[row + k] = f.zmax * 2;
    }
    double pos[3] = {seeds[3 * i], seeds[3 * i + 1], seeds[3 * i + 2]};
    const double init = pos[face];
    xo[row] = pos[0]; yo[row] = pos[1]; zo[row] = pos[2];
    // One loop over the steps of the whole line: a loop per crossing makes the
    // lanes of a warp wait for each other's next crossing (4,000 seeds, 4
    // crossings: 87.7 -> 14.1 ms).
    int icross = 1;
    double length = 0.0;
    bool more = icross <= ncross && length < lmax;  // at most lmax / h steps in all
    while (more) {
        const double pre = pos[face];
        pm_next(f, pos[0], pos[1], pos[2], h, status);
        const double cross = (pre - init) * (pos[face] - init);
        length += h;
        more = length < lmax;
        if (!(cross > 0) && more) {
            xo[row + icross] = pos[0];
            yo[row + icross] = pos[1];
            zo[row + icross] = pos[2];
            ++icross;
            more = icross <= ncross;
        }
    }
    found[i] = icross - 1;
}

// The same for few seeds: four lanes a seed, eight seeds a warp, one warp a
// block.  A seed's stages are a dependent chain whose FP64 instructions issue
// every 64 cycles whatever the number of active lanes; with a component a lane
// (lane 3 repeats component 0) a stage issues 14 of them instead of 41, the
// eight weights two a lane, exchanged as float pairs by shuffles.  Operations
// and order are those of poincare_kernel.  256^3 grid, 4 crossings, against
// that kernel: 1,024 seeds 13.8 -> 7.2 ms, 4,000 14.1 -> 7.4, 16,000 14.0 ->
// 12.9; 30,000 seeds 18.9 -> 26.2, so it stops at kPoincareSmall.  (16 blocks an SM
// let the compiler take 112 registers; by itself it took 96 and spilled, 2 % slower.)
constexpr int kPoincareSmall = 16384;
__device__ __forceinline__ double sgrp(double v, int k) { return __shfl_sync(0xffffffffu, v, (threadIdx.x & 28) | k); }
__device__ __forceinline__ float sgrp(float v, int k) { return __shfl_sync(0xffffffffu, v, (threadIdx.x & 28) | k); }
__device__ __forceinline__ int sgrp(int v, int k) { return __shfl_sync(0xffffffffu, v, (threadIdx.x & 28) | k); }

// Component c of B / |B| at the group's position; x is this lane's coordinate.
__device__ __forceinline__ double pm_unit_lane(const DevField& f, int c, double x, double lo, double hi,
                                               const sd::Divisor& d, int n, int* status)
{
    int i;
    double fr;
    bool ok = f.multi_tframe == 0 && cell64(x, lo, hi, d, n, i, fr);
    const unsigned in = __ballot_sync(0xffffffffu, ok) >> (threadIdx.x & 28);
    ok = (in & 7u) == 7u;
    const double dx = sgrp(fr, 0), dy = sgrp(fr, 1), dz = sgrp(fr, 2);
    const int ix = sgrp(i, 0), iy = sgrp(i, 1), iz = sgrp(i, 2);
    float v = 0.0f;
    bool bad = !ok;
    {
        const size_t sy = 3 * (size_t)f.nx, sz = sy * f.ny;
        const float* g = f.bc_f + (ok ? ((size_t)((size_t)iz * f.ny + iy) * f.nx + ix) * 3 + c : 0);
        const size_t off[8] = {0, sz, sy, 3, 3 + sy, 3 + sz, sy + sz, 3 + sy + sz};  // trilinear64's corner order
        float p[8];
#pragma unroll
        for (int k = 0; k < 8; k++) p[k] = ok ? __ldg(g + off[k]) : 0.0f;
        // lane j: the product of the x and y factors of edge j, times 1 - dz and times dz
        const int j = threadIdx.x & 3;
        const double a = (j & 1 ? dx : 1.0 - dx) * (j & 2 ? dy : 1.0 - dy);
        float ah, al, bh, bl;
        split_weight(a * (1.0 - dz), ah, al, bad);
        split_weight(a * dz, bh, bl, bad);
        // which lane holds each corner's weight, and whether it is the dz one
        // (the reference pairs x weights with z corners, src/interpolation.c:173-180)
        const bool corr = f.interp_corrected != 0;
        const int lane[8] = {0, corr ? 0 : 1, 2, corr ? 1 : 0, corr ? 3 : 2, 1, corr ? 2 : 3, 3};
        const bool top[8] = {false, corr, false, !corr, !corr, true, corr, true};
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float h0 = sgrp(ah, lane[k]), h1 = sgrp(bh, lane[k]), l0 = sgrp(al, lane[k]), l1 = sgrp(bl, lane[k]);
            add_term(v, p[k], top[k] ? h1 : h0, top[k] ? l1 : l0, bad);
        }
    }
    const unsigned any = __ballot_sync(0xffffffffu, bad) >> (threadIdx.x & 28);
    const double px = sgrp(x, 0), py = sgrp(x, 1), pz = sgrp(x, 2);
    if (any & 15u) {  // the whole group: not certain
        const float *g[1] = {f.bc_f}, *ga[1] = {f.ba_f}, *gb[1] = {f.bb_f};
        float w[1];
        interp_exact_lane<1>(f, px, py, pz, 0.0, g, ga, gb, c, w, status);
        v = w[0];
    }
    const double b = v, b2 = b * b;
    const double ib = sd::div(1.0, sd::sqrt_rn(sgrp(b2, 0) + sgrp(b2, 1) + sgrp(b2, 2)));
    return b * ib;
}

__global__ void __launch_bounds__(32, 16) poincare_small_kernel(DevField f, int n, const double* __restrict__ seeds,
                                                            int face, double h, double lmax, int ncross, double* xo,
                                                            double* yo, double* zo, int* found, int* status)
{
    const int i = blockIdx.x * 8 + (threadIdx.x >> 2), il = min(i, n - 1);
    const int c = (threadIdx.x & 3) == 3 ? 0 : threadIdx.x & 3;
    const bool writes = i < n && (threadIdx.x & 3) < 3;
    const double lo = c == 0 ? f.xmin : c == 1 ? f.ymin : f.zmin, hi = c == 0 ? f.xmax : c == 1 ? f.ymax : f.zmax;
    const double dim = hi - lo;
    const sd::Divisor d = c == 0 ? f.d_gdx : c == 1 ? f.d_gdy : f.d_gdz;
    const int nn = c == 0 ? f.nx : c == 1 ? f.ny : f.nz;
    double* out = (c == 0 ? xo : c == 1 ? yo : zo) + (size_t)il * (ncross + 1);
    double x = seeds[3 * il + c];
    if (writes) {
        out[0] = x;
        for (int k = 1; k <= ncross; k++) out[k] = hi * 2;
    }
    auto wrap = [&](double v) {
        if (v > hi) v -= dim;
        if (v < lo) v += dim;
        return v;
    };
    const double init = sgrp(x, face);
    int icross = 1;
    double length = 0.0;
    bool done = !(icross <= ncross && length < lmax);
    while (__any_sync(0xffffffffu, !done)) {
        const double pre = sgrp(x, face);
        const double x0 = wrap(x);
        double xt = x0, s = 0.0;
#pragma unroll 1
        for (int stage = 0; stage < 4; stage++) {
            const double b = pm_unit_lane(f, c, xt, lo, hi, d, nn, done ? nullptr : status);
            if (stage == 0) s = b;
            else s = s + (stage < 3 ? 2.0 : 1.0) * b;
            if (stage == 3) break;
            xt = wrap(x0 + (stage < 2 ? 0.5 * h : h) * b);
        }
        const double xn = x0 + (h / 6) * s;
        const double cross = (pre - init) * (sgrp(xn, face) - init);
        if (!done) {
            x = xn;
            length += h;
            done = !(length < lmax);
            if (!(cross > 0) && !done) {
                if (writes) out[icross] = x;
                ++icross;
                done = icross > ncross;
            }
        }
    }
    if (writes && c == 0) found[i] = icross - 1;
}

cudaError_t launch_poincare(const DevField& f, int n, const double* seeds, int face, double h, double lmax,
                            int ncross, double* xo, double* yo, double* zo, int* found, int* status,
                            cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    if (n <= kPoincareSmall) {
        poincare_small_kernel<<<(n + 7) / 8, 32, 0, s>>>(f, n, seeds, face, h, lmax, ncross, xo, yo, zo, found, status);
        return cudaGetLastError();
    }
    poincare_kernel<<<(n + 127) / 128, 128, 0, s>>>(f, n, seeds, face, h, lmax, ncross, xo, yo, zo, found,
                                                    status);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- host launchers
cudaError_t launch_bc(const DevField& f, int n, double* st, int* iescape, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    bc_kernel<<<(n + 127) / 128, 128, 0, s>>>(f, n, st, iescape);
    return cudaGetLastError();
}

cudaError_t launch_point_interp(const DevField& f, int which, int n, const double* xyzt,
                                double* out, int* status, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    point_interp_kernel<<<(n + 127) / 128, 128, 0, s>>>(f, which, n, xyzt, out, status);
    return cudaGetLastError();
}

// dynamic shared memory of track_kernel: the mode sum's cosine table
static constexpr size_t track_smem(int sys) { return sys == TP_SYS_MODESUM ? sizeof(int4) * (fx::kTab + 1) : 0; }

template <int SYS>
static cudaError_t launch_track_sys(const DevField& f, const TrackBufs& b, const TrackParams& q,
                                    int grid, cudaStream_t s)
{
    track_kernel<SYS><<<grid, kBlock, track_smem(SYS), s>>>(f, b, q);
    return cudaGetLastError();
}

cudaError_t launch_track(const DevField& f, const TrackBufs& b, const TrackParams& q, int grid,
                         cudaStream_t s)
{
    switch (f.system_type) {
    case TP_SYS_TEST: return launch_track_sys<TP_SYS_TEST>(f, b, q, grid, s);
    case TP_SYS_WLCS: return launch_track_sys<TP_SYS_WLCS>(f, b, q, grid, s);
    case TP_SYS_FORCEFREE: return launch_track_sys<TP_SYS_FORCEFREE>(f, b, q, grid, s);
    case TP_SYS_MHD: return launch_track_sys<TP_SYS_MHD>(f, b, q, grid, s);
    case TP_SYS_PIC: return launch_track_sys<TP_SYS_PIC>(f, b, q, grid, s);
    case TP_SYS_MODESUM: return launch_track_sys<TP_SYS_MODESUM>(f, b, q, grid, s);
    default: return cudaErrorInvalidValue;
    }
}

int track_max_blocks_per_sm(int system_type)
{
    int nb = 0;
    cudaError_t e = cudaErrorInvalidValue;
    switch (system_type) {
    case TP_SYS_TEST: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, track_kernel<TP_SYS_TEST>, kBlock, 0); break;
    case TP_SYS_WLCS: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, track_kernel<TP_SYS_WLCS>, kBlock, 0); break;
    case TP_SYS_FORCEFREE: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, track_kernel<TP_SYS_FORCEFREE>, kBlock, 0); break;
    case TP_SYS_MHD: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, track_kernel<TP_SYS_MHD>, kBlock, 0); break;
    case TP_SYS_PIC: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, track_kernel<TP_SYS_PIC>, kBlock, 0); break;
    case TP_SYS_MODESUM: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, track_kernel<TP_SYS_MODESUM>, kBlock, track_smem(TP_SYS_MODESUM)); break;
    default: break;
    }
    return e == cudaSuccess ? nb : 0;
}

cudaError_t launch_reduce_dpart(const double* dpart, int nblocks, int nsdc, double* dsum,
                                cudaStream_t s)
{
    int n = nsdc * 8;
    reduce_dpart_kernel<<<(n + 31) / 32, 32 * kReduceRows, 0, s>>>(dpart, nblocks, nsdc, dsum);
    return cudaGetLastError();
}

cudaError_t launch_emf_batch(const DevField& f, int n, const double* xyzt, double* out,
                             int* status, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    emf_batch_kernel<<<(n + 127) / 128, 128, 0, s>>>(f, n, xyzt, out, status);
    return cudaGetLastError();
}

cudaError_t launch_wirz_steps(const DevField& f, int n, double* st, int nsteps, double dt,
                              int* iescape, int* status, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    int g = (n + 127) / 128;
    switch (f.system_type) {
    case TP_SYS_TEST: wirz_steps_kernel<TP_SYS_TEST><<<g, 128, 0, s>>>(f, n, st, nsteps, dt, iescape, status); break;
    case TP_SYS_WLCS: wirz_steps_kernel<TP_SYS_WLCS><<<g, 128, 0, s>>>(f, n, st, nsteps, dt, iescape, status); break;
    case TP_SYS_FORCEFREE: wirz_steps_kernel<TP_SYS_FORCEFREE><<<g, 128, 0, s>>>(f, n, st, nsteps, dt, iescape, status); break;
    case TP_SYS_MHD: wirz_steps_kernel<TP_SYS_MHD><<<g, 128, 0, s>>>(f, n, st, nsteps, dt, iescape, status); break;
    case TP_SYS_PIC: wirz_steps_kernel<TP_SYS_PIC><<<g, 128, 0, s>>>(f, n, st, nsteps, dt, iescape, status); break;
    case TP_SYS_MODESUM: wirz_steps_kernel<TP_SYS_MODESUM><<<g, 128, 0, s>>>(f, n, st, nsteps, dt, iescape, status); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_ebins(const double* thr, int nbins, int n, const double* st, int* bins,
                         cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    ebin_kernel<<<(n + 127) / 128, 128, 0, s>>>(thr, nbins, n, st, bins);
    return cudaGetLastError();
}

cudaError_t launch_diffc(const DevField& f, int n, const double* st0, const double* st,
                         double dt, double* out, int* status, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    int g = (n + 127) / 128;
    switch (f.system_type) {
    case TP_SYS_TEST: diffc_kernel<TP_SYS_TEST><<<g, 128, 0, s>>>(f, n, st0, st, dt, out, status); break;
    case TP_SYS_WLCS: diffc_kernel<TP_SYS_WLCS><<<g, 128, 0, s>>>(f, n, st0, st, dt, out, status); break;
    case TP_SYS_FORCEFREE: diffc_kernel<TP_SYS_FORCEFREE><<<g, 128, 0, s>>>(f, n, st0, st, dt, out, status); break;
    case TP_SYS_MHD: diffc_kernel<TP_SYS_MHD><<<g, 128, 0, s>>>(f, n, st0, st, dt, out, status); break;
    case TP_SYS_PIC: diffc_kernel<TP_SYS_PIC><<<g, 128, 0, s>>>(f, n, st0, st, dt, out, status); break;
    case TP_SYS_MODESUM: diffc_kernel<TP_SYS_MODESUM><<<g, 128, 0, s>>>(f, n, st0, st, dt, out, status); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_trilinear(const DevField& f, int n, const double* xyzt, long* corners,
                             double* weights, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    trilinear_kernel<<<(n + 127) / 128, 128, 0, s>>>(f, n, xyzt, corners, weights);
    return cudaGetLastError();
}

}  // namespace TP_FP64_NS
}  // namespace tp
