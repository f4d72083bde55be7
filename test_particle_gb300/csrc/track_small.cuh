// track_small.cuh -- the FP64 tracking kernel for runs too small to fill the
// machine (included by track_fp64.cu, in its namespace).
//
// Below about ten thousand particles the one-thread-a-particle kernel leaves
// most sub-partitions empty while each of its warps waits for its own FP64
// pipe, 64 cycles an instruction whatever the number of active lanes.  Here a
// block of 128 threads takes 32 particles, four lanes each: lane c of a group
// holds component c of position and momentum (lane 3 repeats component 0), so
// the vector operations of the push issue once for three components, and
// scalars come from the group by shuffles.  The fields split likewise: one
// sine and cosine a lane (force-free), a quarter of the modes a lane (mode
// sum), and one wire or loop a warp for the block's 32 particles (current
// systems), through shared memory; gridded fields are evaluated by every lane
// where the filtered sums hold and by component where they do not.
// Every particle's operations and their order are those of track_kernel.
// Whole runs: 256 particles x 200 steps, ABC, 3.11 -> 1.79 ms; 4,096 x 200, two
// wires and loops, 23.2 -> 9.2 ms (4.5 with the integrals of ellint_fx.cuh).
#pragma once

constexpr int kSmallTile = 32;      // particles a block
constexpr int kSmallSystems = 8;    // current systems whose parts fit in shared memory

struct SmallShared {
    double x[4][kSmallTile];                        // position and time of the block's particles
    double part[2 * kSmallSystems][6][kSmallTile];  // B (and a wire's E) of each wire and loop
};

__device__ __forceinline__ double grp(double v, int k)
{
    return __shfl_sync(0xffffffffu, v, (threadIdx.x & 28) | k);
}

__device__ __forceinline__ long long grp(long long v, int k)
{
    return __shfl_sync(0xffffffffu, v, (threadIdx.x & 28) | k);
}

// a0 + a1 + a2 of the group's lanes, after s
__device__ __forceinline__ double grp_add(double s, double a)
{
    s += grp(a, 0);
    s += grp(a, 1);
    s += grp(a, 2);
    return s;
}

__device__ __forceinline__ double grp_sum(double a) { return grp(a, 0) + grp(a, 1) + grp(a, 2); }

// Component c of B and E at the group's position (x: this lane's coordinate).
template <int SYS>
__device__ __forceinline__ void small_field(const DevField& f, int c, double x, double t, double& B, double& E,
                                            SmallShared& sh, int* status)
{
    B = 0.0;
    E = 0.0;
    if (SYS == TP_SYS_TEST) {
        B = c == 2 ? 1.0E0 : 0.0;
    } else if (SYS == TP_SYS_FORCEFREE && !(f.vc_d || f.va_d)) {
        // B_c takes the sine of the coordinate before its own and the cosine
        // of the one after it, in cyclic order (src/force_free.c:138-150)
        double s, co;
        sd::sin_cos(f.lambda0 * x, s, co);
        const int pre = c == 0 ? 2 : c - 1, post = c == 2 ? 0 : c + 1;
        const double sp = grp(s, pre), cp = grp(co, post);
        const double as = c == 0 ? f.ffA : c == 1 ? f.ffB : f.ffC, ac = c == 0 ? f.ffC : c == 1 ? f.ffA : f.ffB;
        B = as * sp + ac * cp;
        B *= f.B0;
    } else if (SYS == TP_SYS_MODESUM) {
        extern __shared__ int4 s_ctab[];
        const uint64_t u[3] = {fixed_frac64((grp(x, 0) - f.xmin) / (f.xmax - f.xmin)),
                               fixed_frac64((grp(x, 1) - f.ymin) / (f.ymax - f.ymin)),
                               fixed_frac64((grp(x, 2) - f.zmin) / (f.zmax - f.zmin))};
        // every fourth chunk of modes; the integer sums of the chunks add in any order
        int64_t s[6];
        fx::mode_sum<4>(f.fxm, f.nfx, s_ctab, u, s, threadIdx.x & 3, 4);
        int64_t b = 0, e = 0;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            int64_t tb = 0, te = 0;
#pragma unroll
            for (int l = 0; l < 4; l++) {
                tb += grp((long long)s[k], l);
                te += grp((long long)s[3 + k], l);
            }
            if (c == k) {
                b = tb;
                e = te;
            }
        }
        const double sb = c == 0 ? f.fxs[0] : c == 1 ? f.fxs[1] : f.fxs[2];
        const double se = c == 0 ? f.fxs[3] : c == 1 ? f.fxs[4] : f.fxs[5];
        B = (double)b * sb;
        E = (double)e * se;
        if (c == 2) B = f.B0 + B;
    } else if (SYS == TP_SYS_WLCS) {
        // one wire or loop a warp and pass, for all particles of the block
        const int q = threadIdx.x >> 2, lane = threadIdx.x & 31;
        if ((threadIdx.x & 3) < 3) sh.x[c][q] = x;
        else sh.x[3][q] = t;
        __syncthreads();
        const double px = sh.x[0][lane], py = sh.x[1][lane], pz = sh.x[2][lane], pt = sh.x[3][lane];
        for (int p = threadIdx.x >> 5; p < 2 * f.nwlcs; p += 4) {
            const wlcs w = f.cfg[p >> 1];
            double b[3] = {0.0, 0.0, 0.0}, e[3] = {0.0, 0.0, 0.0};
            if (p & 1) wl_loop(f, w, f.pre[p >> 1], f.ellint_corrected, px, py, pz, b);
            else if (f.iBessel != 0) wl_wire_bessel(w, px, py, pz, pt, b, e);
            else if (w.cur_wr != 0.0) wl_wire_static(w, px, py, pz, b);
#pragma unroll
            for (int k = 0; k < 3; k++) {
                sh.part[p][k][lane] = b[k];
                sh.part[p][3 + k][lane] = e[k];
            }
        }
        __syncthreads();
        for (int p = 0; p < 2 * f.nwlcs; p++) {
            if (!(p & 1) && f.iBessel == 0 && !(f.cfg[p >> 1].cur_wr != 0.0)) continue;  // exact zeros, as in emf64
            B += sh.part[p][c][q];
            if (!(p & 1) && f.iBessel != 0) E += sh.part[p][3 + c][q];
        }
        if (c == 2) B = B + 0.0;
    } else if (SYS == TP_SYS_MHD || SYS == TP_SYS_PIC) {
        // every lane evaluates the whole grid sample where the filtered sums are
        // certain; where they are not, the reference's arithmetic on its own
        // component only (two time frames, 9,000 particles x 110 steps: 7.8 ms with
        // all components in every lane, 4.6 so, 5.5 with a lane a particle)
        const bool mhd = SYS == TP_SYS_MHD;
        const float *g[2] = {mhd ? f.vc_f : f.ec_f, f.bc_f}, *ga[2] = {mhd ? f.va_f : f.ea_f, f.ba_f},
                    *gb[2] = {mhd ? f.vb_f : f.eb_f, f.bb_f};
        const double px = grp(x, 0), py = grp(x, 1), pz = grp(x, 2);
        float all[2][3], own[2];
        if (f.multi_tframe == 0 && interp_filtered<2>(f, px, py, pz, g, all)) {
            own[0] = c == 0 ? all[0][0] : c == 1 ? all[0][1] : all[0][2];
            own[1] = c == 0 ? all[1][0] : c == 1 ? all[1][1] : all[1][2];
        } else {
            interp_exact_lane<2>(f, px, py, pz, t, g, ga, gb, c, own, status);
        }
        B = own[1];
        E = own[0];
        if (mhd) {  // E = B x v (src/emfields.c:107-120), the next two components of each
            const int c1 = c == 2 ? 0 : c + 1, c2 = c == 0 ? 2 : c - 1;
            const double v = own[0];
            E = grp(B, c1) * grp(v, c2) - grp(B, c2) * grp(v, c1);
        }
    } else {
        double e[6];
        emf64<SYS>(f, grp(x, 0), grp(x, 1), grp(x, 2), t, e, status);
        B = c == 0 ? e[0] : c == 1 ? e[1] : e[2];
        E = c == 0 ? e[3] : c == 1 ? e[4] : e[5];
    }
}

// wirz with one component a lane; x, u and t are advanced
template <int SYS>
__device__ __forceinline__ void small_wirz(const DevField& f, int c, double& x, double& u, double& t, double dt,
                                           SmallShared& sh, int* status)
{
    const double cm = f.charge_mass;
    const double dth = dt * 0.5;
    const int c1 = c == 2 ? 0 : c + 1, c2 = c == 0 ? 2 : c - 1;  // the next two components, cyclic
    double gama = 1.0, igama = 1.0, vm = 0.0;
    double iBtot, B, E, h, vdothp, vperp, hp, hr, sind, cosd;
    double px = x;
#pragma unroll 1
    for (int half = 0;; half++) {
        small_field<SYS>(f, c, px, half ? t + dth : t, B, E, sh, status);
        const double Btot = sd::sqrt_rn(grp_sum(B * B));
        iBtot = sd::div(1.0, Btot);
        if (half == 0) {
            const double dm = u + cm * dth * E;
            gama = sd::sqrt_rn(grp_add(1.0, dm * dm));
            igama = sd::div(1.0, gama);
            vm = dm * igama;
        }
        h = B * iBtot;
        vdothp = grp_add(0.0, vm * h);
        const double q = vm - vdothp * h;
        vperp = sd::sqrt_rn(grp_sum(q * q));
        hp = sd::div(q, vperp);
        hr = grp(h, c1) * grp(hp, c2) - grp(h, c2) * grp(hp, c1);
        const double omegac = cm * Btot * igama;
        const double dtheta = omegac * dt;
        const double ang = half ? dtheta : dtheta * 0.5;
        if (SYS == TP_SYS_MHD || SYS == TP_SYS_PIC) {
            sind = sin(ang);
            cosd = cos(ang);
        } else {
            sd::sin_cos(ang, sind, cosd);
        }
        if (half) break;
        const double gyroR = sd::div(vperp * gama * 1.0 * iBtot, f.d_cm);
        const double tmp1 = dth * vdothp * 1.0, tmp2 = gyroR * sind, tmp3 = -gyroR * (1.0 - cosd);
        px = x + h * tmp1 + hp * tmp2 + hr * tmp3;
    }
    const double vp = h * vdothp + vperp * (cosd * hp - sind * hr);
    const double bm = grp_add(0.0, vp * vp);
    const double g2 = sd::div(1.0, sd::sqrt_rn(1.0 - bm));
    u = g2 * vp + cm * dth * E;
    vdothp = grp_add(0.0, vp * h);
    const double q = vp - vdothp * h;
    vperp = sd::sqrt_rn(grp_sum(q * q));
    const double gyroR = sd::div(vperp * gama * 1.0 * iBtot, f.d_cm);
    const double tmp1 = dt * vdothp * 1.0;
    const double tmp2 = gyroR * sind;
    const double tmp3 = -gyroR * (1.0 - cosd);
    x += h * tmp1 + hp * tmp2 + hr * tmp3;
    t += dt;
}

// particle_bc for one component: the new shift, and whether it left the box
__device__ __forceinline__ bool small_bc(const DevField& f, int c, double& x, double& xs)
{
    const double lo = c == 0 ? f.xmin : c == 1 ? f.ymin : f.zmin, hi = c == 0 ? f.xmax : c == 1 ? f.ymax : f.zmax;
    const double dim = hi - lo;
    if (f.bc_flag == 0) {
        if (x > hi) { x -= dim; xs += dim; }
        if (x < lo) { x += dim; xs -= dim; }
        return false;
    }
    return f.bc_flag == 1 && (x > hi || x < lo);
}

// Whole runs without trajectory records; ntiles = gridDim.x blocks of 32 particles.
// OPEN: particles may leave (bc_flag is not 0); a form of its own, as the code for
// them costs the closed box 0.5 to 1 %.
template <int SYS, bool OPEN>
__global__ void __launch_bounds__(128) track_small_kernel(DevField f, TrackBufs b, TrackParams q)
{
    __shared__ double red[(128 / 32) * 8];
    __shared__ SmallShared sh;
    if (SYS == TP_SYS_MODESUM) {
        extern __shared__ int4 s_ctab[];
        for (int k = threadIdx.x; k <= fx::kTab; k += blockDim.x) s_ctab[k] = f.ctab[k];
        __syncthreads();
    }
    const int i = blockIdx.x * kSmallTile + (threadIdx.x >> 2);
    const int c = (threadIdx.x & 3) == 3 ? 0 : threadIdx.x & 3;
    const bool active = i < q.n, lead = (threadIdx.x & 3) == 0;
    // groups past the end follow the last particle and write nothing (a group
    // at rest would divide zeros by zeros and take the FP64 instructions for it)
    const int il = min(i, q.n - 1);
    double x = (c == 0 ? b.x : c == 1 ? b.y : b.z)[il];
    double u = (c == 0 ? b.ux : c == 1 ? b.uy : b.uz)[il];
    double xs = (c == 0 ? b.xs : c == 1 ? b.ys : b.zs)[il];
    double t = b.t[il];
    int nst = b.nsteps_ptl[il];
    // a group's escape: any of its lanes out of the box
    auto group_any = [&](bool v) { return (__ballot_sync(0xffffffffu, v) >> (threadIdx.x & 28) & 7u) != 0u; };
    const bool out = small_bc(f, c, x, xs);
    bool esc_pre = group_any(out), esc_after = esc_pre;
    int ntp = q.ntp0, tstep = 1;
    double sg[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (active && lead && esc_pre && q.nsdc > 1) atomicSub(&b.remain[1], 1);
    double* slot_base = b.dpart + (size_t)blockIdx.x * q.nsdc * 8;
    // countdowns to the next diagnostic steps (j % einterval, j % 100)
    int to_frame = (q.einterval - q.sstep % q.einterval) % q.einterval;
    int to_diff = (kDiffInterval - q.sstep % kDiffInterval) % kDiffInterval;
    for (int j = q.sstep; j <= q.estep; j++) {
        const bool diff = to_diff == 0, frame = to_frame == 0;
        to_diff = diff ? kDiffInterval - 1 : to_diff - 1;
        to_frame = frame ? q.einterval - 1 : to_frame - 1;
        const bool moves = !OPEN || !esc_pre;
        sg[0] = 0.0; sg[4] = 0.0; sg[5] = 0.0;  // src/tracking.c:334-336
        // with open boundaries: groups whose particle has left follow one of their
        // warp that has not (their own position, outside, would cost the slow
        // forms of the field), and a warp without any pushes nothing (the current
        // systems: a block, whose warps share the wires).  400 steps of an open box,
        // 9,000 particles: grid 27.3 -> 8.2 ms, ABC 14.2 -> 3.7; one: 13.3 -> 1.2.
        double xn = x, un = u, tn = t, xsn = xs;
        bool push = true;
        if (OPEN) {
            const unsigned mv = __ballot_sync(0xffffffffu, moves);
            const int from = moves || mv == 0u ? threadIdx.x & 31 : ((__ffs((int)mv) - 1) & 28) | (threadIdx.x & 3);
            xn = __shfl_sync(0xffffffffu, x, from);
            un = __shfl_sync(0xffffffffu, u, from);
            tn = __shfl_sync(0xffffffffu, t, from);
            push = SYS == TP_SYS_WLCS ? __syncthreads_or(mv != 0u) != 0 : mv != 0u;
        }
        if (push) {
            small_wirz<SYS>(f, c, xn, un, tn, q.dt, sh, active && moves ? b.status : nullptr);
            const bool left = small_bc(f, c, xn, xsn);
            const bool any = group_any(left);
            if (moves) {
                x = xn; u = un; t = tn; xs = xsn;
                if (any) esc_after = true;
                if (f.bc_flag == 2) esc_after = false;
                nst += 1;
            }
        }
        const unsigned need = __ballot_sync(0xffffffffu, diff || frame || (esc_after && !esc_pre));
        if (need) {
            P64 p;
            p.x = grp(x, 0); p.y = grp(x, 1); p.z = grp(x, 2);
            p.ux = grp(u, 0); p.uy = grp(u, 1); p.uz = grp(u, 2);
            p.xs = grp(xs, 0); p.ys = grp(xs, 1); p.zs = grp(xs, 2);
            p.t = t;
            if (active && lead) {
                if (moves && !esc_after && diff) {
                    P64 p0 = {};
                    p0.x = b.x0[i]; p0.y = b.y0[i]; p0.z = b.z0[i];
                    p0.ux = b.ux0[i]; p0.uy = b.uy0[i]; p0.uz = b.uz0[i]; p0.t = b.t0[i];
                    calc_diff<SYS, SYS == TP_SYS_MODESUM>(f, p0, p, q.dt, sg, b.status);
                }
                if (!esc_pre && esc_after && f.bc_flag == 1 && ntp < q.nt_out)
                    atomicAdd(&b.espect_esc[ntp * q.nbins + energy_bin(b.ebin_thr, q.nbins, p.ux, p.uy, p.uz)], 1u);
                if (frame && ntp < q.nt_out && !esc_after)
                    atomicAdd(&b.espect[ntp * q.nbins + energy_bin(b.ebin_thr, q.nbins, p.ux, p.uy, p.uz)], 1u);
            }
        }
        if (frame) ntp++;
        if (diff) {  // block-uniform
            block_diff_sum(sg, red, slot_base + (size_t)tstep * 8);
            tstep++;
        }
        if (active && lead && esc_after && diff && tstep < q.nsdc) atomicSub(&b.remain[tstep], 1);
        esc_pre = esc_after;
    }
    if (active && (threadIdx.x & 3) < 3) {
        (c == 0 ? b.x : c == 1 ? b.y : b.z)[i] = x;
        (c == 0 ? b.ux : c == 1 ? b.uy : b.uz)[i] = u;
        (c == 0 ? b.xs : c == 1 ? b.ys : b.zs)[i] = xs;
        if (lead) {
            b.t[i] = t;
            b.nsteps_ptl[i] = nst;
        }
    }
}

template <int SYS>
static cudaError_t launch_small_sys(const DevField& f, const TrackBufs& b, const TrackParams& q, int num_sms,
                                    cudaStream_t s)
{
    const int blocks = (q.n + kSmallTile - 1) / kSmallTile;
    size_t smem = SYS == TP_SYS_MODESUM ? sizeof(int4) * (fx::kTab + 1) : 0;
    // up to one block an SM, each asks for more than half of an SM's shared
    // memory, so that no two share one's FP64 pipes
    if (blocks <= num_sms) smem = std::max(smem, (size_t)120 * 1024);
    auto kernel = f.bc_flag != 0 ? track_small_kernel<SYS, true> : track_small_kernel<SYS, false>;
    if (smem > 0) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    kernel<<<blocks, 128, smem, s>>>(f, b, q);
    return cudaGetLastError();
}

// Blocks of a small run of this field, or 0: track_kernel is the better or the
// only one for it.  Whole runs, host buffers in and out: ABC, 200 steps, 3.0 ms
// in track_kernel up to its first full wave against 1.8 with one block an SM
// here, 2.1 with two, 2.8 with three; 256^3 grid, 50 steps, 1.24 against 0.95,
// 1.25 and 1.64 (every lane evaluates the grid); two wires and loops, 40 steps
// (before ellint_fx.cuh), 4.6 against 1.8 and 2.4; mode sum, 10 steps, 2.3 against 0.7, 1.0 and 1.7
// with four.
int track_small_blocks(const DevField& f, int n, int num_sms)
{
    const bool grids = f.system_type == TP_SYS_PIC || f.system_type == TP_SYS_MHD;
    const int per_sm = f.system_type == TP_SYS_MODESUM ? 4 : grids ? 2 : 3;
    const int blocks = (n + kSmallTile - 1) / kSmallTile;
    if (n < 1 || blocks > per_sm * num_sms) return 0;
    if (f.system_type == TP_SYS_WLCS && f.nwlcs > kSmallSystems) return 0;
    // a mode table that stays in FP64 is not split over the lanes: every lane
    // would sum all of it (17,000 modes, 9,000 particles x 2 steps: 159 ms, 92 in
    // track_kernel; one particle: 92 and 84)
    if (f.system_type == TP_SYS_MODESUM && !f.fxm) return 0;
    return blocks;
}

cudaError_t launch_track_small(const DevField& f, const TrackBufs& b, const TrackParams& q, int num_sms, cudaStream_t s)
{
    switch (f.system_type) {
    case TP_SYS_TEST: return launch_small_sys<TP_SYS_TEST>(f, b, q, num_sms, s);
    case TP_SYS_WLCS: return launch_small_sys<TP_SYS_WLCS>(f, b, q, num_sms, s);
    case TP_SYS_FORCEFREE: return launch_small_sys<TP_SYS_FORCEFREE>(f, b, q, num_sms, s);
    case TP_SYS_MHD: return launch_small_sys<TP_SYS_MHD>(f, b, q, num_sms, s);
    case TP_SYS_PIC: return launch_small_sys<TP_SYS_PIC>(f, b, q, num_sms, s);
    case TP_SYS_MODESUM: return launch_small_sys<TP_SYS_MODESUM>(f, b, q, num_sms, s);
    default: return cudaErrorInvalidValue;
    }
}
