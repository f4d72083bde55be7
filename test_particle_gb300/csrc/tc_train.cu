// tc_train.cu -- the GEMMs of the learned field model's training on the
// 5th-generation tensor cores: BF16 operands, FP32 accumulation in tensor
// memory, and a fused epilogue per use (bias + SiLU of the forward pass, the
// SiLU derivative of the backward pass).
//
// Everything the GEMMs exchange lies in global memory the way shared memory
// wants it: a matrix of samples [M][C] as blocks of 128 samples x 64 columns
// (16 KB), each row 128 bytes with its 16-byte pieces swizzled (tile_offset).
// One block is
//   - a k-atom of the next layer's A operand (rows = samples, K-major),
//   - 128 samples of a weight gradient's operand (its contraction runs over
//     the samples, so the same rows are read MN-major),
//   - in 4 KB strips of 32 rows, what an epilogue warp holds,
// so a single thread moves it with cp.async.bulk, no transposed copy of the
// activations and gradients exists, and the epilogues write 4 KB at a time.
// With row-major activations, 16-byte cp.async and a transposed copy of each
// for the weight gradients, a layer of 65,536 samples took 33 us forward and
// 33 us backward; now 20.4 and 21.2 (96 MB each, 4.5 TB/s).
//
// Every wait is bounded; one that runs out sets the block's abort flag, every
// other wait then gives up, the block waits (bounded) for its copies and MMAs
// in flight, frees tensor memory and raises ST_TIMEOUT.
#include <algorithm>
#include <cstdint>

#include "../../include/tp_gpu.h"
#include "mlp_common.cuh"
#include "tc_sm100.cuh"
#include "tc_train.cuh"
#include "tp_internal.h"

namespace tp {
namespace tct {

constexpr uint32_t kBlk = 16384;     // bytes of a block: 128 samples x 64 columns
constexpr uint32_t kSmem = 230400;   // dynamic shared memory of a CTA (1 KB of it for alignment)
constexpr uint32_t kLimit = 1u << 22;

__device__ __forceinline__ bool ws_wait(uint32_t bar, uint32_t parity, volatile int* abort)
{
    for (uint32_t it = 0; it < kLimit; it++) {
        if (tc::mbar_try_wait(bar, parity)) return true;
        if ((it & 63u) == 63u && *abort) return false;
    }
    *abort = 1;
    return false;
}

// A ring of shared-memory stages as one side walks it: the stage and the
// parity of its use.
struct Ring {
    int st = 0;
    uint32_t use = 0;
    __device__ void next(int n)
    {
        if (++st == n) {
            st = 0;
            use++;
        }
    }
};

// ---------------------------------------------------------------- epilogues
// What an epilogue warp of the layer kernel has: its staging (two strips of
// 32 rows x 64 columns, 4 KB each), its mbarriers (one a strip) and its place.
struct Warp {
    uint32_t stage, bar;
    int lane, q, c64;  // accumulator lanes 32 q.., first 64-column block
    volatile int* abort;
};

// 16-byte piece k of this lane's row in a strip
__device__ __forceinline__ uint32_t piece(uint32_t strip, int lane, int k)
{
    return strip + (uint32_t)lane * 128u + (uint32_t)((k ^ (lane & 7)) << 4);
}

__device__ __forceinline__ void st_piece(uint32_t at, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// strip `c` (64-column block) of the warp's 32 rows of tile t, in a matrix of 256 columns
__device__ __forceinline__ size_t strip_offset(int t, const Warp& w, int c)
{
    return ((size_t)t * 4 + c) * kBlk + (size_t)w.q * 4096u;
}

// z = acc + b; Z, H = silu(z)
struct EpiHidden {
    const float* b;
    unsigned char *Z, *H;
    __device__ void begin(const Warp&, int, int) {}
    __device__ bool block(const Warp& w, int t, int, int h, uint32_t acc)
    {
        const int c = w.c64 + h;
#pragma unroll
        for (int s = 0; s < 2; s++) {
            float v[32];
            tc::tmem_ld32(acc + 32u * s, v);
            uint32_t zp[16], hp[16];
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                const float4 b4 = __ldg(reinterpret_cast<const float4*>(b + 64 * c + 32 * s + j));
                const float z0 = v[j] + b4.x, z1 = v[j + 1] + b4.y, z2 = v[j + 2] + b4.z, z3 = v[j + 3] + b4.w;
                zp[j / 2] = mlp::pack_bf16(z0, z1);
                zp[j / 2 + 1] = mlp::pack_bf16(z2, z3);
                hp[j / 2] = mlp::pack_bf16(mlp::silu(z0), mlp::silu(z1));
                hp[j / 2 + 1] = mlp::pack_bf16(mlp::silu(z2), mlp::silu(z3));
            }
            if (s == 0) {  // the previous block's strips have been read
                if (w.lane == 0) tc::bulk_wait_read();
                __syncwarp();
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                st_piece(piece(w.stage, w.lane, 4 * s + k), zp[4 * k], zp[4 * k + 1], zp[4 * k + 2], zp[4 * k + 3]);
                st_piece(piece(w.stage + 4096u, w.lane, 4 * s + k), hp[4 * k], hp[4 * k + 1], hp[4 * k + 2],
                         hp[4 * k + 3]);
            }
        }
        tc::fence_async_smem();
        __syncwarp();
        if (w.lane == 0) {
            const size_t o = strip_offset(t, w, c);
            tc::bulk_s2g(Z + o, w.stage, 4096);
            tc::bulk_s2g(H + o, w.stage + 4096u, 4096);
            tc::bulk_commit();
        }
        return true;
    }
    __device__ void finish(const Warp& w)
    {
        if (w.lane == 0) tc::bulk_wait_all();
    }
};

// g = acc * silu'(Z).  The strips of Z are fetched two blocks ahead,
// each as soon as the strip of G that replaced it has been read back out.
struct EpiBackSilu {
    const unsigned char* Z;
    unsigned char* G;
    uint32_t got[2];  // uses of each strip's mbarrier so far; loads in flight
    bool pend[2];
    __device__ void fetch(const Warp& w, int t, int h)
    {
        if (w.lane == 0) {
            tc::mbar_expect_tx(w.bar + 8u * h, 4096);
            tc::bulk_g2s(w.stage + 4096u * h, Z + strip_offset(t, w, w.c64 + h), 4096, w.bar + 8u * h);
        }
        pend[h] = true;
    }
    __device__ void begin(const Warp& w, int t, int ntiles)
    {
        for (int h = 0; h < 2; h++) {
            got[h] = 0;
            pend[h] = false;
            if (t < ntiles) fetch(w, t, h);
        }
    }
    __device__ bool block(const Warp& w, int t, int tnext, int h, uint32_t acc)
    {
        if (!__all_sync(0xffffffffu, ws_wait(w.bar + 8u * h, got[h] & 1u, w.abort))) return false;
        got[h]++;
        pend[h] = false;
        const uint32_t strip = w.stage + 4096u * h;
#pragma unroll
        for (int s = 0; s < 2; s++) {
            float v[32];
            tc::tmem_ld32(acc + 32u * s, v);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t at = piece(strip, w.lane, 4 * s + k);
                uint32_t z[4], gp[4];
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(z[0]), "=r"(z[1]), "=r"(z[2]), "=r"(z[3]) : "r"(at) : "memory");
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float2 zf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&z[j]));
                    gp[j] = mlp::pack_bf16(v[8 * k + 2 * j] * mlp::silu_grad(zf.x),
                                           v[8 * k + 2 * j + 1] * mlp::silu_grad(zf.y));
                }
                st_piece(at, gp[0], gp[1], gp[2], gp[3]);
            }
        }
        tc::fence_async_smem();
        __syncwarp();
        if (w.lane == 0) {
            tc::bulk_s2g(G + strip_offset(t, w, w.c64 + h), strip, 4096);
            tc::bulk_commit();
        }
        if (tnext >= 0) {
            if (w.lane == 0) tc::bulk_wait_read();
            fetch(w, tnext, h);
        }
        return true;
    }
    __device__ void finish(const Warp& w)
    {
        if (w.lane == 0) {
            tc::bulk_wait_all();
            for (int h = 0; h < 2; h++)  // after a give-up: a load in flight (bounded)
                if (pend[h]) tc::mbar_wait(w.bar + 8u * h, got[h] & 1u, kLimit);
        }
    }
};

// y = acc + b for the first kOut columns (N = 16)
struct EpiOut {
    const float* b;
    float* Y;
    __device__ void begin(const Warp&, int, int) {}
    __device__ bool block(const Warp& w, int t, int, int, uint32_t acc)
    {
        float v[16];
        tc::tmem_ld16(acc, v);
        const size_t m = (size_t)t * 128 + 32 * w.q + w.lane;
        for (int c = 0; c < mlp::kOut; c++) Y[m * mlp::kOut + c] = v[c] + b[c];
        return true;
    }
    __device__ void finish(const Warp&) {}
};

// The same in a training batch of n samples, with the loss: r = y - (t - mean) /
// std, its gradient dY = 2 r / (n kOut) as FP32 rows and, in BF16, the first
// eight columns of a block (the others stay zero), and the sum of r^2.  (As a
// kernel of its own behind the GEMM this took 5.9 us for 65,536 samples.)
struct EpiOutLoss {
    const float* b;
    float* Y;  // null: not kept
    tctrain::Loss ls;
    float scale;
    __device__ void begin(const Warp&, int, int) {}
    __device__ bool block(const Warp& w, int t, int, int, uint32_t acc)
    {
        const size_t m = (size_t)t * 128 + 32 * w.q + w.lane;
        float tg[mlp::kOut], v[16];
        for (int c = 0; c < mlp::kOut; c++) tg[c] = ls.T[m * mlp::kOut + c];
        tc::tmem_ld16(acc, v);
        float l = 0.f, g[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int c = 0; c < mlp::kOut; c++) {
            const float y = v[c] + b[c];
            if (Y) Y[m * mlp::kOut + c] = y;
            const float r = y - (tg[c] - ls.mean[c]) * ls.istd[c];
            l += r * r;
            g[c] = r * scale;
            ls.dYf[m * mlp::kOut + c] = g[c];
        }
        *reinterpret_cast<uint4*>(ls.dY + tctrain::tile_offset(m, 0, 1)) =
            make_uint4(mlp::pack_bf16(g[0], g[1]), mlp::pack_bf16(g[2], g[3]), mlp::pack_bf16(g[4], g[5]),
                       mlp::pack_bf16(g[6], g[7]));
        for (int off = 16; off > 0; off >>= 1) l += __shfl_down_sync(0xffffffffu, l, off);
        if (w.lane == 0) atomicAdd(ls.sum, (double)l);
        return true;
    }
    __device__ void finish(const Warp&) {}
};

struct EpiStoreF32 {  // D[m][n] = acc (self-check)
    float* D;
    __device__ void begin(const Warp&, int, int) {}
    __device__ bool block(const Warp& w, int t, int, int h, uint32_t acc)
    {
        const size_t m = (size_t)t * 128 + 32 * w.q + w.lane;
#pragma unroll
        for (int s = 0; s < 2; s++) {
            float v[32];
            tc::tmem_ld32(acc + 32u * s, v);
            for (int j = 0; j < 32; j++) D[m * 256 + 64 * (w.c64 + h) + 32 * s + j] = v[j];
        }
        return true;
    }
    __device__ void finish(const Warp&) {}
};

// ---------------------------------------------------------------- a layer
// C[m][n] = sum_k A[m][k] B[n][k] for N = 256 (K <= 256) or 16 columns, A in
// blocks, B as k-atoms of N rows: a persistent kernel with one role per warp,
// one CTA per SM walking 128-row tiles:
//   warp 0  copies: one thread brings the whole B operand (the layer's
//           weights) into shared memory, where it stays, and the A k-atoms of
//           every tile into a ring of stages, as deep as shared memory allows
//           (2 for K = 256: 32 KB in flight, 5 MB over the chip);
//   warp 1  MMA: one thread issues the four K = 16 MMAs per atom into one of
//           two accumulators in tensor memory (alternating per tile), frees
//           the stage on `empty` and signals `accf` per tile;
//   warps 2.. epilogue (eight: two per quadrant of tensor-memory lanes, each
//           taking half of the columns; four for N = 16): each takes its 32
//           rows of a finished tile and signals `acce` when its part of the
//           accumulator is drained.
// So a tile's epilogue overlaps the next tile's copies and MMAs.
constexpr int kMaxRing = 8;
constexpr uint32_t kStageBytes = 8192;  // an epilogue warp's staging
__host__ __device__ constexpr int epi_warps(int n) { return n == 256 ? 8 : 4; }
__host__ __device__ constexpr int ws_threads(int n) { return 64 + 32 * epi_warps(n); }
__host__ __device__ inline int ws_ring(int n, int katoms)
{
    const uint32_t fixed = 1024 + (uint32_t)katoms * n * 128 + (uint32_t)epi_warps(n) * kStageBytes;
    return (kSmem - fixed) / kBlk < (uint32_t)kMaxRing ? (int)((kSmem - fixed) / kBlk) : kMaxRing;
}

template <class Epi, int N>
__global__ void __launch_bounds__(ws_threads(N), 1)
    layer_kernel(const unsigned char* __restrict__ A, const unsigned char* __restrict__ B, int ntiles, int katoms,
                 Epi epi, int* __restrict__ status)
{
    constexpr int EW = epi_warps(N);
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kMaxRing + 6 + 2 * EW];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ring = ws_ring(N, katoms);
    const uint32_t raw = tc::smem_addr(smem_raw);
    const uint32_t sB = raw + ((1024u - (raw & 1023u)) & 1023u);
    const uint32_t sA = sB + (uint32_t)katoms * N * 128u;
    const uint32_t stage0 = sA + (uint32_t)ring * kBlk;
    const uint32_t bar0 = tc::smem_addr(&bars[0]);
    auto full = [&](int st) { return bar0 + 8u * st; };
    auto empty = [&](int st) { return bar0 + 8u * (kMaxRing + st); };
    const uint32_t bfull = bar0 + 8u * (2 * kMaxRing);
    auto accf = [&](int b) { return bar0 + 8u * (2 * kMaxRing + 1 + b); };
    auto acce = [&](int b) { return bar0 + 8u * (2 * kMaxRing + 3 + b); };
    const uint32_t fin = bar0 + 8u * (2 * kMaxRing + 5);
    volatile int* abort = &abort_flag;
    if (tid == 0) {
        for (int st = 0; st < ring; st++) {
            tc::mbar_init(full(st), 1);
            tc::mbar_init(empty(st), 1);
        }
        tc::mbar_init(bfull, 1);
        for (int b = 0; b < 2; b++) {
            tc::mbar_init(accf(b), 1);
            tc::mbar_init(acce(b), 32 * EW);
        }
        tc::mbar_init(fin, 1);
        for (int k = 0; k < 2 * EW; k++) tc::mbar_init(fin + 8u + 8u * k, 1);
        tc::mbar_fence_init();
        abort_flag = 0;
    }
    constexpr uint32_t kAcc = N == 256 ? 256u : 32u;  // tensor-memory columns of an accumulator
    if (warp == 1) {
        tc::tmem_alloc(tc::smem_addr(&tmem_slot), 2 * kAcc);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            const uint32_t batom = (uint32_t)N * 128u;
            tc::mbar_expect_tx(bfull, (uint32_t)katoms * batom);
            for (int a = 0; a < katoms; a++) tc::bulk_g2s(sB + a * batom, B + (size_t)a * batom, batom, bfull);
            Ring r;
            bool ok = true;
            for (int t = blockIdx.x; ok && t < ntiles; t += gridDim.x) {
                const unsigned char* src = A + (size_t)t * katoms * kBlk;
                for (int a = 0; a < katoms; a++, r.next(ring)) {
                    if (r.use > 0) ok = ws_wait(empty(r.st), (r.use - 1) & 1u, abort);
                    if (!ok) break;
                    tc::mbar_expect_tx(full(r.st), kBlk);
                    tc::bulk_g2s(sA + (uint32_t)r.st * kBlk, src + (size_t)a * kBlk, kBlk, full(r.st));
                }
            }
            // nothing in flight when the block ends (only a give-up leaves something)
            if (!tc::mbar_wait(bfull, 0, kLimit)) abort_flag = 1;
            for (int st = 0; st < ring; st++) {
                const int uses = (int)r.use + (st < r.st ? 1 : 0);
                if (uses > 0 && !tc::mbar_wait(full(st), (uint32_t)(uses - 1) & 1u, kLimit)) abort_flag = 1;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0 && ws_wait(bfull, 0, abort)) {
            tc::tc_fence_after();
            const uint32_t idesc = tc::idesc_bf16_f32(128, N);
            Ring r;
            uint32_t j = 0;
            bool ok = true;
            for (int t = blockIdx.x; ok && t < ntiles; t += gridDim.x, j++) {
                const int b = (int)(j & 1u);
                const uint32_t v = j >> 1;
                if (v > 0) ok = ws_wait(acce(b), (v - 1) & 1u, abort);
                if (!ok) break;
                tc::tc_fence_after();
                for (int a = 0; a < katoms; a++, r.next(ring)) {
                    ok = ws_wait(full(r.st), r.use & 1u, abort);
                    if (!ok) break;
                    tc::tc_fence_after();
                    const uint64_t ad = tc::desc_sw128(sA + (uint32_t)r.st * kBlk);
                    const uint64_t bd = tc::desc_sw128(sB + (uint32_t)a * N * 128u);
#pragma unroll
                    for (int kk = 0; kk < 4; kk++)
                        tc::mma_bf16(tmem + (uint32_t)b * kAcc, ad + 2 * kk, bd + 2 * kk, idesc, (a | kk) != 0);
                    tc::mma_commit(empty(r.st));
                }
                if (ok) tc::mma_commit(accf(b));
            }
        }
        __syncwarp();
    } else {
        const int w = warp - 2;
        Warp me;
        me.stage = stage0 + (uint32_t)w * kStageBytes;
        me.bar = fin + 8u + 16u * w;
        me.lane = lane;
        me.q = warp & 3;  // the tensor-memory lanes this warp may read
        me.c64 = (w >> 2) * 2;
        me.abort = abort;
        const uint32_t acc0 = tmem + ((uint32_t)(32 * me.q) << 16) + 64u * me.c64;
        epi.begin(me, blockIdx.x, ntiles);
        uint32_t j = 0;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x, j++) {
            const int b = (int)(j & 1u);
            const int tn = t + (int)gridDim.x < ntiles ? t + (int)gridDim.x : -1;
            if (!__all_sync(0xffffffffu, ws_wait(accf(b), (j >> 1) & 1u, abort))) break;
            tc::tc_fence_after();
            bool ok = true;
#pragma unroll
            for (int h = 0; h < (N == 256 ? 2 : 1); h++)
                ok = ok && epi.block(me, t, tn, h, acc0 + (uint32_t)b * kAcc + 64u * h);
            if (!ok) break;
            tc::tc_fence_before();
            tc::mbar_arrive(acce(b));
        }
        epi.finish(me);
    }
    __syncthreads();
    if (warp == 1) {
        if (lane == 0) {  // every MMA this block issued has completed (bounded)
            tc::mma_commit(fin);
            if (!tc::mbar_wait(fin, 0, kLimit)) abort_flag = 1;
        }
        __syncwarp();
    }
    __syncthreads();
    if (tid == 0 && abort_flag) atomicOr(status, ST_TIMEOUT);
    if (warp == 1) tc::tmem_dealloc(tmem, 2 * kAcc);
}

template <int N, class Epi>
static cudaError_t launch_layer(const void* A, const void* B, int M, int K, const Epi& epi, int* status,
                                cudaStream_t s)
{
    if (M < 128 || M % 128 || K % 64 || K < 64 || K > 256) return cudaErrorInvalidValue;
    cudaError_t e =
        cudaFuncSetAttribute(layer_kernel<Epi, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return e;
    layer_kernel<Epi, N><<<tctrain::layer_blocks(M), ws_threads(N), kSmem, s>>>(
        static_cast<const unsigned char*>(A), static_cast<const unsigned char*>(B), M / 128, K / 64, epi, status);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- weight gradients
// P[split][x][n][m] = sum over the split's samples k of G[k][128 x + m] X[k][n]
// (m < 128, n < 64 xatoms <= 256): both operands are read MN-major from their
// blocks, 64 samples a stage (half a block of every 64 columns, 8 KB each).
// 15.2 us at 65,536 samples (64 + 32 MB; 19.0 from transposed copies) without the sums below.
// One output tile per CTA, the samples split over gridDim.y so that the CTAs
// fill the SMs.  Warp 0 copies, warp 1 issues the MMAs, warps 2..5 write the
// accumulator, 32 consecutive m (128 bytes) a store.
// Those four warps are idle until then: in the first 128 CTAs they take the bias
// gradients, the sums of G's columns, 16 columns and one of eight shares of the
// samples each.  The order of their sums and the shares of the weight gradients
// are those of one thread block per feature and of equal steps per split: a few
// AdamW steps turn the last place of a gradient into 1e-5 of the loss, so the
// order is kept although sums in the data gradient's epilogue would be cheaper
// (a batch of 65,536: this kernel 23 us with and 15 without the sums).
constexpr int kDwThreads = 192;
constexpr uint32_t kHalf = kBlk / 2;

// part[w][c] for the 16 columns from 16 (unit % 16) and w = unit / 16: the samples in
// groups of eight, group t + 256 k to running sum t (its pairs of samples one after
// the other), the 32 sums t = 32 w .. added as a tree.  Thread = (t, 4 columns), four
// groups' rows in flight.
constexpr int kBiasUnits = 128;
__device__ __forceinline__ void bias_unit(const unsigned char* __restrict__ G, int ngroups, int unit,
                                          float* __restrict__ part, float (*sums)[17])
{
    const int th = threadIdx.x - 64, q = th & 3, tl = th >> 2, c0 = (unit & 15) * 16, w = unit >> 4;
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    const int piece = ((c0 & 63) >> 3) + (q >> 1);
    const unsigned char* base = G + (size_t)(c0 >> 6) * kBlk + 8u * (q & 1);
#pragma unroll 4
    for (int i = 32 * w + tl; i < ngroups; i += 256) {
        const unsigned char* src = base + (size_t)(i >> 4) * 4 * kBlk + (size_t)(i & 15) * 1024u;
        uint2 v[8];
#pragma unroll
        for (int r = 0; r < 8; r++) v[r] = __ldg(reinterpret_cast<const uint2*>(src + r * 128 + ((piece ^ r) << 4)));
#pragma unroll
        for (int r = 0; r < 8; r += 2) {
            const uint32_t a[2] = {v[r].x, v[r].y}, b[2] = {v[r + 1].x, v[r + 1].y};
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const float2 fa = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a[j]));
                const float2 fb = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&b[j]));
                s[2 * j] += fa.x + fb.x;
                s[2 * j + 1] += fa.y + fb.y;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) sums[tl][4 * q + j] = s[j];
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (th < 16) {
        float t[32];
#pragma unroll
        for (int k = 0; k < 32; k++) t[k] = sums[k][th];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
#pragma unroll
            for (int k = 0; k < off; k++) t[k] += t[k + off];
        part[w * 256 + c0 + th] = t[0];
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
}
__host__ __device__ inline int dw_ring(int xatoms)
{
    const int n = (int)((kSmem - 1024 - 8192) / ((2 + xatoms) * kHalf));
    return n < kMaxRing ? n : kMaxRing;
}

__global__ void __launch_bounds__(kDwThreads, 1)
    weights_kernel(const unsigned char* __restrict__ G, int gatoms, const unsigned char* __restrict__ X, int xatoms,
                   int nsteps, int splits, float* __restrict__ P, float* __restrict__ bpart, int* __restrict__ status)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kMaxRing + 1];
    __shared__ float sums[32][17];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ring = dw_ring(xatoms);
    const uint32_t stage = (uint32_t)(2 + xatoms) * kHalf;
    const int chunk = (nsteps + splits - 1) / splits;
    const int k0 = blockIdx.y * chunk, k1 = min(nsteps, k0 + chunk);
    const uint32_t raw = tc::smem_addr(smem_raw);
    const uint32_t base = raw + ((1024u - (raw & 1023u)) & 1023u);
    const uint32_t bar0 = tc::smem_addr(&bars[0]);
    auto full = [&](int st) { return bar0 + 8u * st; };
    auto empty = [&](int st) { return bar0 + 8u * (kMaxRing + st); };
    const uint32_t fin = bar0 + 8u * (2 * kMaxRing);
    const uint32_t cols = xatoms == 1 ? 64u : xatoms == 2 ? 128u : 256u;
    volatile int* abort = &abort_flag;
    if (tid == 0) {
        for (int st = 0; st < ring; st++) {
            tc::mbar_init(full(st), 1);
            tc::mbar_init(empty(st), 1);
        }
        tc::mbar_init(fin, 1);
        tc::mbar_fence_init();
        abort_flag = 0;
    }
    if (warp == 1) {
        tc::tmem_alloc(tc::smem_addr(&tmem_slot), cols);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            Ring r;
            for (int k = k0; k < k1; k++, r.next(ring)) {
                if (r.use > 0 && !ws_wait(empty(r.st), (r.use - 1) & 1u, abort)) break;
                const uint32_t dst = base + (uint32_t)r.st * stage;
                const size_t row = (size_t)(k >> 1), half = (size_t)(k & 1) * kHalf;
                tc::mbar_expect_tx(full(r.st), stage);
                for (int a = 0; a < 2; a++)
                    tc::bulk_g2s(dst + a * kHalf, G + (row * gatoms + 2 * blockIdx.x + a) * kBlk + half, kHalf,
                                 full(r.st));
                for (int a = 0; a < xatoms; a++)
                    tc::bulk_g2s(dst + (2 + a) * kHalf, X + (row * xatoms + a) * kBlk + half, kHalf, full(r.st));
            }
            for (int st = 0; st < ring; st++) {  // nothing in flight when the block ends
                const int uses = (int)r.use + (st < r.st ? 1 : 0);
                if (uses > 0 && !tc::mbar_wait(full(st), (uint32_t)(uses - 1) & 1u, kLimit)) abort_flag = 1;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = tc::idesc_bf16_f32(128, 64 * xatoms) | tc::kIdescMnMajorAB;
            Ring r;
            for (int k = k0; k < k1; k++, r.next(ring)) {
                if (!ws_wait(full(r.st), r.use & 1u, abort)) break;
                tc::tc_fence_after();
                const uint32_t src = base + (uint32_t)r.st * stage;
                const uint64_t ad = tc::desc_sw128_mn(src, kHalf), bd = tc::desc_sw128_mn(src + 2 * kHalf, kHalf);
#pragma unroll
                for (int kk = 0; kk < 4; kk++)  // 16 samples: 2 KB of every half block
                    tc::mma_bf16(tmem, ad + 128 * kk, bd + 128 * kk, idesc, k > k0 || kk > 0);
                tc::mma_commit(empty(r.st));
            }
            tc::mma_commit(fin);
            if (!tc::mbar_wait(fin, 0, kLimit)) abort_flag = 1;
        }
        __syncwarp();
    } else if (bpart) {
        for (int u = blockIdx.y * gridDim.x + blockIdx.x; u < kBiasUnits; u += gridDim.x * gridDim.y)
            bias_unit(G, nsteps * 8, u, bpart, sums);
    }
    __syncthreads();
    tc::tc_fence_after();
    if (warp >= 2 && k0 < k1 && !*abort) {
        const int q = warp & 3;
        float* dst = P + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (64 * xatoms) * 128 + 32 * q + lane;
        for (int c = 0; c < 64 * xatoms; c += 32) {
            float v[32];
            tc::tmem_ld32(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)c, v);
#pragma unroll
            for (int j = 0; j < 32; j++) dst[(size_t)(c + j) * 128] = v[j];
        }
    }
    if (tid == 0 && abort_flag) atomicOr(status, ST_TIMEOUT);
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 1) tc::tmem_dealloc(tmem, cols);
}

static cudaError_t launch_weights(const void* G, int mtiles, const void* X, int xatoms, int nsteps, float* P,
                                  int splits, float* bpart, int* status, cudaStream_t s)
{
    if (splits < 1 || splits > nsteps || xatoms < 1 || xatoms > 4) return cudaErrorInvalidValue;
    const uint32_t smem = 1024 + (uint32_t)dw_ring(xatoms) * (2 + xatoms) * kHalf;
    cudaError_t e = cudaFuncSetAttribute(weights_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    // with few splits, CTAs without samples of their own for the column sums (a
    // training in batches of some 2,000 samples 0.79 -> 0.60 ms)
    const int used = tctrain::used_splits(nsteps, splits);
    const int rows = bpart ? std::max(used, (kBiasUnits + mtiles - 1) / mtiles) : used;
    weights_kernel<<<dim3(mtiles, rows), kDwThreads, smem, s>>>(
        static_cast<const unsigned char*>(G), 2 * mtiles, static_cast<const unsigned char*>(X), xatoms, nsteps,
        splits, P, bpart, status);
    return cudaGetLastError();
}

// Self-check: D[m][n] of one split of P
__global__ void from_split_kernel(const float* __restrict__ P, int M, int N, int npad, float* __restrict__ D)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)M * N) return;
    const int m = (int)(i / N), n = (int)(i % N);
    D[i] = P[((size_t)(m >> 7) * npad + n) * 128 + (m & 127)];
}

// Self-check: row-major A [rows][K] into blocks (kind 0), k-atoms of R rows
// (kind 1), or transposed, K the samples, into blocks of `atoms` 64-column
// atoms (kind 2); both operands in one launch (blockIdx.y).
struct PackOp {
    const __nv_bfloat16* A;
    int rows, kind, atoms;
    unsigned char* out;
};

__global__ void to_blocks_kernel(PackOp a, PackOp b, int K)
{
    const PackOp p = blockIdx.y == 0 ? a : b;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)p.rows * K) return;
    const int r = (int)(i / K), k = (int)(i % K);
    const size_t o = p.kind == 0   ? tctrain::tile_offset(r, k, p.atoms)
                     : p.kind == 1 ? (size_t)tc::sw128_offset(p.rows, r, k)
                                   : tctrain::tile_offset(k, r, p.atoms);
    *reinterpret_cast<__nv_bfloat16*>(p.out + o) = p.A[i];
}

}  // namespace tct

namespace tctrain {

using namespace tct;

// splits of equal whole steps: the last ones may be empty and are not launched
int used_splits(int nsteps, int splits)
{
    const int chunk = (nsteps + splits - 1) / splits;
    return (nsteps + chunk - 1) / chunk;
}

int layer_blocks(int M) { return std::min(M / 128, g.num_sms > 0 ? g.num_sms : 148); }

cudaError_t forward_hidden(const void* X, int kin, const void* W, int M, const float* b, void* Z, void* H,
                           int* status, cudaStream_t s)
{
    return launch_layer<256>(X, W, M, kin,
                             EpiHidden{b, static_cast<unsigned char*>(Z), static_cast<unsigned char*>(H)}, status, s);
}

cudaError_t forward_out(const void* H3, const void* W4, int M, const float* b, float* Y, int* status,
                        cudaStream_t s)
{
    return launch_layer<mlp::kOutPad>(H3, W4, M, mlp::kHid, EpiOut{b, Y}, status, s);
}

cudaError_t forward_loss(const void* H3, const void* W4, int M, const float* b, float* Y, const Loss& ls, int* status,
                         cudaStream_t s)
{
    return launch_layer<mlp::kOutPad>(H3, W4, M, mlp::kHid,
                                      EpiOutLoss{b, Y, ls, 2.0f / ((float)M * mlp::kOut)}, status, s);
}

cudaError_t backward_data(const void* Gin, int kout, const void* WT, int M, const void* Zprev, void* G,
                          int* status, cudaStream_t s)
{
    EpiBackSilu e{};
    e.Z = static_cast<const unsigned char*>(Zprev);
    e.G = static_cast<unsigned char*>(G);
    return launch_layer<256>(Gin, WT, M, kout, e, status, s);
}

cudaError_t backward_weights(const void* G, const void* X, int kin, int nsamp, float* P, int splits, float* bpart,
                             int* status, cudaStream_t s)
{
    return launch_weights(G, mlp::kHid / 128, X, kin / 64, nsamp / 64, P, splits, bpart, status, s);
}

// the shapes of the layer GEMMs go through the kernel those use, the others
// through the weight gradients' (operands transposed, columns padded with zeros)
static cudaError_t gemm_f32(const __nv_bfloat16* A, const __nv_bfloat16* B, int M, int N, int K,
                            unsigned char* work, float* D, int* status, cudaStream_t s)
{
    auto grid = [](size_t n) { return (unsigned)((n + 255) / 256); };
    const bool layer = N == 256 && K <= 256;
    const int kpad = (K + 127) / 128 * 128, npad = (N + 63) / 64 * 64;
    unsigned char *wa = work, *wb = work + 2 * (size_t)M * kpad;
    to_blocks_kernel<<<dim3(grid((size_t)std::max(M, N) * K), 2), 256, 0, s>>>(
        PackOp{A, M, layer ? 0 : 2, layer ? K / 64 : M / 64, wa},
        PackOp{B, N, layer ? 1 : 2, layer ? K / 64 : npad / 64, wb}, K);
    if (layer) return launch_layer<256>(wa, wb, M, K, EpiStoreF32{D}, status, s);
    float* P = reinterpret_cast<float*>(wb + 2 * (size_t)npad * kpad);
    cudaError_t e = launch_weights(wa, M / 128, wb, npad / 64, K / 64, P, 1, nullptr, status, s);
    if (e != cudaSuccess) return e;
    from_split_kernel<<<grid((size_t)M * N), 256, 0, s>>>(P, M, N, npad, D);
    return cudaGetLastError();
}

static size_t gemm_work_bytes(int M, int N, int K)
{
    const size_t kpad = (K + 127) / 128 * 128, npad = (N + 63) / 64 * 64;
    return 2 * M * kpad + 2 * npad * kpad + sizeof(float) * (size_t)M * npad;
}

}  // namespace tctrain
}  // namespace tp

using namespace tp;

// D[m][n] = A[m][k] * B[n][k]^T with BF16 inputs (raw 16-bit patterns) and FP32
// output, through the training GEMM kernels: m a multiple of 128, n a multiple
// of 16 in [16, 256], k a multiple of 64.
extern "C" int tp_tc_gemm_train_bf16(int m, int n, int k, const unsigned short* a, const unsigned short* b,
                                     float* d)
{
    if (m < 128 || m % 128 || n < 16 || n > 256 || n % 16 || k < 64 || k % 64 || !a || !b || !d) {
        set_error(6, "tp_tc_gemm_train_bf16: m a multiple of 128, n 16..256 in steps of 16, k a multiple of 64");
        return -1;
    }
    if (!ensure_init()) return -1;
    cudaStream_t s = g.stream;
    const size_t sa = sizeof(uint16_t) * (size_t)m * k, sb = sizeof(uint16_t) * (size_t)n * k,
                 sd = sizeof(float) * (size_t)m * n;
    // all of it in the batch calls' buffer (allocations of its own cost as much as
    // the kernels); the padding of the packed operands is zero
    auto whole = [](size_t b) { return (b + 1023) / 1024 * 1024; };
    const size_t sw = tctrain::gemm_work_bytes(m, n, k), oB = whole(sa), oD = oB + whole(sb), oW = oD + whole(sd);
    unsigned char* d0 = static_cast<unsigned char*>(g.s_batch_a.get(oW + sw));
    if (!d0) return -1;
    cudaMemcpyAsync(d0, a, sa, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(d0 + oB, b, sb, cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(d0 + oD, 0, oW + sw - oD, s);
    if (!cuda_ok(tctrain::gemm_f32(reinterpret_cast<const __nv_bfloat16*>(d0),
                                   reinterpret_cast<const __nv_bfloat16*>(d0 + oB), m, n, k, d0 + oW,
                                   reinterpret_cast<float*>(d0 + oD), g.d_status, s),
                 "train gemm"))
        return -1;
    cudaMemcpyAsync(d, d0 + oD, sd, cudaMemcpyDeviceToHost, s);
    return cuda_ok(cudaStreamSynchronize(s), "train gemm sync") ? 0 : -1;
}
