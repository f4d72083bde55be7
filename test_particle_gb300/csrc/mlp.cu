// mlp.cu -- training and inference of the learned field model: the forward,
// data-gradient and hidden weight-gradient GEMMs on the 5th-generation tensor
// cores (tc_train.cu: tcgen05.mma, FP32 accumulation in tensor memory, fused
// bias / SiLU / SiLU-derivative / loss epilogues), Fourier features, MSE
// loss, the output layer's 6 x 256 weight gradient as a reduction on the CUDA
// cores, and one kernel a batch that sums the partial gradients and takes the
// AdamW step.
//
// The model maps a position u in the periodic box (u = (x - min) / L) to the
// six field components: 64 integer-lattice frequencies f_j give the features
// sin(2 pi f_j . u), cos(2 pi f_j . u) (exact phases in 32-bit fixed point),
// then 128 -> 256 -> 256 -> 256 -> 256 -> 6 with SiLU.  Outputs are trained
// on normalised components (zero mean, unit variance per component).
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/tp_gpu.h"
#include "mlp_common.cuh"
#include "tc_train.cuh"
#include "tp_internal.h"
#include "tp_mixed.cuh"

namespace tp {
namespace mlp {

// ---------------------------------------------------------------- features
// X[b][j] = sin(2 pi f_j . u_b), X[b][64 + j] = cos(...) with u in 32-bit fixed
// point, as BF16 [n][128] in the GEMMs' blocks (tctrain::tile_offset).  A thread
// takes a sample, eight features at a time; a warp's 32 rows of both blocks are
// put together in shared memory (4 KB each, the global layout) and written 512
// bytes a store: 8.1 us for 65,536 samples (12.8 row by row with a transposed copy).
__global__ void __launch_bounds__(128) features_kernel(const uint32_t* __restrict__ U, int n,
                                                       const int* __restrict__ freq, unsigned char* __restrict__ X)
{
    __shared__ int fs[3 * kFeat];
    __shared__ uint4 strip[4][2][256];  // of a warp: sines, cosines
    for (int k = threadIdx.x; k < 3 * kFeat; k += blockDim.x) fs[k] = freq[k];
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t U0 = i < n ? U[3 * i] : 0u, U1 = i < n ? U[3 * i + 1] : 0u, U2 = i < n ? U[3 * i + 2] : 0u;
#pragma unroll 1
    for (int j0 = 0; j0 < kFeat; j0 += 8) {
        uint32_t sp[4], cp[4];
#pragma unroll
        for (int q = 0; q < 8; q += 2) {
            float s0, c0, s1, c1;
            const int j = j0 + q;
            const uint32_t ph0 = (uint32_t)fs[3 * j] * U0 + (uint32_t)fs[3 * j + 1] * U1 + (uint32_t)fs[3 * j + 2] * U2;
            const uint32_t ph1 = (uint32_t)fs[3 * j + 3] * U0 + (uint32_t)fs[3 * j + 4] * U1 +
                                 (uint32_t)fs[3 * j + 5] * U2;
            __sincosf(mixed::rev_to_rad(ph0), &s0, &c0);
            __sincosf(mixed::rev_to_rad(ph1), &s1, &c1);
            sp[q / 2] = pack_bf16(s0, s1);
            cp[q / 2] = pack_bf16(c0, c1);
        }
        const int at = lane * 8 + ((j0 / 8) ^ (lane & 7));
        strip[w][0][at] = make_uint4(sp[0], sp[1], sp[2], sp[3]);
        strip[w][1][at] = make_uint4(cp[0], cp[1], cp[2], cp[3]);
    }
    __syncwarp();
    // rows 32 w.. of the two blocks of this 128-sample tile
    uint4* dst = reinterpret_cast<uint4*>(X + (size_t)blockIdx.x * 32768u) + w * 256;
#pragma unroll
    for (int b = 0; b < 2; b++)
#pragma unroll
        for (int k = 0; k < 8; k++) dst[b * 1024 + k * 32 + lane] = strip[w][b][k * 32 + lane];
}

// ---------------------------------------------------------------- samples
__device__ __forceinline__ uint64_t mix64(uint64_t z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Uniform positions (32-bit fixed point per axis) and the exact FP64 mode-sum
// field there (the plane-wave sum of fields_fp64.cuh in the same phase form).
__global__ void __launch_bounds__(128) samples_kernel(uint64_t seed, long long first, int n, DevField f,
                                                      uint32_t* __restrict__ U, float* __restrict__ T)
{
    __shared__ int4 tab[fx::kTab + 1];
    if (f.fxm) {
        for (int k = threadIdx.x; k <= fx::kTab; k += blockDim.x) tab[k] = f.ctab[k];
        __syncthreads();
    }
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t id = (uint64_t)(first + i);
    uint32_t u[3];
    for (int k = 0; k < 3; k++) u[k] = (uint32_t)(mix64(seed ^ (id * 3 + k) * 0xD1342543DE82EF95ull) >> 32);
    double b[3] = {0, 0, 0}, e[3] = {0, 0, 0};
    if (f.fxm) {
        const uint64_t u64[3] = {(uint64_t)u[0] << 32, (uint64_t)u[1] << 32, (uint64_t)u[2] << 32};
        int64_t s[6];
        fx::mode_sum<fx::kChunk>(f.fxm, f.nfx, tab, u64, s);
        for (int k = 0; k < 3; k++) {
            b[k] = (double)s[k] * f.fxs[k];
            e[k] = (double)s[3 + k] * f.fxs[3 + k];
        }
    }
    for (int m = 0; m < (f.fxm ? 0 : f.nmodes); m++) {
        const tp_mode& md = f.modes[m];
        uint64_t ph = (uint64_t)(int64_t)md.n[0] * ((uint64_t)u[0] << 32) +
                      (uint64_t)(int64_t)md.n[1] * ((uint64_t)u[1] << 32) +
                      (uint64_t)(int64_t)md.n[2] * ((uint64_t)u[2] << 32) +
                      ((uint64_t)(uint32_t)md.pad << 32);
        double c = cos((double)(int64_t)ph * 3.4061215800865545e-19);
        for (int k = 0; k < 3; k++) {
            b[k] += md.amp_b[k] * c;
            e[k] += md.amp_e[k] * c;
        }
    }
    b[2] += f.B0;
    for (int k = 0; k < 3; k++) {
        U[3 * i + k] = u[k];
        T[6 * i + k] = (float)b[k];
        T[6 * i + 3 + k] = (float)e[k];
    }
}

// Sums and sums of squares (FP64) of the six target components over a block's
// samples, part[block][c] and part[block][6 + c]; the host adds the blocks.  FP64
// instructions bound it (two a value); as one chain on the host, the targets
// copied there first, 131,072 samples took 0.7 ms more of a training call.
__global__ void __launch_bounds__(128) moments_kernel(const float* __restrict__ T, int n, double* __restrict__ part)
{
    __shared__ double red[128][2 * kOut];
    __shared__ double col[8][2 * kOut];
    double a[kOut] = {}, b[kOut] = {};
    for (int i = blockIdx.x * 128 + threadIdx.x; i < n; i += gridDim.x * 128)
#pragma unroll
        for (int c = 0; c < kOut; c++) {
            const double x = T[(size_t)i * kOut + c];
            a[c] += x;
            b[c] += x * x;
        }
    for (int c = 0; c < kOut; c++) {
        red[threadIdx.x][c] = a[c];
        red[threadIdx.x][kOut + c] = b[c];
    }
    __syncthreads();
    const int c = threadIdx.x % (2 * kOut), g8 = threadIdx.x / (2 * kOut);
    if (g8 < 8) {
        double s = 0.0;
        for (int k = 0; k < 16; k++) s += red[g8 * 16 + k][c];
        col[g8][c] = s;
    }
    __syncthreads();
    if (g8 == 0) {
        double s = 0.0;
        for (int k = 0; k < 8; k++) s += col[k][c];
        part[blockIdx.x * 2 * kOut + c] = s;
    }
}

// ---------------------------------------------------------------- loss, output layer, AdamW
constexpr int kDYld = 64;         // columns of dY: one k-atom of the output layer's data-gradient GEMM
constexpr int kWgradSplits = 76;  // most split-K parts of a weight-gradient GEMM: two CTAs each, one an SM

// Partial sums of the output layer's gradients from the FP32 loss gradient dYf
// [n][6] and the last hidden activations H3 [n][256]: part[block] holds
// dW4[o][k] = sum_r dYf[r][o] H3[r][k] and, behind, db4[o] = sum_r dYf[r][o] over
// the block's 128-sample tiles.  Thread (g, c) takes columns 8 c.. of the 16
// rows 16 g.. of a tile: a warp reads a row's 512 bytes, 48 FMAs a thread and
// 16-byte load; the eight groups of rows are added in shared memory at the end.
// 17 us for 65,536 samples (32 MB, from HBM); with a column a thread, 2-byte loads
// and 128 samples a block added with atomics 25 us (39 from the blocks).
constexpr int kOutGrad = kOut * kHid + kOut;
__global__ void __launch_bounds__(256) out_grad_kernel(const float* __restrict__ dYf,
                                                       const unsigned char* __restrict__ H3, int ntiles,
                                                       float* __restrict__ part)
{
    __shared__ float4 dy[128 * 2];  // rows padded to eight values
    __shared__ float red[8][kHid + 1];
    const int c = threadIdx.x & 31, gr = threadIdx.x >> 5;
    float acc[kOut][8] = {}, accb = 0.f;
    float* dys = reinterpret_cast<float*>(dy);
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        __syncthreads();
        for (int i = threadIdx.x; i < 128 * kOut; i += 256)
            dys[(i / kOut) * 8 + i % kOut] = dYf[(size_t)t * 128 * kOut + i];
        const unsigned char* src = H3 + (size_t)t * 4 * 16384u + (size_t)(c >> 3) * 16384u;
        uint4 h[16];
#pragma unroll
        for (int r = 0; r < 16; r++)
            h[r] = *reinterpret_cast<const uint4*>(src + tc::sw128_offset(128, 16 * gr + r, 8 * (c & 7)));
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 16; r++) {
            const float4 a = dy[2 * (16 * gr + r)];
            const float2 b = *reinterpret_cast<const float2*>(&dy[2 * (16 * gr + r) + 1]);
            const float d[kOut] = {a.x, a.y, a.z, a.w, b.x, b.y};
            const uint32_t w[4] = {h[r].x, h[r].y, h[r].z, h[r].w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[j]));
#pragma unroll
                for (int o = 0; o < kOut; o++) {
                    acc[o][2 * j] = fmaf(d[o], f.x, acc[o][2 * j]);
                    acc[o][2 * j + 1] = fmaf(d[o], f.y, acc[o][2 * j + 1]);
                }
            }
        }
        if (threadIdx.x < 8 * kOut)  // sixteen rows of one output
            for (int r = 0; r < 16; r++) accb += dys[((threadIdx.x / kOut) * 16 + r) * 8 + threadIdx.x % kOut];
    }
    float* dst = part + (size_t)blockIdx.x * kOutGrad;
#pragma unroll
    for (int o = 0; o < kOut; o++) {
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 8; j++) red[gr][8 * c + j] = acc[o][j];
        __syncthreads();
        float s = 0.f;
        for (int g8 = 0; g8 < 8; g8++) s += red[g8][threadIdx.x];
        dst[o * kHid + threadIdx.x] = s;
    }
    __syncthreads();
    if (threadIdx.x < 8 * kOut) red[threadIdx.x / kOut][threadIdx.x % kOut] = accb;
    __syncthreads();
    if (threadIdx.x < kOut) {
        float s = 0.f;
        for (int g8 = 0; g8 < 8; g8++) s += red[g8][threadIdx.x];
        dst[kOut * kHid + threadIdx.x] = s;
    }
}

struct Adam {
    float lr, b1, b2, eps, wd, c1, c2;  // c1 = 1 / (1 - b1^t), c2 = 1 / (1 - b2^t)
};

// BF16 copies of the weights: as the forward GEMM's k-atoms of out_pad rows (wk),
// transposed, as the data gradient's k-atoms of `in` rows (wn, not layer 0; the
// output layer's columns past kOut stay zero) and in the tracking kernel's chunks.
struct Copies {
    unsigned char *wk[kLayers], *wn[kLayers], *pack;
};

__device__ __forceinline__ void store_weight(const Copies& c, int l, int o, int k, float w)
{
    const __nv_bfloat16 v = __float2bfloat16(w);
    *reinterpret_cast<__nv_bfloat16*>(c.wk[l] + tc::sw128_offset(layer_out_pad(l), o, k)) = v;
    if (l > 0) *reinterpret_cast<__nv_bfloat16*>(c.wn[l] + tc::sw128_offset(layer_in(l), k, o)) = v;
    *reinterpret_cast<__nv_bfloat16*>(c.pack + pack_offset(l, o, k)) = v;
}

// First parameter of layer l (weights [out][in], then biases) in the flat layout
__host__ __device__ constexpr int param_offset(int l)
{
    int off = 0;
    for (int k = 0; k < l; k++) off += layer_out(k) * (layer_in(k) + 1);
    return off;
}
constexpr int kParams = param_offset(kLayers);

__global__ void copies_kernel(const float* __restrict__ p, const __grid_constant__ Copies cp)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    for (int l = 0; l < kLayers; l++) {
        const int nw = layer_out(l) * layer_in(l);
        if (i < nw) {
            store_weight(cp, l, i / layer_in(l), i % layer_in(l), p[param_offset(l) + i]);
            return;
        }
        i -= nw;
    }
}

// Partial sums of the gradients: the hidden layers' weights by split
// (backward_weights), their biases in kBiasParts shares, the output layer by block of out_grad_kernel.
struct Partials {
    const float *w[4], *b[4], *out;
    int splits, oblocks;
};

// The end of a batch in one launch: every gradient is summed from its partial
// sums, in a fixed order, and either stored (gr) or used at once for the AdamW
// step, the new weights going out as FP32 and in their three BF16 copies.
// A block takes 32 x 8 of a hidden layer's weights (thread = one, 128-byte reads
// of every split, turned through shared memory for the row-major parameters), 32
// biases, or 32 of the output layer's parameters (eight threads each).  17.8
// us for 74 splits (66 MB read); a kernel per layer and purpose (four sums of
// splits, four of biases, AdamW, six of copies) took 137 us.
constexpr int kPatches0 = (kHid / 32) * (kIn / 8), kPatches = (kHid / 32) * (kHid / 8);
constexpr int kBiasBlocks = 4 * kHid / 32, kOutBlocks = (kOutGrad + 31) / 32;
constexpr int kUpdateBlocks = kPatches0 + 3 * kPatches + kBiasBlocks + kOutBlocks;

template <bool STEP>
__global__ void __launch_bounds__(256) update_kernel(const __grid_constant__ Partials ps, float* __restrict__ gr,
                                                     float* __restrict__ p, float* __restrict__ m,
                                                     float* __restrict__ v, Adam a, const __grid_constant__ Copies cp)
{
    __shared__ float red[8][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int blk = blockIdx.x, l, o, k, idx;
    float g;
    if (blk < kPatches0 + 3 * kPatches) {
        l = blk < kPatches0 ? 0 : 1 + (blk - kPatches0) / kPatches;
        const int i = blk < kPatches0 ? blk : (blk - kPatches0) % kPatches;
        const int in = layer_in(l), m0 = (i & 7) * 32, n0 = (i >> 3) * 8;
        const float* src = ps.w[l] + ((size_t)(m0 >> 7) * in + n0 + w) * 128 + (m0 & 127) + lane;
        const size_t step = (size_t)(kHid / 128) * in * 128;
        float s = 0.f;
#pragma unroll 8
        for (int q = 0; q < ps.splits; q++) s += src[q * step];
        red[w][lane] = s;
        __syncthreads();
        o = m0 + (threadIdx.x >> 3);
        k = n0 + (threadIdx.x & 7);
        g = red[threadIdx.x & 7][threadIdx.x >> 3];
        idx = param_offset(l) + o * in + k;
    } else {
        blk -= kPatches0 + 3 * kPatches;
        const bool bias = blk < kBiasBlocks;
        const float* src;
        int stride, n;
        bool in_range = true;
        if (bias) {
            l = blk / (kHid / 32);
            const int e = (blk % (kHid / 32)) * 32 + lane;
            src = ps.b[l] + e;
            stride = kHid;
            n = tctrain::kBiasParts;
            idx = param_offset(l) + kHid * layer_in(l) + e;
            o = k = -1;
        } else {
            l = kLayers - 1;
            const int e = (blk - kBiasBlocks) * 32 + lane;
            in_range = e < kOutGrad;
            src = ps.out + (in_range ? e : 0);
            stride = kOutGrad;
            n = ps.oblocks;
            idx = param_offset(l) + e;
            o = e < kOut * kHid ? e / kHid : -1;
            k = e % kHid;
        }
        float s = 0.f;
#pragma unroll 8
        for (int q = w; q < n; q += 8) s += src[(size_t)q * stride];
        red[w][lane] = s;
        __syncthreads();
        if (w > 0 || !in_range) return;
        g = 0.f;
#pragma unroll
        for (int q = 0; q < 8; q++) g += red[q][lane];
    }
    if (!STEP) {
        gr[idx] = g;
        return;
    }
    const float mi = a.b1 * m[idx] + (1.f - a.b1) * g;
    const float vi = a.b2 * v[idx] + (1.f - a.b2) * g * g;
    m[idx] = mi;
    v[idx] = vi;
    const float upd = (mi * a.c1) / (sqrtf(vi * a.c2) + a.eps);
    const float pn = p[idx] - a.lr * (upd + a.wd * p[idx]);
    p[idx] = pn;
    if (o >= 0) store_weight(cp, l, o, k, pn);
}

}  // namespace mlp

// ---------------------------------------------------------------- host model
using namespace mlp;

struct MlpState {
    bool ready = false, have_params = false;
    int freq_h[kFeat * 3];
    // parameters (FP32 master), gradients, Adam moments: one flat buffer each
    size_t nparam = 0;
    size_t woff[kLayers], boff[kLayers];
    float *p = nullptr, *gr = nullptr, *m = nullptr, *v = nullptr;
    Copies cp{};                            // BF16 copies of the weights
    int* freq = nullptr;
    float out_mean[kOut] = {0}, out_std[kOut] = {1, 1, 1, 1, 1, 1};
    float *d_mean = nullptr, *d_istd = nullptr;
    long step = 0;
    // batch workspaces
    int cap = 0;
    // samples x columns, BF16 in the GEMMs' blocks
    unsigned char* X = nullptr;             // [cap][128]
    unsigned char *Z[4] = {}, *H[4] = {};   // [cap][256]
    unsigned char *G0 = nullptr, *G1 = nullptr;  // [cap][256] backward scratch
    unsigned char* dY = nullptr;            // [cap][kDYld]
    // partial gradients: hidden weights by split, biases and output layer by block
    float *wpart[4] = {}, *bpart[4] = {}, *opart = nullptr;
    float* Y = nullptr;                     // [cap][6]
    float* dYf = nullptr;                   // [cap][6]
    double* loss = nullptr;
};

static MlpState M;

// most blocks of a kernel whose partial sums are kept by block
static int max_blocks() { return 2 * tctrain::layer_blocks(INT_MAX / 128 * 128); }

template <class T>
static void drop(T*& p)
{
    if (p) cudaFree(p);
    p = nullptr;
}

// Everything of the model itself, or nothing of it.
static bool mlp_alloc_params()
{
    if (M.have_params) return true;
    size_t off = 0;
    for (int l = 0; l < kLayers; l++) {
        M.woff[l] = off;
        off += (size_t)layer_out(l) * layer_in(l);
        M.boff[l] = off;
        off += layer_out(l);
    }
    M.nparam = off;  // = kParams
    const size_t b = sizeof(float) * off;
    bool ok = cuda_ok(cudaMalloc(&M.p, b), "mlp params") && cuda_ok(cudaMalloc(&M.gr, b), "mlp grads") &&
              cuda_ok(cudaMalloc(&M.m, b), "mlp m") && cuda_ok(cudaMalloc(&M.v, b), "mlp v");
    // the rows and columns that pad the output layer's copies stay zero
    auto zeroed = [](unsigned char*& d, size_t n, const char* what) {
        return cuda_ok(cudaMalloc(&d, n), what) && cuda_ok(cudaMemsetAsync(d, 0, n, g.stream), what);
    };
    for (int l = 0; l < kLayers && ok; l++) {
        ok = zeroed(M.cp.wk[l], sizeof(__nv_bfloat16) * layer_out_pad(l) * layer_in(l), "mlp wk") &&
             (l == 0 || zeroed(M.cp.wn[l],
                               sizeof(__nv_bfloat16) * (size_t)layer_in(l) * (l == kLayers - 1 ? kDYld : kHid),
                               "mlp wn"));
        if (l == kLayers - 1) continue;
        ok = ok &&
             cuda_ok(cudaMalloc(&M.wpart[l], sizeof(float) * (size_t)kWgradSplits * kHid * layer_in(l)),
                     "mlp weight partial") &&
             cuda_ok(cudaMalloc(&M.bpart[l], sizeof(float) * (size_t)tctrain::kBiasParts * kHid), "mlp bias partial");
    }
    ok = ok && zeroed(M.cp.pack, kPackBytes, "mlp wpack") &&
         cuda_ok(cudaMalloc(&M.opart, sizeof(float) * (size_t)max_blocks() * kOutGrad), "mlp output partial") &&
         cuda_ok(cudaMalloc(&M.freq, sizeof(int) * 3 * kFeat), "mlp freq") &&
         cuda_ok(cudaMalloc(&M.d_mean, sizeof(float) * kOut), "mlp mean") &&
         cuda_ok(cudaMalloc(&M.d_istd, sizeof(float) * kOut), "mlp std") &&
         cuda_ok(cudaMalloc(&M.loss, sizeof(double)), "mlp loss");
    if (!ok) {
        drop(M.p); drop(M.gr); drop(M.m); drop(M.v);
        for (int l = 0; l < kLayers; l++) { drop(M.cp.wk[l]); drop(M.cp.wn[l]); }
        for (int l = 0; l < 4; l++) { drop(M.wpart[l]); drop(M.bpart[l]); }
        drop(M.cp.pack); drop(M.opart); drop(M.freq); drop(M.d_mean); drop(M.d_istd); drop(M.loss);
    }
    M.have_params = ok;
    return ok;
}

static void mlp_drop_batch()
{
    M.cap = 0;
    drop(M.X); drop(M.G0); drop(M.G1); drop(M.dY); drop(M.Y); drop(M.dYf);
    for (int l = 0; l < 4; l++) { drop(M.Z[l]); drop(M.H[l]); }
}

// workspaces for batches of up to n samples (rounded up to a whole 128-row tile);
// none are left when they cannot all be had
static bool mlp_reserve(int n)
{
    if (n > INT_MAX / 128 * 128) {
        set_error(12, "batches of up to %d samples", INT_MAX / 128 * 128);
        return false;
    }
    n = (n + 127) / 128 * 128;
    if (n <= M.cap) return true;
    mlp_drop_batch();
    size_t h = sizeof(__nv_bfloat16) * (size_t)n * kHid;
    bool ok = cuda_ok(cudaMalloc(&M.X, sizeof(__nv_bfloat16) * (size_t)n * kIn), "X") &&
              cuda_ok(cudaMalloc(&M.G0, h), "G0") && cuda_ok(cudaMalloc(&M.G1, h), "G1") &&
              cuda_ok(cudaMalloc(&M.dY, sizeof(__nv_bfloat16) * (size_t)n * kDYld), "dY") &&
              cuda_ok(cudaMalloc(&M.Y, sizeof(float) * (size_t)n * kOut), "Y") &&
              cuda_ok(cudaMalloc(&M.dYf, sizeof(float) * (size_t)n * kOut), "dYf");
    for (int l = 0; l < 4 && ok; l++)
        ok = cuda_ok(cudaMalloc(&M.Z[l], h), "Z") && cuda_ok(cudaMalloc(&M.H[l], h), "H");
    // the padding columns of dY (beyond the 8 that forward_loss writes) stay zero
    if (ok) ok = cuda_ok(cudaMemsetAsync(M.dY, 0, sizeof(__nv_bfloat16) * (size_t)n * kDYld, g.stream), "dY zero");
    if (ok) M.cap = n;
    else mlp_drop_batch();
    return ok;
}

// the BF16 copies and the output normalisation on the device
static bool mlp_refresh()
{
    cudaStream_t s = g.stream;
    copies_kernel<<<(kParams + 255) / 256, 256, 0, s>>>(M.p, M.cp);
    float istd[kOut];
    for (int c = 0; c < kOut; c++) istd[c] = 1.0f / M.out_std[c];
    cudaMemcpyAsync(M.d_mean, M.out_mean, sizeof(float) * kOut, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(M.d_istd, istd, sizeof(float) * kOut, cudaMemcpyHostToDevice, s);
    return cuda_ok(cudaGetLastError(), "weights refresh");
}

// forward of n samples from features X (rows up to the next multiple of 128
// are computed too and ignored): fills Z/H and Y (normalised outputs), on the
// tensor cores
static bool mlp_hidden(int n)
{
    cudaStream_t s = g.stream;
    const int np = (n + 127) / 128 * 128;
    const unsigned char* in = M.X;
    for (int l = 0; l < 4; l++) {
        if (!cuda_ok(tctrain::forward_hidden(in, layer_in(l), M.cp.wk[l], np, M.p + M.boff[l], M.Z[l], M.H[l],
                                             g.d_status, s),
                     "fwd gemm")) return false;
        in = M.H[l];
    }
    return true;
}

static bool mlp_forward(int n)
{
    return mlp_hidden(n) && cuda_ok(tctrain::forward_out(M.H[3], M.cp.wk[4], (n + 127) / 128 * 128, M.p + M.boff[4],
                                                         M.Y, g.d_status, g.stream),
                                    "out gemm");
}

// the same for a multiple of 128 samples with targets T: the loss gradient and,
// with loss_out, the mean loss; Y only with keep_y
static bool mlp_forward_loss(int n, const float* T, bool keep_y, double* loss_out)
{
    cudaStream_t s = g.stream;
    cudaMemsetAsync(M.loss, 0, sizeof(double), s);
    const tctrain::Loss ls = {T, M.d_mean, M.d_istd, M.dY, M.dYf, M.loss};
    if (!mlp_hidden(n) || !cuda_ok(tctrain::forward_loss(M.H[3], M.cp.wk[4], n, M.p + M.boff[4],
                                                         keep_y ? M.Y : nullptr, ls, g.d_status, s),
                                   "out gemm"))
        return false;
    if (loss_out) {
        cudaMemcpyAsync(loss_out, M.loss, sizeof(double), cudaMemcpyDeviceToHost, s);
        if (!cuda_ok(cudaStreamSynchronize(s), "loss")) return false;
        *loss_out /= (double)n * kOut;
    }
    return true;
}

// backward of n samples (a multiple of 128) after mlp_forward_loss: the gradients into M.gr, or, with `step`, one AdamW step from them.
// Data gradients and the hidden layers' weight gradients on the tensor cores;
// bias gradients beside the latter, the output layer's on the CUDA cores.
static bool mlp_backward(int n, const Adam* step)
{
    cudaStream_t s = g.stream;
    const int oblocks = std::min(n / 128, max_blocks());
    out_grad_kernel<<<oblocks, 256, 0, s>>>(M.dYf, M.H[3], n / 128, M.opart);
    // split the samples so that the two 128-row tiles fill the SMs, at least
    // four steps of 64 per split
    const int splits = std::max(1, std::min(kWgradSplits, n / 256));
    const unsigned char* gin = M.dY;
    unsigned char *gcur = M.G0, *gnext = M.G1;
    Partials ps;
    for (int l = 3; l >= 0; l--) {
        if (!cuda_ok(tctrain::backward_data(gin, l == 3 ? kDYld : kHid, M.cp.wn[l + 1], n, M.Z[l], gcur, g.d_status,
                                            s),
                     "dH") ||
            !cuda_ok(tctrain::backward_weights(gcur, l == 0 ? M.X : M.H[l - 1], layer_in(l), n, M.wpart[l], splits,
                                               M.bpart[l], g.d_status, s),
                     "dW"))
            return false;
        ps.w[l] = M.wpart[l];
        ps.b[l] = M.bpart[l];
        gin = gcur;
        std::swap(gcur, gnext);
    }
    ps.out = M.opart;
    ps.splits = tctrain::used_splits(n / 64, splits);
    ps.oblocks = oblocks;
    if (step)
        update_kernel<true><<<kUpdateBlocks, 256, 0, s>>>(ps, nullptr, M.p, M.m, M.v, *step, M.cp);
    else
        update_kernel<false><<<kUpdateBlocks, 256, 0, s>>>(ps, M.gr, nullptr, nullptr, nullptr, Adam{}, M.cp);
    return cuda_ok(cudaGetLastError(), "update");
}

bool mlp::mlp_model(Model& md)
{
    if (!M.ready) {
        set_error(12, "the learned field model is not trained (tp_mlp_train)");
        return false;
    }
    for (int l = 0; l < kLayers; l++) md.b[l] = M.p + M.boff[l];
    md.freq = M.freq;
    md.wpack = M.cp.pack;
    for (int c = 0; c < kOut; c++) {
        md.out_scale[c] = M.out_std[c];
        md.out_shift[c] = M.out_mean[c];
    }
    return true;
}

}  // namespace tp

using namespace tp;

// Initialise the model: frequencies (kFeat x 3 lattice vectors) and weights
// (flat FP32 layout W0, b0, ..., W4, b4 with W_l [out][in]); NULL weights:
// seeded He-uniform initialisation.
extern "C" int tp_mlp_init(const int* freq, const float* weights, unsigned long long seed)
{
    if (!ensure_init() || !mlp_alloc_params()) return -1;
    memcpy(M.freq_h, freq, sizeof(int) * 3 * kFeat);
    cudaMemcpyAsync(M.freq, freq, sizeof(int) * 3 * kFeat, cudaMemcpyHostToDevice, g.stream);
    std::vector<float> h(M.nparam, 0.f);
    if (weights) {
        memcpy(h.data(), weights, sizeof(float) * M.nparam);
    } else {
        uint64_t st = seed * 2654435761ull + 1;
        auto rnd = [&]() {
            st ^= st << 13; st ^= st >> 7; st ^= st << 17;
            return (double)(st >> 11) * (1.0 / 9007199254740992.0);
        };
        for (int l = 0; l < kLayers; l++) {
            double lim = std::sqrt(6.0 / layer_in(l));
            if (l == kLayers - 1) lim *= 0.5;
            for (size_t k = 0; k < (size_t)layer_out(l) * layer_in(l); k++)
                h[M.woff[l] + k] = (float)((2.0 * rnd() - 1.0) * lim);
        }
    }
    cudaMemcpyAsync(M.p, h.data(), sizeof(float) * M.nparam, cudaMemcpyHostToDevice, g.stream);
    cudaMemsetAsync(M.m, 0, sizeof(float) * M.nparam, g.stream);
    cudaMemsetAsync(M.v, 0, sizeof(float) * M.nparam, g.stream);
    M.step = 0;
    M.ready = true;
    return mlp_refresh() && cuda_ok(cudaStreamSynchronize(g.stream), "mlp init") ? 0 : -1;
}

extern "C" int tp_mlp_param_count(void)
{
    int n = 0;
    for (int l = 0; l < kLayers; l++) n += layer_out(l) * layer_in(l) + layer_out(l);
    return n;
}

extern "C" int tp_mlp_set_output_norm(const float* mean, const float* stdv)
{
    for (int c = 0; c < kOut; c++) {
        M.out_mean[c] = mean[c];
        M.out_std[c] = stdv[c];
    }
    return M.ready && mlp_refresh() ? 0 : -1;
}

extern "C" int tp_mlp_get_weights(float* weights)
{
    if (!M.ready) return -1;
    cudaMemcpyAsync(weights, M.p, sizeof(float) * M.nparam, cudaMemcpyDeviceToHost, g.stream);
    return cuda_ok(cudaStreamSynchronize(g.stream), "get weights") ? 0 : -1;
}

// One forward + backward on given samples (u: n*3 box fractions as 32-bit fixed
// point, t: n*6 targets); returns the loss, the normalised outputs and the FP32
// gradients in the flat parameter layout.  For gradient checks.
extern "C" int tp_mlp_grad(int n, const unsigned int* u, const float* t, double* loss, float* y,
                           float* grads)
{
    if (n < 128 || n % 128) {
        set_error(12, "tp_mlp_grad: n must be a positive multiple of 128");
        return -1;
    }
    if (!M.ready || !mlp_reserve(n)) return -1;
    cudaStream_t s = g.stream;
    uint32_t* dU;
    float* dT;
    if (!cuda_ok(cudaMalloc(&dU, sizeof(uint32_t) * 3 * n), "u") ||
        !cuda_ok(cudaMalloc(&dT, sizeof(float) * 6 * n), "t")) return -1;
    cudaMemcpyAsync(dU, u, sizeof(uint32_t) * 3 * n, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(dT, t, sizeof(float) * 6 * n, cudaMemcpyHostToDevice, s);
    features_kernel<<<(n + 127) / 128, 128, 0, s>>>(dU, n, M.freq, M.X);
    bool ok = mlp_forward_loss(n, dT, true, loss) && mlp_backward(n, nullptr);
    if (ok) {
        if (y) cudaMemcpyAsync(y, M.Y, sizeof(float) * 6 * n, cudaMemcpyDeviceToHost, s);
        if (grads) cudaMemcpyAsync(grads, M.gr, sizeof(float) * M.nparam, cudaMemcpyDeviceToHost, s);
        ok = cuda_ok(cudaStreamSynchronize(s), "grad");
    }
    cudaFree(dU);
    cudaFree(dT);
    return ok ? 0 : -1;
}

// Train on nsamples field samples of the current mode table (tp_set_modes),
// drawn uniformly in the box from `seed` and evaluated with the FP64 mode sum.
// Output normalisation comes from the samples.  lr: peak AdamW rate with a
// cosine decay over epochs * (nsamples / batch) steps.  Returns the final
// mean loss (normalised units) in *loss_out and the device time in *ms_out.
extern "C" int tp_mlp_train(long long nsamples, int batch, int epochs, double lr, double wd,
                            unsigned long long seed, double* loss_out, double* ms_out)
{
    if (!M.ready) {
        set_error(12, "tp_mlp_init first");
        return -1;
    }
    if (g.modes.empty()) {
        set_error(12, "no mode table to learn (tp_set_modes)");
        return -1;
    }
    if (batch < 128 || batch % 128 || nsamples < batch) {
        set_error(12, "batch must be a positive multiple of 128 not above nsamples");
        return -1;
    }
    cudaStream_t s = g.stream;
    DevField f;
    if (!build_field(TP_SYS_MODESUM, f) || !mlp_reserve(batch)) return -1;
    uint32_t* dU = nullptr;
    float* dT = nullptr;
    if (!cuda_ok(cudaMalloc(&dU, sizeof(uint32_t) * 3 * (size_t)nsamples), "train u") ||
        !cuda_ok(cudaMalloc(&dT, sizeof(float) * 6 * (size_t)nsamples), "train t")) return -1;
    for (long long off = 0; off < nsamples; off += 1 << 22) {
        int cnt = (int)std::min<long long>(1 << 22, nsamples - off);
        samples_kernel<<<(cnt + 127) / 128, 128, 0, s>>>(seed, off, cnt, f, dU + 3 * off, dT + 6 * off);
    }
    // output normalisation from the training targets
    {
        const int cnt = (int)std::min<long long>(nsamples, 1 << 20);
        const int blocks = std::min((cnt + 127) / 128, max_blocks());
        static_assert(2 * sizeof(double) * kOut <= sizeof(float) * kOutGrad, "the moments fit a block's partial gradients");
        double* part = reinterpret_cast<double*>(M.opart);
        std::vector<double> hp((size_t)blocks * 2 * kOut);
        moments_kernel<<<blocks, 128, 0, s>>>(dT, cnt, part);
        cudaMemcpyAsync(hp.data(), part, sizeof(double) * hp.size(), cudaMemcpyDeviceToHost, s);
        if (!cuda_ok(cudaStreamSynchronize(s), "samples")) return -1;
        for (int c = 0; c < kOut; c++) {
            double a = 0, b = 0;
            for (int k = 0; k < blocks; k++) {
                a += hp[(size_t)k * 2 * kOut + c];
                b += hp[(size_t)k * 2 * kOut + kOut + c];
            }
            a /= cnt;
            double var = b / cnt - a * a;
            M.out_mean[c] = (float)a;
            M.out_std[c] = (float)std::sqrt(var > 1e-30 ? var : 1e-30);
        }
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    long long nb = nsamples / batch;
    long long total = nb * epochs;
    double loss = 0.0;
    bool ok = mlp_refresh();
    for (long long it = 0; it < total && ok; it++) {
        long long bi = it % nb;
        features_kernel<<<(batch + 127) / 128, 128, 0, s>>>(dU + 3 * bi * batch, batch, M.freq, M.X);
        const bool last = it == total - 1;
        const long step = M.step + 1;
        Adam a;
        double frac = (double)it / (double)total;
        a.lr = (float)(lr * 0.5 * (1.0 + std::cos(M_PI * frac)));
        a.b1 = 0.9f;
        a.b2 = 0.999f;
        a.eps = 1e-8f;
        a.wd = (float)wd;
        a.c1 = (float)(1.0 / (1.0 - std::pow(0.9, (double)step)));
        a.c2 = (float)(1.0 / (1.0 - std::pow(0.999, (double)step)));
        ok = mlp_forward_loss(batch, dT + 6 * bi * batch, false, last ? &loss : nullptr) && mlp_backward(batch, &a);
        if (ok) M.step = step;
    }
    cudaEventRecord(e1, s);
    ok = ok && cuda_ok(cudaStreamSynchronize(s), "train");
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(dU);
    cudaFree(dT);
    if (loss_out) *loss_out = loss;
    if (ms_out) *ms_out = ms;
    return ok ? 0 : -1;
}

// Model field at n positions (u: n*3 32-bit fixed point) through the training
// forward pass; out: n*6 physical components.
extern "C" int tp_mlp_eval(int n, const unsigned int* u, float* out)
{
    if (n <= 0) return 0;
    if (!M.ready || !mlp_reserve(n < 128 ? 128 : n)) return -1;
    cudaStream_t s = g.stream;
    uint32_t* dU;
    if (!cuda_ok(cudaMalloc(&dU, sizeof(uint32_t) * 3 * n), "u")) return -1;
    cudaMemcpyAsync(dU, u, sizeof(uint32_t) * 3 * n, cudaMemcpyHostToDevice, s);
    features_kernel<<<(n + 127) / 128, 128, 0, s>>>(dU, n, M.freq, M.X);
    bool ok = mlp_forward(n);
    std::vector<float> y(6 * (size_t)n);
    if (ok) {
        cudaMemcpyAsync(y.data(), M.Y, sizeof(float) * 6 * n, cudaMemcpyDeviceToHost, s);
        ok = cuda_ok(cudaStreamSynchronize(s), "eval");
    }
    cudaFree(dU);
    if (!ok) return -1;
    for (int i = 0; i < n; i++)
        for (int c = 0; c < kOut; c++) out[6 * i + c] = y[6 * i + c] * M.out_std[c] + M.out_mean[c];
    return 0;
}
