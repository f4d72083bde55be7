// tc_train.cuh -- host launchers of the tensor-core training GEMMs (tc_train.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "tc_sm100.cuh"

namespace tp {
namespace tctrain {

// Byte offset of element (m, c) of a matrix of samples [M][64 atoms] in BF16: 16 KB
// blocks of 128 samples x 64 columns, swizzled rows of 128 bytes (M a multiple of 128).
__host__ __device__ __forceinline__ size_t tile_offset(size_t m, int c, int atoms)
{
    return (m >> 7) * (size_t)atoms * 16384u + tc::sw128_offset(128, (int)(m & 127), c);
}

// Weights are k-atoms of all rows: element (n, k) of [N][K] at sw128_offset(N, n, k).

// Blocks of a layer kernel over M samples.
int layer_blocks(int M);

// Z, H = silu(X W^T + b) of a hidden layer: X [M][kin], W [256][kin]; Z, H [M][256].
// M a multiple of 128.
cudaError_t forward_hidden(const void* X, int kin, const void* W, int M, const float* b, void* Z, void* H,
                           int* status, cudaStream_t s);

// Y = H3 W4^T + b: H3 [M][256], W4 [16][256] (rows past the 6 outputs zero); Y FP32 [M][6], row-major.
cudaError_t forward_out(const void* H3, const void* W4, int M, const float* b, float* Y, int* status,
                        cudaStream_t s);

// The same with the loss of M samples against the targets T [M][6]: the gradient dYf
// (FP32 rows) and dY (BF16 blocks of 64 columns, of which the first 8 are written), the
// sum of the squares added to *sum; Y may be null.
struct Loss {
    const float *T, *mean, *istd;
    unsigned char* dY;
    float* dYf;
    double* sum;
};
cudaError_t forward_loss(const void* H3, const void* W4, int M, const float* b, float* Y, const Loss& ls, int* status,
                         cudaStream_t s);

// G = (Gin WT^T) * silu'(Zprev): Gin [M][kout], WT [256][kout] (the layer's weights
// transposed); G [M][256].
cudaError_t backward_data(const void* Gin, int kout, const void* WT, int M, const void* Zprev, void* G,
                          int* status, cudaStream_t s);

// The gradient G^T X [256][kin] over nsamp samples, G [nsamp][256], X [nsamp][kin],
// as used_splits(nsamp / 64, splits) partial sums (splits at most nsamp / 64), each over
// the next nsamp / 64 / splits, rounded up, steps of 64 samples: P[split][m / 128][k][m % 128].
// G's column sums as kBiasParts partial sums in bpart [kBiasParts][256].
constexpr int kBiasParts = 8;
int used_splits(int nsteps, int splits);
cudaError_t backward_weights(const void* G, const void* X, int kin, int nsamp, float* P, int splits,
                             float* bpart, int* status, cudaStream_t s);

}  // namespace tctrain
}  // namespace tp
