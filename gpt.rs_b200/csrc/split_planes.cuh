// f32 matmul on the tcgen05 tensor cores from operands that are three bf16 planes in memory already (split_planes.cu).
#pragma once
#include "common.cuh"

namespace gptrs {

// The planes of a matrix [rows][K] (K a multiple of 64): first [rows][K / 32][32 of plane 1, 32 of plane 2], behind them [rows][K] of plane 3.
inline size_t plane_bytes(int64_t rows, int64_t k) { return (size_t)rows * k * 6; }

int split_weight_planes(const float* w, void* planes, int64_t k, int64_t n, cudaStream_t st);   // of the transpose of w [K][N]
int split_row_planes(const float* x, void* planes, int64_t m, int64_t k, cudaStream_t st);      // of x [M][K]

struct PlanesMatmul {
    const void *w_planes, *x_planes;
    const float *x, *w;         // the operands themselves, [M][K] and [K][N]: sums that are not finite are computed again from them
    const float* bias;          // optional [N]
    const float* residual;      // optional [M][N]
    float* y;                   // [M][N]
    void* y_planes;             // optional: the planes of y, too
    int M, N, K;
    int act;                    // 1: gelu (erf)
    int* status;                // code 3: a bounded wait gave up
};
int planes_matmul(const PlanesMatmul& p, cudaStream_t st);

// LayerNorm (beta may be null) or RMSNorm of rows [rows][k] into y and its planes, for the k that norm_planes_takes says.
bool norm_planes_takes(int64_t k);
int norm_planes(const float* x, const float* gamma, const float* beta, float eps, bool layer_norm, float* y, void* planes, int64_t rows, int64_t k, cudaStream_t st);

}  // namespace gptrs
