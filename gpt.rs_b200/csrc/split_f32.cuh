// f32 matmul on the tcgen05 tensor cores (split_f32.cu), called by dense_f32.cu for more than a few rows.
#pragma once
#include "matmul_common.cuh"

namespace gptrs {

struct SplitF32Params {
    const float* x;         // [M][K], rows ldx apart
    const float* w;         // [K][N]
    const float* bias;      // optional [N]
    const float* residual;  // optional [M][N]
    float* y;               // [M][N], rows ldy apart
    int M, N, K;
    int act;                // 1: gelu (erf)
    DenseAct dense;
    int64_t ldx, ldy, x_step, y_step;   // steps between the entries of a batch; their weights follow each other
    int batch;
    int* status;            // code 3: a bounded wait gave up
    bool w_constant;        // no kernel in front writes w: its first stages may be read before that kernel has ended (a template: a branch cost 2 %)
    int m_tiles, n_split;   // set by the launcher
    uint32_t spin_limit;
    int debug_starve;       // test switch: the first stage's products are never begun
};

// Least rows, the line against the kernel for few rows, and whether it takes this shape (the rule stands at the definitions).
constexpr int kSplitF32Rows = 24;
bool split_f32_line(int64_t m, int64_t n, int64_t k);
bool split_f32_takes(const SplitF32Params& p);
int split_f32_matmul(SplitF32Params p, cudaStream_t st);

}  // namespace gptrs
