// Single-kernel decode step of up to eight sequences of a GPT-2-style f32 model (gpt_decode_mega.cu).
#pragma once

#include "common.cuh"

namespace gptrs {

struct MegaLayer {
    const float *ln1_g, *ln1_b, *w_qkv_t, *b_qkv, *w_out_t, *b_out, *ln2_g, *ln2_b, *w_mlp_in_t, *b_mlp_in, *w_mlp_out_t, *b_mlp_out;
    float *k_cache, *v_cache;   // [slot][head][capacity][head_dim] of this layer
};

constexpr int kMegaMaxLayers = 16, kMegaMaxRows = 8;

struct MegaParams {
    MegaLayer layers[kMegaMaxLayers];   // in the kernel parameters themselves (constant bank)
    int n_layers;
    const float *tok_emb, *pos_emb, *lnf_g, *lnf_b, *lm_head_t;
    int rows;                        // sequences of the step
    int *token, *pos, *ctx;          // [rows]
    const int* slot;                 // [rows], distinct
    int given, advance;              // given: the ids are token_in. advance: as the kernel of that name does for the other steps (the slots are 0 ... rows - 1)
    int token_in[kMegaMaxRows];
    int *history, *out;              // [slots][n_pos]; [rows] in pinned memory
    unsigned char *qkv, *att_part, *att, *pc, *mh, *pe, *cand;   // {value, flag} words: vectors of kMegaMaxRows rows, partials and candidates per CTA
    uint32_t epoch;                  // flags of this step are epoch + 1 ... epoch + n_layers + 1
    float* logits;                   // [rows][vocab]
    int* sampled;
    int* status;
    unsigned long long* timing;   // optional (GPTRS_MEGA_TIMING=1): globaltimer of CTA 0 at kernel start, where its part in attention has ended, and around every projection
    int H, hd, vocab, ctx_cap, n_pos;
    int big_floats;                  // set by the launcher
    uint32_t flag_polls;             // of a thread, over the whole step; set by the launcher, too
    int starve;                      // test switch: the first CTA hands its part of the first projection over with an old flag
    float eps;
    int greedy;
};

bool mega_supported(int D, int H, int hd, int MLP, int ctx_cap, int n_layers);
int mega_max_rows(int H, int hd, int ctx_cap);   // most sequences of a step
int mega_transpose(const float* src_in_out, float* dst_out_in, int64_t in, int64_t out, cudaStream_t st);
int mega_launch(MegaParams p, cudaStream_t st);

}  // namespace gptrs
