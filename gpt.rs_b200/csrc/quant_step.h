// Single-kernel decode step of a few sequences of a quantised Ministral-style model (quant_step.cu).
#pragma once

#include "common.cuh"

namespace gptrs {

struct QuantStepLayer {
    const unsigned char *w_qkv, *w_out, *w_gate_up, *w_down;   // packed weights, layout A in front
    const float *ln1, *ln2;
};

constexpr int kStepMaxLayers = 64, kStepMaxRows = 8;

// Byte offsets of what the CTAs exchange (buffers of {value, flag} words), and of a CTA's shared memory.
struct StepExchange { uint32_t x_in, x_mid, qkv, attn, mlp, ss_in, ss_mid, part, best, total; };
struct StepSmem { uint32_t x, zero, slots, qkv, h, inv, tiles, ranges, spans, best, bars, ring, total; };

struct QuantStepParams {
    QuantStepLayer layers[kStepMaxLayers];   // in the kernel parameters themselves (constant bank)
    int n_layers, rows;                      // rows: sequences of the step, in slots that are distinct
    int D, FF, Hq, Hkv, vocab;
    const float *tok_emb, *final_gain, *cos_table, *sin_table;   // rotary tables [positions][64]
    const unsigned char* w_head;
    int *token, *pos, *ctx;                                      // [rows]; ctx: visible tokens with the new one
    const int *slot, *page_table;
    int given, advance, context_length;                          // given: the ids are token_in. advance: as the kernel of that name does for the other steps
    int token_in[kStepMaxRows];
    int *history, *out;                                          // [slots][context_length]; [rows] in pinned memory
    int max_pages, max_len;                                      // lengths above max_len are clamped to it and flagged
    unsigned char* pool;                                         // KV pool of layer 0
    size_t pool_layer_bytes;
    unsigned char* exchange;                                     // what CTAs hand to each other (quant_step_exchange_bytes), zeros before the first step
    uint32_t epoch;                                              // flags of this step are epoch + 1 ... epoch + n_layers
    float* logits;                                               // [rows][vocab]
    int *sampled, *status;
    float eps, scale_log2;
    // set by the launcher
    int splits, stages;
    uint32_t ring_polls, flag_polls;   // of a wait for weights; of a thread for words, over the whole step
    int starve;                        // test switch, 1: the first tile of the first projection is handed over with an old flag; 2: every CTA's last warp, which has a unit if any has, gets no weights
    StepExchange ex;
    StepSmem sm;
};

// Most sequences of a step of this shape on this device, 0: the shape is not taken.
int quant_step_max_rows(int bits, int n_layers, int D, int FF, int Hq, int Hkv, int vocab);
// Whether a step of these lengths (the longest, all together) is faster as one kernel.
bool quant_step_pays(int bits, int rows, int n_q_heads, int n_kv_heads, int max_ctx, int64_t all_ctx);
size_t quant_step_exchange_bytes(int D, int FF, int Hq, int Hkv);
// max_ctx: the longest visible length of the step's sequences (sizes the splits of attention).
int quant_step_launch(int bits, QuantStepParams p, int max_ctx, cudaStream_t st);

}  // namespace gptrs
