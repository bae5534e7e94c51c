// One decode step of up to eight sequences of a GPT-2-style f32 model as a single cooperative kernel:
// Gpt::forward_with_decode_cache for a one-token chunk (crates/gpt-rs/src/model/gpt.rs:585-751; block order of
// GptBlock::forward_with_decode_cache, gpt.rs:81-97: ln_1 -> qkv -> attention over the cache -> out projection + residual
// -> ln_2 -> MLP in + GELU -> MLP out + residual), final LayerNorm, lm_head and the greedy pick.
//
// Why one kernel: at one row every projection is a 2-9 MB weight stream that takes about a microsecond of HBM time and
// 6-9 us as a launch of its own (launch, first DRAM round trip, barrier, reduction); 64 launches per token left the step
// at 0.13 of its weight-stream roofline. Here the CTAs stay (one per SM, all co-resident: the launch is cooperative), and what crosses from
// phase to phase are short vectors of {value, flag} words in global memory (flag_words.cuh):
//   * every CTA keeps the residual stream (d_model floats per sequence) in its own shared memory and updates it redundantly, so
//     the LayerNorms need no exchange at all,
//   * a projection is a set of items (output row, K chunk of 768) dealt round-robin to all warps of the grid;
//     weights are read from transposed copies [out][in] (built once at finalize), so a warp streams one contiguous row
//     segment with 16-byte loads, multiplies it with the rows of all sequences and reduces with shuffles. Rows whose K is split
//     leave per-chunk partial sums that the next phase adds up in a fixed order (no atomics: results are reproducible); the grid is
//     a multiple of the four chunks, so a CTA meets one chunk of the MLP hidden only,
//   * attention: CTA (sequence, head, context chunk) computes scores, a local softmax and a partial (max, sum, context) over its
//     slice of the cache; the CTA whose slice holds the new position takes K/V of the token from the qkv vector and stores
//     them into the cache; the CTA of the first chunk adds the others' parts,
//   * a context is cut into chunks of 64 keys and more: a short one leaves nothing to merge,
//   * every phase of every layer goes through one copy of the code: with a copy per projection (103 KB at one row, 201 KB at eight) the phases
//     ran from a cold instruction cache.
// A buffer is written again a layer later: a CTA that gets that far has consumed outputs of all CTAs (every phase's vector has items of every
// CTA), and these were computed after their readings. With grid barriers in place of the words, partials of 12 chunks merged by every CTA and a
// copy of the code per projection a token took 326 us (one sequence), 517 (six sequences); now 240 and 369: a phase's exchange is 2.5 to 3.2 us, of
// which the round trips alone are 1.3, its projection 0.7 to 1.0, attention 4.4, the head 20. Every wait is bounded (a thread that gives up records status 5 and goes on).
#include <algorithm>

#include "flag_words.cuh"
#include "gpt_decode_mega.h"

namespace gptrs {
namespace {

constexpr int kMegaThreads = 256, kMegaWarps = kMegaThreads / 32;
constexpr int kD = 768, kMlp = 3072;   // the widths it is built for (mega_supported)
constexpr int kEarlyV = 16;            // values of a thread that attention asks for early: 64 keys of heads of 64

__device__ __forceinline__ float4 ldg_stream_f4(const float4* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
    return t;
}
__device__ __forceinline__ float block_sum(float v, float* red) {
    v = warp_sum(v);
    __syncthreads();   // red may still be read from the previous use
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kMegaWarps; ++w) t += red[w];
    return t;
}

// h += bias + the PARTS partial sums per element that other CTAs left (part null: h is complete), xn = LayerNorm(h) * gamma + beta, for R
// rows at once: 8 / R warps per row, the row in registers between the two sums.
template <int R, int PARTS>
__device__ __forceinline__ void residual_norm(float* h, float* xn, const unsigned char* part, uint32_t flag, FlagWaiter& wait, int rows,
                                              const float* __restrict__ bias, const float* __restrict__ gamma, const float* __restrict__ beta, float eps,
                                              float* red) {
    constexpr int W = kMegaWarps / R, N = kD / (32 * W);
    const int warp = threadIdx.x >> 5, row = warp / W, first = threadIdx.x - row * W * 32;
    constexpr int G = PARTS == 4 ? (N < 6 ? N : N % 8 ? 6 : 8) : N;   // elements under way at once: the next projection's weights already hold 96 registers
    static_assert(N % G == 0, "whole groups");
    float v[N];
    const unsigned char* const own = part + (size_t)(row * kD + first) * (8 * PARTS);
    const bool adds = part && row < rows;
    // what does not depend on the other CTAs is asked for first (of eight rows a thread has 24 elements: their gains come later)
    constexpr bool kEarly = R < 8;
    float b_in[N], g_in[kEarly ? N : 1], s_in[kEarly ? N : 1];
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const int i = first + j * W * 32;
        b_in[j] = part ? __ldg(bias + i) : 0.f;
        if (kEarly) { g_in[j] = __ldg(gamma + i); s_in[j] = __ldg(beta + i); }
    }
    if (R > 1 && adds) {   // (one row: a warp's whole request is three of these)
        if ((threadIdx.x & 31) == 0) wait.wait_word(own, flag);
        __syncwarp();
    }
#pragma unroll
    for (int j0 = 0; j0 < N; j0 += G) {
#pragma unroll
        for (int j = 0; j < G; ++j) v[j0 + j] = 0.f;
        if (!adds) continue;
        bool found;
        if constexpr (PARTS == 4) {
            FlagWords p[G][2];
#pragma unroll 1
            do {
                found = true;
#pragma unroll
                for (int j = 0; j < G; ++j) { p[j][0] = peek_words(own + (j0 + j) * W * 1024); p[j][1] = peek_words(own + (j0 + j) * W * 1024 + 16); }
#pragma unroll
                for (int j = 0; j < G; ++j) found = found && has_flag(p[j][0], flag) && has_flag(p[j][1], flag);
            } while (!found && wait.again());
#pragma unroll
            for (int j = 0; j < G; ++j) v[j0 + j] = (word_f32(p[j][0].a) + word_f32(p[j][0].b)) + (word_f32(p[j][1].a) + word_f32(p[j][1].b));
        } else {
            uint64_t p[G];
#pragma unroll 1
            do {
                found = true;
#pragma unroll
                for (int j = 0; j < G; ++j) p[j] = peek_word(own + (j0 + j) * W * 256);
#pragma unroll
                for (int j = 0; j < G; ++j) found = found && has_flag(p[j], flag);
            } while (!found && wait.again());
#pragma unroll
            for (int j = 0; j < G; ++j) v[j0 + j] = word_f32(p[j]);
        }
    }
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const int i = first + j * W * 32;
        v[j] = part ? h[row * kD + i] + (b_in[j] + v[j]) : h[row * kD + i];
        s += v[j];
    }
    auto row_sum = [&](float t, float* at) {
        t = warp_sum(t);
        if constexpr (W == 1) return t;
        if ((threadIdx.x & 31) == 0) at[warp] = t;
        __syncthreads();
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < W; ++w) sum += at[row * W + w];
        return sum;
    };
    const float mean = row_sum(s, red) / (float)kD;
    float q = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) { const float c = v[j] - mean; q += c * c; }
    const float inv = 1.f / sqrtf(row_sum(q, red + kMegaWarps) / (float)kD + eps);
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const int e = first + j * W * 32;
        h[row * kD + e] = v[j];
        xn[row * kD + e] = (v[j] - mean) * inv * (kEarly ? g_in[kEarly ? j : 0] : gamma[e]) + (kEarly ? s_in[kEarly ? j : 0] : beta[e]);
    }
    __syncthreads();
}

// The sums over a warp of R values: lane l gets the one of row l / (32 / R).
template <int R>
__device__ __forceinline__ float row_sums(float (&v)[R], int lane) {
    if constexpr (R == 8) {
#pragma unroll
        for (int i = 0; i < 4; ++i) { const bool up = lane & 16; const float send = up ? v[i] : v[i + 4]; v[i] = (up ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, send, 16); }
#pragma unroll
        for (int i = 0; i < 2; ++i) { const bool up = lane & 8; const float send = up ? v[i] : v[i + 2]; v[i] = (up ? v[i + 2] : v[i]) + __shfl_xor_sync(0xffffffffu, send, 8); }
        { const bool up = lane & 4; const float send = up ? v[0] : v[1]; v[0] = (up ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, send, 4); }
    } else if constexpr (R == 4) {
#pragma unroll
        for (int i = 0; i < 2; ++i) { const bool up = lane & 16; const float send = up ? v[i] : v[i + 2]; v[i] = (up ? v[i + 2] : v[i]) + __shfl_xor_sync(0xffffffffu, send, 16); }
        { const bool up = lane & 8; const float send = up ? v[0] : v[1]; v[0] = (up ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, send, 8); }
    } else if constexpr (R == 2) {
        const bool up = lane & 16;
        const float send = up ? v[0] : v[1];
        v[0] = (up ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, send, 16);
    }
    float t = v[0];
#pragma unroll
    for (int o = 16 / R; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

// Items (row, chunk of 768) of y = Wt . x dealt to the warps of the whole grid, U at a time per warp. The raw dot products
// of sequence s go to word out[s][row * n_chunks + chunk], or to the logits; biases are applied by whoever reads them (gelu_bias: bias and GELU here). The loads of a
// warp's FIRST round are a call of their own (gemv_prefetch), made BEFORE the waits of the phase: the weights do not
// depend on what those wait for, so their DRAM latency hides behind them. With logits, the lanes that store also keep the largest
// value of their sequence that they have produced (ties: the smaller row).
constexpr int kF4 = 6;   // float4 per lane per item
constexpr int kU = 4;    // items in flight per warp
struct Round { float4 w[kU][kF4]; float bias[kU]; };   // bias: of the items, where GELU follows

__device__ __forceinline__ void gemv_load(Round& r, const float* __restrict__ Wt, int n_items, int item0, int total, int lane) {
#pragma unroll
    for (int u = 0; u < kU; ++u) {
        const int item = min(item0 + u * total, n_items - 1);   // the tail repeats the last item (its result is dropped)
        const float4* src = reinterpret_cast<const float4*>(Wt + (size_t)item * (kF4 * 128)) + lane;   // row * K + chunk * 768 == item * 768
#pragma unroll
        for (int j = 0; j < kF4; ++j) r.w[u][j] = ldg_stream_f4(src + 32 * j);
    }
}
__device__ __forceinline__ void load_bias(Round& r, const float* __restrict__ bias, int n_items, int item0, int total) {
#pragma unroll
    for (int u = 0; u < kU; ++u) r.bias[u] = __ldg(bias + min(item0 + u * total, n_items - 1));
}
__device__ __forceinline__ void gemv_prefetch(Round& r, const float* __restrict__ Wt, int n_items, const float* __restrict__ gelu_bias) {
    const int total = gridDim.x * kMegaWarps, gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    if (gw < n_items) gemv_load(r, Wt, n_items, gw, total, threadIdx.x & 31);
    if (gw < n_items && gelu_bias) load_bias(r, gelu_bias, n_items, gw, total);
}
template <int R>
__device__ __forceinline__ void gemv_items(Round& r, const float* __restrict__ Wt, int n_items, const float* xs, unsigned char* __restrict__ out, uint32_t flag,
                                           float* __restrict__ logits, int rows, float& best, int& best_i, const float* __restrict__ gelu_bias) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int total = gridDim.x * kMegaWarps, gw = warp * gridDim.x + blockIdx.x;
    const int seq = lane / (32 / R);
    const bool stores = lane % (32 / R) == 0 && seq < rows;
#pragma unroll 1
    for (int item0 = gw; item0 < n_items; item0 += kU * total) {
        if (item0 != gw) {   // the first round is already on its way
            gemv_load(r, Wt, n_items, item0, total, lane);
            if (gelu_bias) load_bias(r, gelu_bias, n_items, item0, total);
        }
        float acc[kU][R];
#pragma unroll
        for (int s = 0; s < R; ++s) {   // a sequence's values are read once for the four items
            const float4* xv = reinterpret_cast<const float4*>(xs + s * kD) + lane;
#pragma unroll
            for (int u = 0; u < kU; ++u) acc[u][s] = 0.f;
#pragma unroll
            for (int j = 0; j < kF4; ++j) {
                const float4 x = xv[32 * j];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    acc[u][s] = fmaf(r.w[u][j].x, x.x, acc[u][s]); acc[u][s] = fmaf(r.w[u][j].y, x.y, acc[u][s]);
                    acc[u][s] = fmaf(r.w[u][j].z, x.z, acc[u][s]); acc[u][s] = fmaf(r.w[u][j].w, x.w, acc[u][s]);
                }
            }
        }
        float sum[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) sum[u] = row_sums<R>(acc[u], lane);
#pragma unroll 1
        for (int u = 0; u < kU; ++u) {
            const int item = item0 + u * total;
            float v = u == 0 ? sum[0] : u == 1 ? sum[1] : u == 2 ? sum[2] : sum[3];
            if (stores && item < n_items) {
                if (gelu_bias) {
                    v += u == 0 ? r.bias[0] : u == 1 ? r.bias[1] : u == 2 ? r.bias[2] : r.bias[3];
                    v = (0.5f * v) * (1.f + erff(v / 1.4142135f));
                }
                if (!logits) {
                    put_word(out + ((size_t)seq * n_items + item) * 8, __float_as_uint(v), flag);
                } else {
                    logits[(size_t)seq * n_items + item] = v;
                    if (v > best || (v == best && item < best_i)) { best = v; best_i = item; }
                }
            }
        }
    }
}

// Context chunks per (sequence, head): as many as the grid has CTAs for.
__host__ __device__ inline int mega_chunks(int grid, int rows, int heads) {
    const int n = grid / (rows * heads);
    return n < 1 ? 1 : n > 32 ? 32 : n;
}
__host__ __device__ inline int mega_scores(int grid, int rows, int heads, int ctx_cap) {
    const int n = mega_chunks(grid, rows, heads);
    return (ctx_cap + n - 1) / n;
}

// Chunks that the context of a sequence of `len` is cut into: 64 keys are one pass of a CTA, so a short context leaves few partial results to merge.
__device__ __forceinline__ int mega_live_chunks(int len, int n_chunks) { return max(1, min(n_chunks, (len + 63) >> 6)); }

// R: rows that the arithmetic is laid out for; p.rows of them are sequences.
template <int R>
__global__ void __launch_bounds__(kMegaThreads, 1) gpt_decode_mega_kernel(const MegaParams p) {
    extern __shared__ __align__(16) float sm[];
    float* h = sm;                     // [R][D] residual streams (every CTA holds its own copy)
    float* xn = h + R * kD;            // [R][D] LayerNorm output / merged attention output
    float* big = xn + R * kD;          // [R][D] this CTA's chunk of the MLP hidden / scores of the attention phase
    float* red = big + p.big_floats;   // [64]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rows = p.rows;
    const int H = p.H, hd = p.hd;
    FlagWaiter wait = {p.flag_polls, p.status};
    int n_time = 0;
    auto stamp = [&]() { if (p.timing && blockIdx.x == 0 && tid == 0) p.timing[n_time++] = global_ns(); };
    stamp();
    float best = -INFINITY;   // lm_head: the largest logit this lane has produced
    int best_i = 0x7fffffff;
    Round rnd;                // the weights of this warp's first items of the next projection
    gemv_prefetch(rnd, p.layers[0].w_qkv_t, 3 * kD, nullptr);
    uint32_t flag = p.epoch;   // of the layer; every phase's vector has a buffer of its own

    for (int s = 0; s < R; ++s) {
        const int token = s < rows ? (p.given ? p.token_in[s] : p.token[s]) : 0;
        const bool ok = s < rows && token >= 0 && token < p.vocab;
        if (s < rows && !ok && tid == 0 && blockIdx.x == 0) atomicExch(p.status, 2);
        const int pos = ok ? min(max(p.pos[s], 0), p.n_pos - 1) : 0;
        for (int i = tid; i < kD; i += kMegaThreads) h[s * kD + i] = ok ? p.tok_emb[(size_t)token * kD + i] + p.pos_emb[(size_t)pos * kD + i] : 0.f;
    }
    __syncthreads();

    // this CTA's part in attention: a slice of the context of one head of one sequence
    const int n_chunks = mega_chunks(gridDim.x, rows, H), n_tasks = rows * H * n_chunks;
    const bool attends = (int)blockIdx.x < n_tasks;
    const int seq = attends ? blockIdx.x / (H * n_chunks) : 0, head = (blockIdx.x / n_chunks) % H, ck = blockIdx.x % n_chunks;
    const int pos = min(max(p.pos[seq], 0), p.ctx_cap - 1), len = pos + 1;
    const int live = mega_live_chunks(len, n_chunks);
    const int chunk_len = (len + live - 1) / live, j0 = min(len, ck * chunk_len), j1 = min(len, j0 + chunk_len);
    const size_t cache_at = ((size_t)p.slot[seq] * H + head) * p.ctx_cap * hd;
    const float scale = 1.0f / sqrtf((float)hd);
    const int part_stride = (hd + 4) * 8;   // context, maximum, sum

#pragma unroll 1
    for (int phase = 0;; ++phase) {
        // phases of a layer: qkv, out projection (attention in front of it), MLP in, MLP out; after the last layer the head
        const int l = phase >> 2, kind = phase & 3;
        const bool at_head = l == p.n_layers;
        const MegaLayer& L = p.layers[at_head ? l - 1 : l];   // the table is part of the kernel parameters: no pointer chase through memory
        const float* xs = xn;
        if (kind == 0) ++flag;
        if (kind == 0) {
            // residual update from the previous block's MLP (four partial sums), ln_1 or the final LayerNorm
            residual_norm<R, 4>(h, xn, l > 0 ? p.pe : nullptr, flag - 1, wait, rows, l > 0 ? p.layers[l - 1].b_mlp_out : nullptr, at_head ? p.lnf_g : L.ln1_g, at_head ? p.lnf_b : L.ln1_b,
                                p.eps, red);
        } else if (kind == 1) {
            // ---- attention: CTA = (sequence, head, context chunk) ---------------------------------------------------------
            if (attends && ck < live) {
                float* kc = L.k_cache + cache_at;
                float* vc = L.v_cache + cache_at;
                // q, and K / V of the new token, from the qkv vector the other CTAs write
                float* qs = xn;            // [hd]
                float* k_new = xn + hd;    // [hd]
                float* v_new = xn + 2 * hd;
                // the first 64 keys and values of the slice are asked for before the token's vectors have arrived
                const int lanes = hd >> 2, per = 32 / lanes, sub = lane / lanes, c4 = (lane - sub * lanes) * 4;
                const int parts = kMegaThreads / hd, c = tid % hd, part = tid / hd;
                float4 k4[4];
                float v_in[kEarlyV];
                auto load_keys = [&](int base) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int j = base + u * kMegaWarps * per + sub;
                        k4[u] = j >= j1 || j == pos ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>(kc + (size_t)j * hd + c4);
                    }
                };
                load_keys(j0 + warp * per);
#pragma unroll
                for (int u = 0; u < kEarlyV; ++u) {
                    const int j = j0 + part + u * parts;
                    v_in[u] = j < j1 && j != pos ? vc[(size_t)j * hd + c] : 0.f;
                }
                const unsigned char* qkv = p.qkv + (size_t)(seq * 3 * kD + head * hd) * 8;
#pragma unroll 1
                for (int i = tid; i < 3 * hd; i += kMegaThreads) {
                    const int which = i / hd, e = i - which * hd;
                    const float bias = L.b_qkv[which * kD + head * hd + e];
                    xn[i] = __uint_as_float(wait.wait_word(qkv + (which * kD + e) * 8, flag)) + bias;
                }
                __syncthreads();
                float* sc = big;   // scores of this slice
                if (j0 <= pos && pos < j1)   // the new token's row goes into the cache for the steps to come
                    for (int i = tid; i < hd; i += kMegaThreads) { kc[(size_t)pos * hd + i] = k_new[i]; vc[(size_t)pos * hd + i] = v_new[i]; }
                // scores: hd / 4 lanes per key, four times 128 / hd keys of a warp under way at once
                {
                    const float4 q4 = *reinterpret_cast<const float4*>(qs + c4), own = *reinterpret_cast<const float4*>(k_new + c4);
#pragma unroll 1
                    for (int base = j0 + warp * per; base < j1; base += 4 * kMegaWarps * per) {
                        if (base != j0 + warp * per) load_keys(base);
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int j = base + u * kMegaWarps * per + sub;
                            const float4 k = j == pos ? own : k4[u];
                            float t = fmaf(q4.w, k.w, fmaf(q4.z, k.z, fmaf(q4.y, k.y, q4.x * k.x)));
#pragma unroll 1
                            for (int o = lanes >> 1; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                            if (c4 == 0 && j < j1) sc[j - j0] = t * scale;
                        }
                    }
                }
                __syncthreads();
                float mx = -INFINITY;
#pragma unroll 1
                for (int j = tid; j < j1 - j0; j += kMegaThreads) mx = fmaxf(mx, sc[j]);
                mx = warp_max(mx);
                if (lane == 0) red[32 + warp] = mx;
                __syncthreads();
                mx = red[32];
#pragma unroll
                for (int w = 1; w < kMegaWarps; ++w) mx = fmaxf(mx, red[32 + w]);
                float sum = 0.f;
#pragma unroll 1
                for (int j = tid; j < j1 - j0; j += kMegaThreads) {
                    const float e = expf(sc[j] - mx);
                    sc[j] = e;
                    sum += e;
                }
                sum = block_sum(sum, red);
                // context: thread (part, c) walks positions part, part + parts, ...
                float acc = 0.f;
#pragma unroll
                for (int u = 0; u < kEarlyV; ++u) {
                    const int j = j0 + part + u * parts;
                    if (j < j1) acc = fmaf(sc[j - j0], j == pos ? v_new[c] : v_in[u], acc);
                }
#pragma unroll 4
                for (int j = j0 + part + kEarlyV * parts; j < j1; j += parts) acc = fmaf(sc[j - j0], (j == pos ? v_new : vc + (size_t)j * hd)[c], acc);
                float* comb = red + 64;   // [parts][hd]
                comb[part * hd + c] = acc;
                __syncthreads();
                float m_all = j1 > j0 ? mx : -INFINITY, l_all = j1 > j0 ? sum : 0.f;
                unsigned char* out = p.att_part + (size_t)blockIdx.x * part_stride;
                if (tid < hd) {
                    float v = 0.f;
#pragma unroll 2
                    for (int q2 = 0; q2 < parts; ++q2) v += comb[q2 * hd + tid];
                    if (ck > 0) {
                        put_word(out + tid * 8, __float_as_uint(v), flag);
                        if (tid == 0) put_words(out + hd * 8, __float_as_uint(m_all), __float_as_uint(l_all), flag);
                    } else {   // the first chunk's CTA adds the others' parts, in order
#pragma unroll 1
                        for (int k0 = 1; k0 < live; k0 += 4) {
                            uint64_t o[4];
                            FlagWords ms[4];
                            bool found;
#pragma unroll 1
                            do {
                                found = true;
#pragma unroll
                                for (int k = 0; k < 4; ++k) {   // past the end: the last one once more
                                    const unsigned char* from = out + (size_t)min(k0 + k, live - 1) * part_stride;
                                    o[k] = peek_word(from + tid * 8);
                                    ms[k] = peek_words(from + hd * 8);
                                }
#pragma unroll
                                for (int k = 0; k < 4; ++k) found = found && has_flag(o[k], flag) && has_flag(ms[k], flag);
                            } while (!found && wait.again());
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const float mk = word_f32(ms[k].a);
                                if (k0 + k >= live || mk == -INFINITY) continue;
                                const float top = fmaxf(m_all, mk), fa = m_all == -INFINITY ? 0.f : expf(m_all - top), fb = expf(mk - top);
                                l_all = fmaf(word_f32(ms[k].b), fb, l_all * fa);
                                v = fmaf(word_f32(o[k]), fb, v * fa);
                                m_all = top;
                            }
                        }
                        put_word(p.att + (size_t)(seq * kD + head * hd + tid) * 8, __float_as_uint(v / l_all), flag);
                    }
                }
                __syncthreads();   // scores, comb and the token's vectors have been read
            }
            stamp();
        } else if (kind == 2) {
            residual_norm<R, 1>(h, xn, p.pc, flag, wait, rows, L.b_out, L.ln2_g, L.ln2_b, p.eps, red);
        }
        if (kind & 1) {   // the attention output, or the 768 values of the MLP hidden that this CTA's items of the last projection need
            constexpr int N = (R * kD / 2 + kMegaThreads - 1) / kMegaThreads;
            const int n2 = rows * (kD / 2);   // pairs of words
            auto word_at = [&](int i) {
                const int s2 = i / (kD / 2), e = i - s2 * (kD / 2);
                return kind == 1 ? p.att + (size_t)i * 16 : p.mh + ((size_t)s2 * kMlp + (blockIdx.x & 3) * kD) * 8 + e * 16;
            };
            if (lane == 0 && tid < n2) wait.wait_word(word_at(tid), flag);
            __syncwarp();
            FlagWords v[N];
            bool found;
#pragma unroll 1
            do {   // past the end: the last pair once more
                found = true;
#pragma unroll
                for (int j = 0; j < N; ++j) v[j] = peek_words(word_at(min(tid + j * kMegaThreads, n2 - 1)));
#pragma unroll
                for (int j = 0; j < N; ++j) found = found && has_flag(v[j], flag);
            } while (!found && wait.again());
#pragma unroll
            for (int j = 0; j < N; ++j)
                if (tid + j * kMegaThreads < n2) reinterpret_cast<float2*>(big)[tid + j * kMegaThreads] = make_float2(word_f32(v[j].a), word_f32(v[j].b));
            __syncthreads();
            xs = big;
        }
        const float* w = at_head ? p.lm_head_t : kind == 0 ? L.w_qkv_t : kind == 1 ? L.w_out_t : kind == 2 ? L.w_mlp_in_t : L.w_mlp_out_t;
        const int n_items = at_head ? p.vocab : kind == 0 ? 3 * kD : kind == 1 ? kD : kMlp;   // MLP out: four chunks of 768 rows
        stamp();
        gemv_items<R>(rnd, w, n_items, xs, kind == 0 ? p.qkv : kind == 1 ? p.pc : kind == 2 ? p.mh : p.pe, flag - (p.starve && phase == 0 && blockIdx.x == 0 ? 1u : 0u), at_head ? p.logits : nullptr, rows, best, best_i,
                      kind == 2 ? L.b_mlp_in : nullptr);
        stamp();
        if (at_head) break;
        __syncthreads();   // xn and big have been read
        const float* next = kind == 0 ? L.w_out_t : kind == 1 ? L.w_mlp_in_t : kind == 2 ? L.w_mlp_out_t : l + 1 < p.n_layers ? p.layers[l + 1].w_qkv_t : p.lm_head_t;
        gemv_prefetch(rnd, next, kind == 0 ? kD : kind < 3 ? kMlp : l + 1 < p.n_layers ? 3 * kD : p.vocab, kind == 1 ? L.b_mlp_in : nullptr);   // of the out projection: kept across attention
    }
    // ---- the greedy pick ------------------------------------------------------------------------------------------------
    // the storing lanes hold their warp's best of a sequence; CTA best -> cand[sequence][blockIdx.x]
    float* bv = big;                                        // [warp][R]
    int* bi = reinterpret_cast<int*>(big + kMegaWarps * R);
    __syncthreads();
    if (lane % (32 / R) == 0) { bv[warp * R + lane / (32 / R)] = best; bi[warp * R + lane / (32 / R)] = best_i; }
    __syncthreads();
    if (tid < rows) {
        for (int w = 1; w < kMegaWarps; ++w)
            if (bv[w * R + tid] > bv[tid] || (bv[w * R + tid] == bv[tid] && bi[w * R + tid] < bi[tid])) { bv[tid] = bv[w * R + tid]; bi[tid] = bi[w * R + tid]; }
        put_words(p.cand + (size_t)(tid * gridDim.x + blockIdx.x) * 16, __float_as_uint(bv[tid]), (uint32_t)bi[tid], flag);
    }
    if (blockIdx.x == 0 && warp < rows) {
        float v = -INFINITY;
        int ix = 0x7fffffff;
#pragma unroll 1
        for (int k = lane; k < (int)gridDim.x; k += 32) {
            const FlagWords w = wait.wait_words(p.cand + (size_t)(warp * gridDim.x + k) * 16, flag);
            const float cv = word_f32(w.a);
            const int ci = (int)(uint32_t)w.b;
            if (cv > v || (cv == v && ci < ix)) { v = cv; ix = ci; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
            if (ov > v || (ov == v && oi < ix)) { v = ov; ix = oi; }
        }
        if (lane == 0 && p.greedy) {
            p.sampled[warp] = ix;
            if (p.advance) {   // every CTA has read its token and position by now: its candidate came behind
                const int at = p.pos[warp];
                if (at >= 0 && at < p.n_pos) p.history[(size_t)warp * p.n_pos + at] = p.given ? p.token_in[warp] : p.token[warp];
                p.token[warp] = ix;
                p.pos[warp] = at + 1;
                p.ctx[warp] += 1;
                p.out[warp] = ix;
            }
        }
    }
}

struct TransposeParams { const float* src; float* dst; int rows, cols; };
// dst[c][r] = src[r][c], 32 x 32 tiles through shared memory
__global__ void transpose_kernel(const TransposeParams p) {
    __shared__ float tile[32][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int i = threadIdx.y; i < 32; i += 8) {
        const int r = r0 + i, c = c0 + threadIdx.x;
        if (r < p.rows && c < p.cols) tile[i][threadIdx.x] = p.src[(size_t)r * p.cols + c];
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += 8) {
        const int c = c0 + i, r = r0 + threadIdx.x;
        if (r < p.rows && c < p.cols) p.dst[(size_t)c * p.rows + r] = tile[threadIdx.x][i];
    }
}

}  // namespace

int mega_transpose(const float* src_in_out, float* dst_out_in, int64_t in, int64_t out, cudaStream_t st) {
    TransposeParams p = {src_in_out, dst_out_in, (int)in, (int)out};
    transpose_kernel<<<dim3((unsigned)((out + 31) / 32), (unsigned)((in + 31) / 32)), dim3(32, 8), 0, st>>>(p);
    GPTRS_CUDA_OK(cudaGetLastError());
    return GPTRS_OK;
}

bool mega_supported(int D, int H, int hd, int MLP, int ctx_cap, int n_layers) {
    // every item is a 768-float row segment: d_model-wide rows in one piece, MLP out in four chunks that the consumer adds
    return D == kD && H * hd == D && (hd == 32 || hd == 64 || hd == 128) && MLP == kMlp && sm_count() % 4 == 0 && ctx_cap >= 1 && n_layers >= 1 &&
           n_layers <= kMegaMaxLayers && mega_max_rows(H, hd, ctx_cap) >= 1;
}

namespace {
size_t mega_big_floats(int layout, int rows, int H, int ctx_cap) {
    const size_t scores = (size_t)(mega_scores(sm_count(), rows, H, ctx_cap) + 3) / 4 * 4, hidden = (size_t)layout * kD;
    return scores > hidden ? scores : hidden;
}
size_t mega_smem_bytes(int layout, int rows, int H, int hd, int ctx_cap) {
    (void)hd;
    return (2 * (size_t)layout * kD + mega_big_floats(layout, rows, H, ctx_cap) + 64 + std::max(kMegaThreads, 2 * sm_count()) + 64) * sizeof(float);
}
int mega_layout(int rows) { return rows <= 1 ? 1 : rows <= 2 ? 2 : rows <= 4 ? 4 : 8; }
constexpr size_t kMegaSmem = 227 * 1024;
}  // namespace

int mega_max_rows(int H, int hd, int ctx_cap) {
    int n = 0;
    while (n < kMegaMaxRows && (n + 1) * H <= sm_count() && mega_smem_bytes(mega_layout(n + 1), n + 1, H, hd, ctx_cap) <= kMegaSmem) ++n;
    return n;
}

int mega_launch(MegaParams p, cudaStream_t st) {
    void (*kerns[4])(MegaParams) = {gpt_decode_mega_kernel<1>, gpt_decode_mega_kernel<2>, gpt_decode_mega_kernel<4>, gpt_decode_mega_kernel<8>};
    static PerDeviceOnce attr_once;
    if (attr_once.first_time())
        for (auto k : kerns) GPTRS_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMegaSmem));
    const int layout = mega_layout(p.rows);
    p.big_floats = (int)mega_big_floats(layout, p.rows, p.H, p.ctx_cap);
    uint32_t barrier_polls;
    step_wait_limits(&barrier_polls, &p.flag_polls, &p.starve);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)sm_count());
    cfg.blockDim = dim3(kMegaThreads);
    cfg.dynamicSmemBytes = mega_smem_bytes(layout, p.rows, p.H, p.hd, p.ctx_cap);
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeCooperative;   // all CTAs co-resident: they wait for each other's words
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kerns[layout == 1 ? 0 : layout == 2 ? 1 : layout == 4 ? 2 : 3], p);
    if (e != cudaSuccess) return fail(GPTRS_EXECUTION, std::string("cooperative launch failed: ") + cudaGetErrorString(e));
    return GPTRS_OK;
}

}  // namespace gptrs
