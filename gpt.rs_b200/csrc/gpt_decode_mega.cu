// One decode step of up to eight sequences of a GPT-2-style f32 model as a single cooperative kernel:
// Gpt::forward_with_decode_cache for a one-token chunk (crates/gpt-rs/src/model/gpt.rs:585-751; block order of
// GptBlock::forward_with_decode_cache, gpt.rs:81-97: ln_1 -> qkv -> attention over the cache -> out projection + residual
// -> ln_2 -> MLP in + GELU -> MLP out + residual), final LayerNorm, lm_head and the greedy pick.
//
// Why one kernel: at one row every projection is a 2-9 MB weight stream that takes about a microsecond of HBM time and
// 6-9 us as a launch of its own (launch, first DRAM round trip, barrier, reduction); 64 launches per token left the step
// at 0.13 of its weight-stream roofline. Here the launch boundary becomes a grid-wide barrier (one CTA per SM, all
// co-resident: the launch is cooperative), and what crosses a barrier is a short vector in global memory:
//   * every CTA keeps the residual stream (d_model floats per sequence) in its own shared memory and updates it redundantly, so
//     the LayerNorms need no exchange at all,
//   * a projection is a set of items (output row, K chunk of 768) dealt round-robin to all warps of the grid;
//     weights are read from transposed copies [out][in] (built once at finalize), so a warp streams one contiguous row
//     segment with 16-byte loads, multiplies it with the rows of all sequences and reduces with shuffles. Rows whose K is split
//     leave per-chunk partial sums that the next phase adds up in a fixed order (no atomics: results are reproducible); the grid is
//     a multiple of the four chunks, so a CTA meets one chunk of the MLP hidden only,
//   * attention: CTA (sequence, head, context chunk) computes scores, a local softmax and a partial (max, sum, context) over its
//     slice of the cache; the CTA whose slice holds the new position takes K/V of the token from the qkv vector and stores
//     them into the cache; every CTA merges the partials of all heads when it stages the input of the out projection.
// 5 barriers per layer + 1. Every barrier wait is bounded (a CTA that gives up records status 5 and goes on).
#include "gpt_decode_mega.h"

namespace gptrs {
namespace {

constexpr int kMegaThreads = 256, kMegaWarps = kMegaThreads / 32;
constexpr uint32_t kMegaSpin = 1u << 24;
constexpr int kD = 768, kMlp = 3072;   // the widths it is built for (mega_supported)

struct BarrierState { unsigned* ctr; unsigned target; unsigned step; int* status; unsigned long long* timing; int n; };

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
// A grid barrier in two halves, so that the loads of the next projection's weights can be issued BETWEEN them: issued
// before the arrival they would sit in front of its fence (a fence waits for the thread's outstanding loads too: the
// prefetch would delay every arrival by a DRAM round trip), issued after the wait they would hide nothing.
__device__ __forceinline__ void grid_arrive(BarrierState& b) {
    b.target += b.step;
    __syncthreads();
    if (b.timing && blockIdx.x == 0 && threadIdx.x == 0) b.timing[b.n++] = global_ns();   // arrival of CTA 0
    if (threadIdx.x == 0) {
        __threadfence();
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(b.ctr) : "memory");
    }
}
__device__ __forceinline__ void grid_wait(BarrierState& b) {
    if (threadIdx.x == 0) {
        unsigned v = 0;
        uint32_t it = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(b.ctr) : "memory");
        } while (v < b.target && ++it < kMegaSpin);
        if (v < b.target) atomicExch(b.status, 5);
        if (b.timing && blockIdx.x == 0) b.timing[b.n++] = global_ns();   // release of CTA 0
    }
    __syncthreads();
}
__device__ __forceinline__ void grid_barrier(BarrierState& b) {
    grid_arrive(b);
    grid_wait(b);
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

// h += bias + the PARTS partial sums per element that other CTAs left (PARTS 0: h is complete), xn = LayerNorm(h) * gamma + beta, for R
// rows at once: 8 / R warps per row, the row in registers between the two sums.
template <int R, int PARTS>
__device__ __forceinline__ void residual_norm(float* h, float* xn, const float* part, const float* __restrict__ bias, const float* __restrict__ gamma,
                                              const float* __restrict__ beta, float eps, float* red) {
    constexpr int W = kMegaWarps / R, N = kD / (32 * W);
    const int warp = threadIdx.x >> 5, row = warp / W, first = threadIdx.x - row * W * 32;
    constexpr int G = N < 6 ? N : 6;   // loads under way at once: the next projection's weights already hold 96 registers
    float v[N];
#pragma unroll
    for (int j0 = 0; j0 < N; j0 += G) {
        if constexpr (PARTS == 4) {
            float4 p4[G];
#pragma unroll
            for (int j = 0; j < G; ++j) p4[j] = __ldcg(reinterpret_cast<const float4*>(part) + row * kD + first + (j0 + j) * W * 32);
#pragma unroll
            for (int j = 0; j < G; ++j) v[j0 + j] = (p4[j].x + p4[j].y) + (p4[j].z + p4[j].w);
        } else if constexpr (PARTS == 1) {
#pragma unroll
            for (int j = 0; j < G; ++j) v[j0 + j] = __ldcg(part + row * kD + first + (j0 + j) * W * 32);
        }
    }
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const int i = first + j * W * 32;
        v[j] = PARTS ? h[row * kD + i] + (bias[i] + v[j]) : h[row * kD + i];
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
        xn[row * kD + e] = (v[j] - mean) * inv * gamma[e] + beta[e];
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
// of sequence s go to out[s][row * n_chunks + chunk]; biases are applied by whoever reads them (kGelu: bias and GELU here). The loads of a warp's FIRST
// round are a call of their own (gemv_prefetch), made BEFORE the grid barrier in front of the phase: the weights do not
// depend on what the barrier waits for, so their DRAM latency hides behind it. With kBest, the lanes that store also keep the largest
// value of their sequence that they have produced (ties: the smaller row).
constexpr int kF4 = 6;   // float4 per lane per item
constexpr int kU = 4;    // items in flight per warp
struct Round { float4 w[kU][kF4]; };

__device__ __forceinline__ void gemv_load(Round& r, const float* __restrict__ Wt, int n_items, int item0, int total, int lane) {
#pragma unroll
    for (int u = 0; u < kU; ++u) {
        const int item = min(item0 + u * total, n_items - 1);   // the tail repeats the last item (its result is dropped)
        const float4* src = reinterpret_cast<const float4*>(Wt + (size_t)item * (kF4 * 128)) + lane;   // row * K + chunk * 768 == item * 768
#pragma unroll
        for (int j = 0; j < kF4; ++j) r.w[u][j] = ldg_stream_f4(src + 32 * j);
    }
}
__device__ __forceinline__ void gemv_prefetch(Round& r, const float* __restrict__ Wt, int n_rows, int K) {
    const int total = gridDim.x * kMegaWarps, gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const int n_items = n_rows * (K / (kF4 * 128));
    if (gw < n_items) gemv_load(r, Wt, n_items, gw, total, threadIdx.x & 31);
}
template <int R, bool kBest, bool kGelu = false>
__device__ __forceinline__ void gemv_items(Round& r, const float* __restrict__ Wt, int n_items, const float* xs, float* __restrict__ out, int rows,
                                           float& best, int& best_i, const float* __restrict__ bias = nullptr) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int total = gridDim.x * kMegaWarps, gw = warp * gridDim.x + blockIdx.x;
    const int seq = lane / (32 / R);
    const bool stores = lane % (32 / R) == 0 && seq < rows;
#pragma unroll 1
    for (int item0 = gw; item0 < n_items; item0 += kU * total) {
        if (item0 != gw) gemv_load(r, Wt, n_items, item0, total, lane);   // the first round is already on its way
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
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int item = item0 + u * total;
            float v = row_sums<R>(acc[u], lane);
            if (stores && item < n_items) {
                if constexpr (kGelu) {
                    v += bias[item];
                    v = (0.5f * v) * (1.f + erff(v / 1.4142135f));
                }
                out[(size_t)seq * n_items + item] = v;
                if (kBest && (v > best || (v == best && item < best_i))) { best = v; best_i = item; }
            }
        }
    }
}

// n4 float4 written by other CTAs -> shared memory, read past L1, with every load of a thread in flight at once (a loop the
// compiler unrolls by four waits for DRAM / L2 once per four elements: nine round trips for the attention partials).
template <int kPer>
__device__ __forceinline__ void stage_f4(float* dst, const float* src, int n4) {
    float4 v[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const int i = threadIdx.x + j * kMegaThreads;
        if (i < n4) v[j] = __ldcg(reinterpret_cast<const float4*>(src) + i);
    }
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const int i = threadIdx.x + j * kMegaThreads;
        if (i < n4) reinterpret_cast<float4*>(dst)[i] = v[j];
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
    BarrierState bar = {p.barrier, 0u, gridDim.x, p.status, p.timing, 0};
    if (p.timing && blockIdx.x == 0 && threadIdx.x == 0) p.timing[bar.n++] = global_ns();
    float best = -INFINITY;   // lm_head: the largest logit this lane has produced
    int best_i = 0x7fffffff;
    Round rnd;                // the weights of this warp's first items of the next projection
    gemv_prefetch(rnd, p.layers[0].w_qkv_t, 3 * kD, kD);

    for (int s = 0; s < R; ++s) {
        const int token = s < rows ? p.token[s] : 0;
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
    const int chunk_len = (len + n_chunks - 1) / n_chunks, j0 = ck * chunk_len, j1 = min(len, j0 + chunk_len);
    const size_t cache_at = ((size_t)p.slot[seq] * H + head) * p.ctx_cap * hd;
    const float scale = 1.0f / sqrtf((float)hd);
    const int part_stride = hd + 2;

#pragma unroll 1
    for (int l = 0; l < p.n_layers; ++l) {
        const MegaLayer& L = p.layers[l];   // the table is part of the kernel parameters: no pointer chase through memory
        // ---- residual update from the previous block's MLP (four partial sums), ln_1, qkv --------------------------
        if (l > 0) residual_norm<R, 4>(h, xn, p.pe, p.layers[l - 1].b_mlp_out, L.ln1_g, L.ln1_b, p.eps, red);
        else residual_norm<R, 0>(h, xn, nullptr, nullptr, L.ln1_g, L.ln1_b, p.eps, red);
        gemv_items<R, false>(rnd, L.w_qkv_t, 3 * kD, xn, p.qkv, rows, best, best_i);
        grid_arrive(bar);
        gemv_prefetch(rnd, L.w_out_t, kD, kD);   // kept across the attention phase
        grid_wait(bar);
        // ---- attention: CTA = (sequence, head, context chunk) ---------------------------------------------------------
        if (attends) {
            float* kc = L.k_cache + cache_at;
            float* vc = L.v_cache + cache_at;
            // q, and K / V of the new token, from the qkv vector the other CTAs wrote (read past L1)
            float* qs = xn;            // [hd]
            float* k_new = xn + hd;    // [hd]
            float* v_new = xn + 2 * hd;
            const float* qkv = p.qkv + (size_t)seq * 3 * kD + head * hd;
            for (int c = tid; c < 3 * hd; c += kMegaThreads) {
                const int which = c / hd, e = c - which * hd;
                xn[c] = __ldcg(qkv + which * kD + e) + L.b_qkv[which * kD + head * hd + e];
            }
            __syncthreads();
            float* sc = big;   // scores of this slice
            if (j0 <= pos && pos < j1)   // the new token's row goes into the cache for the steps to come
                for (int c = tid; c < hd; c += kMegaThreads) { kc[(size_t)pos * hd + c] = k_new[c]; vc[(size_t)pos * hd + c] = v_new[c]; }
            // scores: hd / 4 lanes per key, four times 128 / hd keys of a warp under way at once
            {
                const int lanes = hd >> 2, per = 32 / lanes, sub = lane / lanes, c4 = (lane - sub * lanes) * 4;
                const float4 q4 = *reinterpret_cast<const float4*>(qs + c4);
                for (int base = j0 + warp * per; base < j1; base += 4 * kMegaWarps * per) {
                    float4 k4[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int j = base + u * kMegaWarps * per + sub;
                        k4[u] = j >= j1 ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>((j == pos ? k_new : kc + (size_t)j * hd) + c4);
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int j = base + u * kMegaWarps * per + sub;
                        float t = fmaf(q4.w, k4[u].w, fmaf(q4.z, k4[u].z, fmaf(q4.y, k4[u].y, q4.x * k4[u].x)));
                        for (int o = lanes >> 1; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                        if (c4 == 0 && j < j1) sc[j - j0] = t * scale;
                    }
                }
            }
            __syncthreads();
            float mx = -INFINITY;
            for (int j = tid; j < j1 - j0; j += kMegaThreads) mx = fmaxf(mx, sc[j]);
            mx = warp_max(mx);
            if (lane == 0) red[32 + warp] = mx;
            __syncthreads();
            mx = red[32];
#pragma unroll
            for (int w = 1; w < kMegaWarps; ++w) mx = fmaxf(mx, red[32 + w]);
            float sum = 0.f;
            for (int j = tid; j < j1 - j0; j += kMegaThreads) {
                const float e = expf(sc[j] - mx);
                sc[j] = e;
                sum += e;
            }
            sum = block_sum(sum, red);
            // context: thread (part, c) walks positions part, part + parts, ...
            const int parts = kMegaThreads / hd;
            const int c = tid % hd, part = tid / hd;
            float acc = 0.f;
#pragma unroll 8
            for (int j = j0 + part; j < j1; j += parts) acc = fmaf(sc[j - j0], (j == pos ? v_new : vc + (size_t)j * hd)[c], acc);
            float* comb = red + 64;   // [parts][hd], where the partials of all heads are staged later
            comb[part * hd + c] = acc;
            __syncthreads();
            float* out = p.att_part + (size_t)blockIdx.x * part_stride;
            if (tid < hd) {
                float v = 0.f;
                for (int q2 = 0; q2 < parts; ++q2) v += comb[q2 * hd + tid];
                out[2 + tid] = v;
            }
            if (tid == 0) { out[0] = j1 > j0 ? mx : -INFINITY; out[1] = j1 > j0 ? sum : 0.f; }
        }
        grid_barrier(bar);
        // ---- merge the attention partials (every CTA, all heads), out projection --------------------------------------
        {
            // all partials -> shared memory with independent loads (a dependent chain of L2 round trips per element cost
            // 7 us here), then the merge from shared memory
            float* parts_s = red + 64;   // [rows * H * n_chunks][hd + 2]
            const int n_part = n_tasks * part_stride;
            for (int base = 0; base < n_part / 4; base += 12 * kMegaThreads)   // one pass for GPT-2's 12 x 12 x 66 floats
                stage_f4<12>(parts_s + 4 * base, p.att_part + 4 * base, n_part / 4 - base);
            for (int i = (n_part / 4) * 4 + tid; i < n_part; i += kMegaThreads) parts_s[i] = __ldcg(p.att_part + i);
            __syncthreads();
            for (int i = tid; i < rows * kD; i += kMegaThreads) {
                const int unit = i / hd, c = i - unit * hd;   // sequence * H + head
                const float* part = parts_s + unit * n_chunks * part_stride;
                float M = -INFINITY;
                for (int k = 0; k < n_chunks; ++k) M = fmaxf(M, part[k * part_stride]);
                float Ls = 0.f, O = 0.f;
                for (int k = 0; k < n_chunks; ++k) {
                    const float m_k = part[k * part_stride];
                    if (m_k == -INFINITY) continue;
                    const float wgt = expf(m_k - M);
                    Ls = fmaf(part[k * part_stride + 1], wgt, Ls);
                    O = fmaf(part[k * part_stride + 2 + c], wgt, O);
                }
                xn[i] = O / Ls;
            }
            __syncthreads();
        }
        gemv_items<R, false>(rnd, L.w_out_t, kD, xn, p.pc, rows, best, best_i);
        grid_arrive(bar);
        gemv_prefetch(rnd, L.w_mlp_in_t, kMlp, kD);
        grid_wait(bar);
        // ---- residual update, ln_2, MLP in + GELU ---------------------------------------------------------------------
        residual_norm<R, 1>(h, xn, p.pc, L.b_out, L.ln2_g, L.ln2_b, p.eps, red);
        gemv_items<R, false, true>(rnd, L.w_mlp_in_t, kMlp, xn, p.mh, rows, best, best_i, L.b_mlp_in);
        grid_arrive(bar);
        gemv_prefetch(rnd, L.w_mlp_out_t, kD, kMlp);
        grid_wait(bar);
        // ---- MLP out: partial sums per 768-k chunk; a CTA's items all lie in chunk blockIdx % 4 --------------------------
        {
            constexpr int N = (R * kD / 4 + kMegaThreads - 1) / kMegaThreads;
            float4 v[N];
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const int i = tid + j * kMegaThreads, s = i / (kD / 4), e = i - s * (kD / 4);
                if (i < R * kD / 4) v[j] = __ldcg(reinterpret_cast<const float4*>(p.mh + (size_t)s * kMlp + (blockIdx.x & 3) * kD) + e);
            }
#pragma unroll
            for (int j = 0; j < N; ++j)
                if (tid + j * kMegaThreads < R * kD / 4) reinterpret_cast<float4*>(big)[tid + j * kMegaThreads] = v[j];
            __syncthreads();
        }
        gemv_items<R, false>(rnd, L.w_mlp_out_t, kMlp, big, p.pe, rows, best, best_i);
        grid_arrive(bar);
        if (l + 1 < p.n_layers) gemv_prefetch(rnd, p.layers[l + 1].w_qkv_t, 3 * kD, kD);
        else gemv_prefetch(rnd, p.lm_head_t, p.vocab, kD);
        grid_wait(bar);
    }
    // ---- last residual update, final LayerNorm, lm_head, greedy pick ----------------------------------------------------
    residual_norm<R, 4>(h, xn, p.pe, p.layers[p.n_layers - 1].b_mlp_out, p.lnf_g, p.lnf_b, p.eps, red);
    gemv_items<R, true>(rnd, p.lm_head_t, p.vocab, xn, p.logits, rows, best, best_i);
    // the storing lanes hold their warp's best of a sequence; CTA best -> cand[sequence][blockIdx.x]
    float* bv = big;                                        // [warp][R]
    int* bi = reinterpret_cast<int*>(big + kMegaWarps * R);
    __syncthreads();
    if (lane % (32 / R) == 0) { bv[warp * R + lane / (32 / R)] = best; bi[warp * R + lane / (32 / R)] = best_i; }
    __syncthreads();
    if (tid < rows) {
        for (int w = 1; w < kMegaWarps; ++w)
            if (bv[w * R + tid] > bv[tid] || (bv[w * R + tid] == bv[tid] && bi[w * R + tid] < bi[tid])) { bv[tid] = bv[w * R + tid]; bi[tid] = bi[w * R + tid]; }
        p.cand_val[tid * gridDim.x + blockIdx.x] = bv[tid];
        p.cand_idx[tid * gridDim.x + blockIdx.x] = bi[tid];
    }
    grid_barrier(bar);
    if (blockIdx.x == 0 && warp < rows) {
        float v = -INFINITY;
        int ix = 0x7fffffff;
        for (int k = lane; k < (int)gridDim.x; k += 32) {
            const float cv = __ldcg(p.cand_val + warp * gridDim.x + k);
            const int ci = __ldcg(p.cand_idx + warp * gridDim.x + k);
            if (cv > v || (cv == v && ci < ix)) { v = cv; ix = ci; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
            if (ov > v || (ov == v && oi < ix)) { v = ov; ix = oi; }
        }
        if (lane == 0 && p.greedy) p.sampled[warp] = ix;
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
    return (2 * (size_t)layout * kD + mega_big_floats(layout, rows, H, ctx_cap) + 64 + (size_t)sm_count() * (hd + 2) + 64) * sizeof(float);
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
    GPTRS_CUDA_OK(cudaMemsetAsync(p.barrier, 0, sizeof(unsigned), st));
    const int layout = mega_layout(p.rows);
    p.big_floats = (int)mega_big_floats(layout, p.rows, p.H, p.ctx_cap);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)sm_count());
    cfg.blockDim = dim3(kMegaThreads);
    cfg.dynamicSmemBytes = mega_smem_bytes(layout, p.rows, p.H, p.hd, p.ctx_cap);
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeCooperative;   // all CTAs co-resident: they meet at grid-wide barriers
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kerns[layout == 1 ? 0 : layout == 2 ? 1 : layout == 4 ? 2 : 3], p);
    if (e != cudaSuccess) return fail(GPTRS_EXECUTION, std::string("cooperative launch failed: ") + cudaGetErrorString(e));
    return GPTRS_OK;
}

}  // namespace gptrs
