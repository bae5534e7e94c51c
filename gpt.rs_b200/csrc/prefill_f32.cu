// Attention of prompt rows in f32 over the dense KV cache (attention_decode_cache, crates/gpt-rs/src/ops/functional/attention.rs:657-779,
// for the rows of prompts): a CTA takes one query head of up to 32 neighbouring rows of one sequence, so that a key is read once for
// all of them instead of once for each.
//
// Two groups of 128 threads take the blocks of 64 keys in turn, each with its own online softmax, and merge at the end: the last rows'
// CTAs are a chain of blocks (15 at 937 rows), and that chain is what the kernel takes. Per block a group has 32 x 64 scores with a 4 x 4
// tile per thread (operands in shared memory, 16-byte reads: 4 + 4 of them feed 64 fused multiply-adds), the softmax in f32 over the 16
// threads of a row, then 4 rows x HD / 16 columns of the output per thread. Heads are the fastest grid axis, so that the longest chains
// start first. 937 rows of 12 heads of 64: 72 us; 109 with one group, 464 with a CTA per row and head.
//
// Which rows are worth a tile (us, a CTA per row and head / tiles cut at the sequences' ends, 12 heads of 64): a row kernel's CTA takes
// 3.3 + 0.039 per key and many run side by side, a tile's takes 3 + 5.2 per 128 keys whatever its rows. 32 sequences of one row at 900
// keys 94 / 140, of four 209 / 140, of eight 322 / 140; eight rows of each of 8 sequences at 32 keys 6.3 / 8.3, at 128 keys 14.9 / 10.4.
// One sequence of 16 rows at 32, 300, 900 keys: 5.1 / 7.2, 17.3 / 18.1, 44 / 45; of 32 rows: 5.4 / 8.1, 20 / 19, 53 / 46. So runs of
// eight rows and more become tiles in passes of more than 256 (row, head) pairs.
#include "engine.h"

namespace gptrs {
namespace {

struct PrefillF32Params {
    const float* qkv;   // [T][(Hq + 2 Hkv) * hd]; only the Q part is read
    const float* k_cache;
    const float* v_cache;
    const int* positions;
    const int* slot;
    const int2* tiles;  // (first row, rows) of the tiles: rows of one sequence each
    float* out;         // [T][Hq * hd]
    int Hq, Hkv, capacity;
    float scale;
};

constexpr int kPfRows = 32, kPfKeys = 64, kPfGroup = 4 * kPfRows, kPfThreads = 2 * kPfGroup;

template <int HD>
__global__ void __launch_bounds__(kPfThreads, HD == 64 ? 2 : 1) attention_tiles_f32_kernel(const PrefillF32Params p) {
    constexpr int LD = HD + 4, LP = kPfKeys + 4, OC = HD / 64;   // OC float4 columns of a thread
    extern __shared__ __align__(16) float pf_smem[];
    const int group = threadIdx.x / kPfGroup, tid = threadIdx.x % kPfGroup, ty = tid >> 4, tx = tid & 15;
    float* qs = pf_smem;                                             // [32][LD]
    float* ks = qs + kPfRows * LD + group * (2 * kPfKeys * LD + kPfRows * LP);   // a group's [64][LD]
    float* vs = ks + kPfKeys * LD;                                   // [64][LD]
    float* ps = vs + kPfKeys * LD;                                   // [32][LP]
    __shared__ int pos_s[kPfRows];
    auto group_sync = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(1 + group), "n"(kPfGroup) : "memory"); };
    auto group_any = [&](bool mine) {   // a barrier that says whether it is so for a thread of the group
        uint32_t any;
        asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.or.pred q, %2, %3, p;\nselp.u32 %0, 1, 0, q;\n}\n"
                     : "=r"(any) : "r"((uint32_t)mine), "r"(1 + group), "n"(kPfGroup) : "memory");
        return any != 0;
    };
    const int h = blockIdx.x, hk = h / (p.Hq / p.Hkv);
    const int width = (p.Hq + 2 * p.Hkv) * HD;
    pdl_launch_dependents();
    pdl_wait();
    const int2 tile = p.tiles[gridDim.y - 1 - blockIdx.y];           // the last rows see the most keys: they start first
    const int t0 = tile.x, rows = tile.y, slot = p.slot[t0];
    if (threadIdx.x < kPfRows) pos_s[tid] = tid < rows ? min(max(p.positions[t0 + tid], 0), p.capacity - 1) : -1;   // DynamicUpdateSlice clamps its start
    for (int i = threadIdx.x; i < kPfRows * (HD / 4); i += kPfThreads) {
        const int r = i / (HD / 4), c = i % (HD / 4) * 4;
        *reinterpret_cast<float4*>(qs + r * LD + c) =
            r < rows ? *reinterpret_cast<const float4*>(p.qkv + (size_t)(t0 + r) * width + h * HD + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    float o[4][4 * OC], mx[4], sum[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        mx[r] = -INFINITY; sum[r] = 0.f;
#pragma unroll
        for (int c = 0; c < 4 * OC; ++c) o[r][c] = 0.f;
    }
    int last = 0;
    for (int i = 0; i < rows; ++i) last = max(last, pos_s[i]);
    const float* kc = p.k_cache + ((size_t)slot * p.Hkv + hk) * p.capacity * HD;
    const float* vc = p.v_cache + ((size_t)slot * p.Hkv + hk) * p.capacity * HD;
    int limit[4];   // last visible key of this thread's rows
#pragma unroll
    for (int r = 0; r < 4; ++r) limit[r] = pos_s[4 * ty + r];
    for (int j0 = group * kPfKeys; j0 <= last; j0 += 2 * kPfKeys) {
        group_sync();   // the block before has been used
        float probe = 0.f;   // NaN once a value of this block is not finite
#pragma unroll 8
        for (int i = tid; i < kPfKeys * (HD / 4); i += kPfGroup) {
            const int j = i / (HD / 4), c = i % (HD / 4) * 4;
            const bool in = j0 + j <= last;
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            *reinterpret_cast<float4*>(ks + j * LD + c) = in ? *reinterpret_cast<const float4*>(kc + (size_t)(j0 + j) * HD + c) : zero;
            const float4 v = in ? *reinterpret_cast<const float4*>(vc + (size_t)(j0 + j) * HD + c) : zero;
            *reinterpret_cast<float4*>(vs + j * LD + c) = v;
            probe = fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, fmaf(v.w, 0.f, probe))));
        }
        const bool special = group_any(probe != probe);
        float s[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[r][j] = 0.f;
#pragma unroll 4
        for (int c = 0; c < HD; c += 4) {
            float4 q[4], k[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) q[r] = *reinterpret_cast<const float4*>(qs + (4 * ty + r) * LD + c);
#pragma unroll
            for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const float4*>(ks + (tx + 16 * j) * LD + c);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    s[r][j] = fmaf(q[r].x, k[j].x, s[r][j]); s[r][j] = fmaf(q[r].y, k[j].y, s[r][j]);
                    s[r][j] = fmaf(q[r].z, k[j].z, s[r][j]); s[r][j] = fmaf(q[r].w, k[j].w, s[r][j]);
                }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float top = mx[r];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[r][j] = j0 + tx + 16 * j <= limit[r] ? s[r][j] * p.scale : -INFINITY;
                top = fmaxf(top, s[r][j]);
            }
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
            const float base = top == -INFINITY ? 0.f : top;   // nothing visible so far
            const float keep = expf(mx[r] - base);
            mx[r] = top;
            float part = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float e = j0 + tx + 16 * j <= limit[r] ? expf(s[r][j] - base) : 0.f;
                ps[(4 * ty + r) * LP + tx + 16 * j] = e;
                part += e;
            }
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
            sum[r] = sum[r] * keep + part;
#pragma unroll
            for (int c = 0; c < 4 * OC; ++c) o[r][c] *= keep;
        }
        __syncwarp();   // the 16 threads of a row write and read its weights, and they are in one warp
        if (special) {   // the weight 0 of a key that a row does not see would not keep an infinity or NaN from it
#pragma unroll 1
            for (int j = 0; j < kPfKeys; ++j)
#pragma unroll
                for (int c = 0; c < OC; ++c) {
                    const float4 v = *reinterpret_cast<const float4*>(vs + j * LD + 4 * tx + 64 * c);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        if (j0 + j > limit[r]) continue;
                        const float w = ps[(4 * ty + r) * LP + j];
                        o[r][4 * c] = fmaf(w, v.x, o[r][4 * c]); o[r][4 * c + 1] = fmaf(w, v.y, o[r][4 * c + 1]);
                        o[r][4 * c + 2] = fmaf(w, v.z, o[r][4 * c + 2]); o[r][4 * c + 3] = fmaf(w, v.w, o[r][4 * c + 3]);
                    }
                }
            continue;
        }
#pragma unroll 4
        for (int j = 0; j < kPfKeys; j += 4) {
            float4 e[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) e[r] = *reinterpret_cast<const float4*>(ps + (4 * ty + r) * LP + j);
#pragma unroll
            for (int jj = 0; jj < 4; ++jj)
#pragma unroll
                for (int c = 0; c < OC; ++c) {
                    const float4 v = *reinterpret_cast<const float4*>(vs + (j + jj) * LD + 4 * tx + 64 * c);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const float w = jj == 0 ? e[r].x : jj == 1 ? e[r].y : jj == 2 ? e[r].z : e[r].w;
                        o[r][4 * c] = fmaf(w, v.x, o[r][4 * c]); o[r][4 * c + 1] = fmaf(w, v.y, o[r][4 * c + 1]);
                        o[r][4 * c + 2] = fmaf(w, v.z, o[r][4 * c + 2]); o[r][4 * c + 3] = fmaf(w, v.w, o[r][4 * c + 3]);
                    }
                }
        }
    }
    // group 1 hands its state over in its own buffers: [row][16 threads][4 OC], then maximum and sum
    float* other = qs + kPfRows * LD + 2 * kPfKeys * LD + kPfRows * LP;
    float* other_ml = other + kPfRows * HD;
    if (group == 1) {
        group_sync();   // its last block has been used
#pragma unroll
        for (int r = 0; r < 4; ++r) {
#pragma unroll
            for (int c = 0; c < OC; ++c)
                *reinterpret_cast<float4*>(other + (4 * ty + r) * HD + 4 * tx + 64 * c) = make_float4(o[r][4 * c], o[r][4 * c + 1], o[r][4 * c + 2], o[r][4 * c + 3]);
            if (tx == 0) { other_ml[2 * (4 * ty + r)] = mx[r]; other_ml[2 * (4 * ty + r) + 1] = sum[r]; }
        }
    }
    __syncthreads();
    if (group == 1) return;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        if (4 * ty + r >= rows) continue;
        // group 0 has seen position 0 of every row: its maximum is a number
        const float m1 = other_ml[2 * (4 * ty + r)], top = fmaxf(mx[r], m1), f0 = expf(mx[r] - top), f1 = expf(m1 - top);
        const float inv = sum[r] * f0 + other_ml[2 * (4 * ty + r) + 1] * f1;
#pragma unroll
        for (int c = 0; c < OC; ++c) {
            const float4 u = *reinterpret_cast<const float4*>(other + (4 * ty + r) * HD + 4 * tx + 64 * c);
            *reinterpret_cast<float4*>(p.out + ((size_t)(t0 + 4 * ty + r) * p.Hq + h) * HD + 4 * tx + 64 * c) =
                make_float4((o[r][4 * c] * f0 + u.x * f1) / inv, (o[r][4 * c + 1] * f0 + u.y * f1) / inv, (o[r][4 * c + 2] * f0 + u.z * f1) / inv,
                            (o[r][4 * c + 3] * f0 + u.w * f1) / inv);
        }
    }
}

template <int HD>
int launch(const PrefillF32Params& p, int64_t n_tiles, cudaStream_t st) {
    constexpr size_t smem = (size_t)(kPfRows * (HD + 4) + 2 * (2 * kPfKeys * (HD + 4) + kPfRows * (kPfKeys + 4))) * sizeof(float);
    static PerDeviceOnce attr_once;
    if (attr_once.first_time()) GPTRS_CUDA_OK(cudaFuncSetAttribute(attention_tiles_f32_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return launch_kernel(attention_tiles_f32_kernel<HD>, dim3((unsigned)p.Hq, (unsigned)n_tiles), dim3(kPfThreads), smem, st, 1, p);
}

}  // namespace

// Splits the rows of a pass: runs of rows of one sequence that are worth it into tiles, (first row, rows) pairs at `lists`, the other rows'
// numbers behind them. Without tiles the lists are empty: every row goes to the kernel with a CTA per row and head.
AttentionF32Plan attention_f32_plan(const int32_t* slots, int n_tokens, int n_q_heads, int head_dim, int capacity, int32_t* lists) {
    AttentionF32Plan plan;
    if ((head_dim != 64 && head_dim != 128) || capacity > 32768 || (int64_t)n_tokens * n_q_heads <= 256) return plan;
    auto each_run = [&](auto&& f) {
        for (int i = 0, end; i < n_tokens; i = end) {
            for (end = i + 1; end < n_tokens && slots[end] == slots[i]; ++end) {}
            f(i, end);
        }
    };
    each_run([&](int i, int end) {
        if (end - i < 8) return;
        for (; i < end; i += kPfRows, ++plan.tiles) { lists[2 * plan.tiles] = i; lists[2 * plan.tiles + 1] = end - i < kPfRows ? end - i : kPfRows; }
    });
    if (!plan.tiles) return plan;
    each_run([&](int i, int end) {
        if (end - i < 8)
            for (; i < end; ++i) lists[2 * plan.tiles + plan.rows++] = i;
    });
    return plan;
}

int attention_tiles_f32(const float* qkv, const float* k_cache, const float* v_cache, const int32_t* positions, const int32_t* slot, float* out,
                        const int32_t* tiles, int n_tiles, int64_t n_q_heads, int64_t n_kv_heads, int64_t head_dim, int64_t capacity, cudaStream_t st) {
    const PrefillF32Params p = {qkv, k_cache, v_cache, positions, slot, reinterpret_cast<const int2*>(tiles), out, (int)n_q_heads, (int)n_kv_heads, (int)capacity,
                                1.0f / sqrtf((float)head_dim)};
    return head_dim == 64 ? launch<64>(p, n_tiles, st) : launch<128>(p, n_tiles, st);
}

}  // namespace gptrs
