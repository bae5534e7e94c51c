// One decode step of up to eight sequences of a W4 or W8 Ministral-style model as a single cooperative kernel:
// Ministral::forward_with_decode_cache for a one-token chunk (crates/gpt-rs/src/model/ministral.rs:613-766): norm_1 -> qkv -> RoPE ->
// attention over the paged cache -> out projection + residual -> norm_2 -> gate / up + SwiGLU -> down + residual, final norm, lm_head and
// the greedy pick.
//
// Why one kernel: a projection of a few rows is a weight stream of 1 to 4 us, but five dependent launches per layer took 7 to 9 us each
// (launch, first DRAM round trip, pipeline fill, drain). Here
//   * one CTA per SM stays for the whole step. Every one of its 15 warps has a private ring of weight stages that one further warp
//     (lane w serves warp w) fills with bulk copies in the order in which the step consumes them, across projections and layers: what the
//     weights wait for is only room in the ring, never the activations, so HBM streams while the chain of activations goes on.
//   * a CTA owns whole 16-channel tiles, neighbours in memory, and its warps share their K range evenly: a warp's part of a projection is
//     one contiguous run of (tile, 128-k group) units. The warps' partial sums meet in shared memory, in a fixed order.
//   * there is no grid barrier: what CTAs hand to each other are words {value, flag} that their readers poll (flag_words.cuh).
//   * the residual stream stays in f32 in the shared memory of the CTA that owns its columns (out and down share the column split); the
//     exchanged activations are bf16(h * gain) with sums of squares per tile, and the consumer scales its result by 1 / rms.
//   * attention: CTA (row, kv head, slice of the pages); pairs of warps take a page each (bulk copies, mma.sync, half of the value
//     channels per warp of the pair), partial outputs of several slices travel to the CTA of slice 0.
//   * every projection runs through one copy of the code: with a copy per projection (180 KB of code) the phases ran from a cold instruction
//     cache and took three times as long.
// What bounds it: the widening of the weights (a unit of 16 channels x 128 k costs a scheduler 200 to 230 cycles in W4, of which 112 are the shifts and
// logic operations at half rate; 350 in W8), then 1.6 to 3 us per exchange. A step, kernel per projection / this one, us, 150 tokens: W4 of width
// 3072, six layers, one sequence 305 / 263, three 346 / 258, seven 451 / 319; width 1024, four layers, one 128 / 109, seven 158 / 112; W8 of width 2048,
// four layers, one 187 / 159, seven 197 / 173. 3000 tokens, where it gains least, four layers: W4 of width 3072, one 231 / 219, of width 1024 136 / 130; W8
// of width 1024, eight 164 / 160, of width 2048 232 / 231. 8000 tokens, W4 of width 2048, one 255 / 178. Other lengths and where it is not taken:
// quant_step_max_rows and quant_step_pays. It has every SM for itself: two models that step on two threads take turns (one sequence each, four
// layers, us a step, W4 of width 3072 287 / 344, of width 1024 170 / 176; W8 of width 2048 241 / 279); GPTRS_QUANT_STEP=0 at finalize leaves a model with
// the kernel per projection.
// Arithmetic of the tiles as in w4_gemv_kernel / quant_matmul_kernel: exact integers in bf16 through mma.sync, group scales on f32 sums.
// Every wait is bounded: a thread that gives up records a status and stops waiting (code 5; ring or page copies: 3).
#include <algorithm>
#include <climits>

#include "flag_words.cuh"
#include "matmul_common.cuh"
#include "quant_step.h"

namespace gptrs {
void matmul_wait_limits(uint32_t* spin_limit, int* starve);   // umma_matmul.cu
int attention_step_splits(int64_t max_ctx_len, int64_t n_tokens, int64_t n_q_heads, int64_t n_kv_heads);   // paged_attention.cu
void step_wait_limits(uint32_t* spin_limit, uint32_t* flag_polls, int* starve) {
    matmul_wait_limits(spin_limit, starve);
    *flag_polls = *starve ? *spin_limit : kFlagPolls;
}
namespace {

// 15 warps that multiply and the producer: 16 warps may have 128 registers a thread. (With 16 + 1 it is 96; what is spilled then does not fit
// into the L1 that the rings leave, and a layer took twice as long.)
constexpr int kWarps = 15, kConsumers = kWarps * 32, kThreads = kConsumers + 32;
constexpr int kPairs = kWarps / 2;             // page slots of attention
constexpr int kPageBytes = 8192;               // K and V of 16 tokens of a kv head
constexpr int kSlotFloats = 8 * 16;            // partial sums of one tile: [row][channel]
constexpr int kPartStride = 132;               // floats of a query head's partial output: 128 values, maximum, sum
constexpr uint32_t kProducerLimit = 1u << 24;  // polls of the producer without a free stage

// stage of a warp's ring: W4 up to two units (one unit = one tile x 128 k; 1 KB of nibbles and 16 scales) of a tile, W8 one (2 KB). A stage's
// hand-over costs a warp about as much issue time as a third of a unit's arithmetic.
template <int BITS> constexpr int kUnitBytes = BITS == 4 ? 1024 : 2048;
template <int BITS> constexpr int kUnits = BITS == 4 ? 2 : 1;
template <int BITS> constexpr int kStageBytes = BITS == 4 ? 2 * (1024 + 32) : 2048;

// ---- what the CTAs exchange: buffers of {value, flag} words, in bytes from the start of the exchange area ----------------------------
StepExchange exchange_layout(int D, int FF, int Hq, int Hkv) {
    StepExchange e;
    uint32_t at = 0;
    auto take = [&](uint32_t words) { const uint32_t a = at; at += (words * 8 + 255) & ~255u; return a; };
    const uint32_t R = kStepMaxRows;
    e.x_in = take(R * D / 2);                       // two bf16 per word
    e.x_mid = take(R * D / 2);
    e.qkv = take(R * (Hq + 2 * Hkv) * 64);
    e.attn = take(R * Hq * 64);
    e.mlp = take(R * FF / 2);
    e.ss_in = take(R * (D / 16));                   // one f32 per word, [row][tile]
    e.ss_mid = take(R * (D / 16));
    e.part = take(256u * 8 * kPartStride);          // [task of attention][query head of the group][128 values, maximum, sum, -, -]
    e.best = take(256u * R * 2);                    // [row][CTA] value, index
    e.total = at;
    return e;
}

// ---- shared memory -------------------------------------------------------------------------------------------------------------------
StepSmem smem_plan(int rows, int k_max, int group, int h_cols, int max_tiles, int stages, int stage_bytes) {
    StepSmem s;
    uint32_t at = 0;
    auto take = [&](uint32_t bytes) { const uint32_t a = at; at += (bytes + 255u) & ~255u; return a; };
    const uint32_t x = (uint32_t)rows * k_max * 2, pages = kPairs * kPageBytes;
    s.x = take(x > pages ? x : pages);              // activations of a phase; pages of attention
    s.zero = take(256);
    const uint32_t slots = (uint32_t)(kWarps + max_tiles) * kSlotFloats * 4, parts = (uint32_t)kPairs * group * kPartStride * 4;
    s.slots = take(slots > parts ? slots : parts);  // partial sums of a phase; partial outputs of attention
    s.qkv = take((uint32_t)(group + 2) * 256);      // this CTA's queries, new key and value
    s.h = take((uint32_t)rows * h_cols * 4);        // its columns of the residual stream
    s.inv = take(8 * 4);
    s.tiles = take(5 * 16);                         // per projection: the CTA's first tile and tiles, 128-k groups, all tiles
    s.ranges = take(5 * kWarps * 16);               // per projection and warp: its units [from, to), tile and group of the first
    s.spans = take(4 * 32 * 2);                     // first and last warp of every tile, per projection
    s.best = take(kWarps * 8 * 8);
    s.bars = take((uint32_t)(kWarps * stages * 2 + kPairs) * 8);
    s.ring = take((uint32_t)kWarps * stages * stage_bytes);
    s.total = at;
    return s;
}

__device__ __forceinline__ int part_lo(int n, int parts, int i) { return (int)((uint32_t)n * (uint32_t)i / (uint32_t)parts); }

__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;\n" ::"n"(kConsumers) : "memory"); }
__device__ __forceinline__ void pair_sync(int pair) { asm volatile("bar.sync %0, 64;\n" ::"r"(2 + pair) : "memory"); }

__device__ __forceinline__ bool test_wait(uint64_t* bar, uint32_t parity) {   // never suspends: the lanes of the producer wait for different barriers
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool wait_bounded(uint64_t* bar, uint32_t parity) {
#pragma unroll 1
    for (uint32_t i = 0; i < kSpinLimit; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ uint4 lds_128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds_32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Eight nibbles of layout A -> four bf16 pairs q (128 + (q + 8) by three shifts and four three-input logic operations, minus 136: exact),
// times the rows. One block, so that this shape survives the optimiser (see quant_gemv.cu). The subtraction runs beside the logic pipe that
// bounds the rest: 193 cycles of a scheduler per unit; with the offset taken out by a second mma against ones 220, without any 174.
__device__ __forceinline__ void nibbles_mma(float (&d)[4], uint32_t q, uint32_t b0, uint32_t b1) {
    asm volatile("{\n"
                 ".reg .b32 t1, t2, t3, a0, a1, a2, a3, o;\n"
                 "mov.b32 o, 0x43084308;\n"
                 "shr.u32 t1, %4, 4;\n"
                 "shr.u32 t2, %4, 8;\n"
                 "shr.u32 t3, %4, 12;\n"
                 "lop3.b32 a0, %4, 0x000f000f, 0x43004300, 0xEA;\n"
                 "lop3.b32 a1, t1, 0x000f000f, 0x43004300, 0xEA;\n"
                 "lop3.b32 a2, t2, 0x000f000f, 0x43004300, 0xEA;\n"
                 "lop3.b32 a3, t3, 0x000f000f, 0x43004300, 0xEA;\n"
                 "sub.rn.bf16x2 a0, a0, o;\n"
                 "sub.rn.bf16x2 a1, a1, o;\n"
                 "sub.rn.bf16x2 a2, a2, o;\n"
                 "sub.rn.bf16x2 a3, a3, o;\n"
                 "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {a0,a1,a2,a3}, {%5,%6}, {%0,%1,%2,%3};\n"
                 "}\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(q), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t bytes_pair(uint32_t w, int first_byte) {   // bytes hold q + 128; 0x4B0000bb as f32 is 2^23 + bb
    const float lo = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650 + first_byte)) - 8388736.f;
    const float hi = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650 + first_byte + 1)) - 8388736.f;
    return pack_bf16x2(lo, hi);
}

// The projections of a layer in order, and the head.
enum { kQkv = 0, kOut = 1, kGateUp = 2, kDown = 3, kHead = 4 };

// What a warp needs to walk its units.
struct Ring {
    uint32_t base, bars;   // shared addresses: the warp's stages; its full barriers (the empty ones behind them)
    int stages, at;
    uint32_t phase, limit;   // limit: polls of a wait, 0 after one that gave up
};

// n units of a tile, a stage: acc (m16n8 fragment: channels g, g + 8; rows 2t, 2t + 1) += scale * (weights x rows of the unit's 128 k).
template <int BITS>
__device__ __forceinline__ void stage_units(Ring& r, int n, float (&acc)[4], uint32_t xblk, uint32_t xstep, int lane, int* status) {
    constexpr int U = kUnits<BITS>, L = BITS == 4 ? 2 : 4;
    const uint32_t full = r.bars + r.at * 8;
    uint32_t tries = 0;
    bool ok;
#pragma unroll 1
    do {
        uint32_t v;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(v) : "r"(full), "r"(r.phase) : "memory");
        ok = v != 0;
    } while (!ok && ++tries < r.limit);
    if (!ok) {   // nothing is read any more, by no later stage either
        r.limit = 0;
        if (lane == 0) atomicExch(status, 3);
        return;
    }
    const uint32_t st = r.base + r.at * kStageBytes<BITS>;
    uint4 q[U][L];
    uint32_t sc[U];
#pragma unroll
    for (int j = 0; j < U; ++j) {   // a second unit that is not there: what the stage holds
#pragma unroll
        for (int i = 0; i < L; ++i) q[j][i] = lds_128(st + j * kUnitBytes<BITS> + i * 512 + lane * 16);
        sc[j] = BITS == 4 ? lds_32(st + U * 1024 + j * 32 + (lane >> 2) * 4) : 0u;
    }
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(full + r.stages * 8) : "memory");
    if (++r.at == r.stages) { r.at = 0; r.phase ^= 1u; }
#pragma unroll
    for (int j = 0; j < U; ++j) {
        if (j >= n) break;
        if constexpr (BITS == 4) {
            float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k2 = 0; k2 < 4; ++k2) {
                uint32_t b[4];
                ldmatrix_x4(b, (xblk + j * xstep) ^ (k2 << 6));
                const uint4 c = q[j][k2 >> 1];
                nibbles_mma(part, (k2 & 1) ? c.z : c.x, b[0], b[1]);
                nibbles_mma(part, (k2 & 1) ? c.w : c.y, b[2], b[3]);
            }
            const __half2 sh = *reinterpret_cast<const __half2*>(&sc[j]);
            const float lo = __low2float(sh), hi = __high2float(sh);
            acc[0] = fmaf(part[0], lo, acc[0]); acc[1] = fmaf(part[1], lo, acc[1]);
            acc[2] = fmaf(part[2], hi, acc[2]); acc[3] = fmaf(part[3], hi, acc[3]);
        } else {
#pragma unroll
            for (int k2 = 0; k2 < 4; ++k2) {
                uint32_t b[4];
                ldmatrix_x4(b, (xblk + j * xstep) ^ (k2 << 6));
                const uint4 c = q[j][k2];
                mma_16816(acc, bytes_pair(c.x, 0), bytes_pair(c.x, 2), bytes_pair(c.y, 0), bytes_pair(c.y, 2), b[0], b[1]);
                mma_16816(acc, bytes_pair(c.z, 0), bytes_pair(c.z, 2), bytes_pair(c.w, 0), bytes_pair(c.w, 2), b[2], b[3]);
            }
        }
    }
}

template <int BITS>
__global__ void __launch_bounds__(kThreads, 1) quant_step_kernel(const __grid_constant__ QuantStepParams p) {
    extern __shared__ __align__(1024) unsigned char sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = blockIdx.x, grid = gridDim.x;
    const int D = p.D, FF = p.FF, QD = p.Hq * 128, M = p.rows, group = p.Hq / p.Hkv;
    const StepSmem& S = p.sm;
    const StepExchange& E = p.ex;
    int4* const tiles = reinterpret_cast<int4*>(sm + S.tiles);
    int4* const ranges = reinterpret_cast<int4*>(sm + S.ranges);
    uchar2* const spans = reinterpret_cast<uchar2*>(sm + S.spans);
    uint64_t* const bars = reinterpret_cast<uint64_t*>(sm + S.bars);
    uint64_t* const page_bar = bars + kWarps * p.stages * 2;

    // ---- tables of this CTA's part, barriers ----------------------------------------------------------------------------------------
    auto tiles_of = [&](int kind) { return kind == kQkv ? (p.Hq + 2 * p.Hkv) * 8 : kind == kGateUp ? FF / 8 : kind == kHead ? p.vocab / 16 : D / 16; };
    auto groups_of = [&](int kind) { return (kind == kOut ? QD : kind == kDown ? FF : D) / 128; };
    if (tid < 5 * kWarps) {
        const int kind = tid / kWarps, w = tid % kWarps, T = tiles_of(kind), G = groups_of(kind);
        const int t0 = part_lo(T, grid, cta), nt = part_lo(T, grid, cta + 1) - t0;
        if (w == 0) tiles[kind] = make_int4(t0, nt, G, T);
        // the head: whole tiles per warp, nothing to add up between warps
        const int lo = kind == kHead ? part_lo(nt, kWarps, w) * G : part_lo(nt * G, kWarps, w);
        const int hi = kind == kHead ? part_lo(nt, kWarps, w + 1) * G : part_lo(nt * G, kWarps, w + 1);
        ranges[tid] = make_int4(lo, hi, lo / G, lo % G);
    }
    if (tid >= 128 && tid < 256) {
        const int kind = (tid - 128) >> 5, i = tid & 31, T = tiles_of(kind), G = groups_of(kind);
        const int nt = part_lo(T, grid, cta + 1) - part_lo(T, grid, cta), U = nt * G;
        if (i < nt) {   // the last warp whose range begins at or before a unit holds it
            const int first = (kWarps * (i * G + 1) + U - 1) / U - 1, last = (kWarps * ((i + 1) * G) + U - 1) / U - 1;
            spans[tid - 128] = make_uchar2((unsigned char)min(first, kWarps - 1), (unsigned char)min(last, kWarps - 1));
        }
    }
    if (tid == kConsumers) {
#pragma unroll 1
        for (int i = 0; i < kWarps * p.stages * 2 + kPairs; ++i) mbar_init(bars + i, 1);
        mbar_fence_init();
    }
    if (tid >= 256 && tid < 320) reinterpret_cast<uint32_t*>(sm + S.zero)[tid - 256] = 0u;
    __syncthreads();

    const uint32_t ring_bytes = (uint32_t)p.stages * kStageBytes<BITS>;
    if (warp == kWarps) {
        // ---- the producer: lane w keeps the ring of warp w full ----------------------------------------------------------------------
        const bool mine = lane < kWarps && !(p.starve == 2 && lane == kWarps - 1);
        const uint32_t base = smem_u32(sm + S.ring) + min(lane, kWarps - 1) * ring_bytes;
        uint64_t* const full = bars + min(lane, kWarps - 1) * p.stages * 2;
        int layer = 0, kind = -1, left = 0, stage = 0, grp = 0, G = 1;
        uint32_t phase = 1, issued = 0, idle = 0;    // a wait for the phase before the first one passes
        const unsigned char *src = nullptr, *scales = nullptr;
        bool done = !mine;
#pragma unroll 1
        while (!__all_sync(0xffffffffu, done)) {
            bool moved = false;
#pragma unroll 1
            while (left == 0 && !done) {   // the next projection of which this warp has units
                if (kind == kHead) { done = true; break; }
                if (++kind == kHead && ++layer < p.n_layers) kind = kQkv;
                const int l = min(layer, p.n_layers - 1);
                const unsigned char* w = kind == kQkv ? p.layers[l].w_qkv : kind == kOut ? p.layers[l].w_out : kind == kGateUp ? p.layers[l].w_gate_up
                                         : kind == kDown ? p.layers[l].w_down : p.w_head;
                const int4 part = tiles[kind];
                const int4 r = ranges[kind * kWarps + lane];
                const size_t u0 = (size_t)part.x * part.z + r.x;
                left = r.y - r.x;
                grp = r.w;
                G = part.z;
                src = w + u0 * kUnitBytes<BITS>;
                scales = w + (size_t)part.w * part.z * 1024 + u0 * 32;   // W4: behind the nibbles
            }
            if (!done && test_wait(full + p.stages + stage, phase)) {
                const uint32_t bar = smem_u32(full + stage), dst = base + stage * kStageBytes<BITS>;
                const int n = min(kUnits<BITS>, min(left, G - grp));   // units of one tile
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"((uint32_t)(n * (kStageBytes<BITS> / kUnits<BITS>))) : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src),
                             "r"((uint32_t)(n * kUnitBytes<BITS>)), "r"(bar) : "memory");
                if (BITS == 4)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst + 2 * 1024), "l"(scales),
                                 "r"((uint32_t)(n * 32)), "r"(bar) : "memory");
                src += n * kUnitBytes<BITS>;
                scales += n * 32;
                grp = grp + n == G ? 0 : grp + n;
                ++issued;
                if (++stage == p.stages) { stage = 0; phase ^= 1u; }
                left -= n;
                moved = true;
            }
            if (__any_sync(0xffffffffu, moved)) idle = 0;
            else if (++idle > kProducerLimit) break;
            else __nanosleep(40);
        }
        // copies of a warp that gave up: all of them land before the CTA ends
        if (mine)
#pragma unroll 1
            for (uint32_t i = issued > (uint32_t)p.stages ? issued - p.stages : 0; i < issued; ++i) wait_bounded(full + i % p.stages, (i / p.stages) & 1u);
        return;
    }

    // ---- the consumers ---------------------------------------------------------------------------------------------------------------
    Ring ring = {smem_u32(sm + S.ring) + warp * ring_bytes, smem_u32(bars + warp * p.stages * 2), p.stages, 0, 0u, p.ring_polls};
    FlagWaiter wait = {p.flag_polls, p.status};
    const int g = lane >> 2, t = lane & 3;
    float* const slots = reinterpret_cast<float*>(sm + S.slots);
    float* const h_own = reinterpret_cast<float*>(sm + S.h);   // [row][this CTA's columns]
    float* const inv = reinterpret_cast<float*>(sm + S.inv);
    const int t_h0 = tiles[kOut].x, h_cols = tiles[kOut].y * 16;   // columns of the residual stream
    unsigned char* const ex = p.exchange;
    const int ss_tiles = D / 16;
    // rows of x in shared memory: block of 128 k = [row][256 bytes], 16-byte chunk c of a row at c ^ (row & 7)
    const bool row_valid = (lane & 7) < M;
    const uint32_t lane_base = row_valid ? smem_u32(sm + S.x) + (lane & 7) * 256 + (((lane >> 3) ^ (lane & 7)) << 4) : smem_u32(sm + S.zero);
    const uint32_t lane_stride = row_valid ? (uint32_t)M * 256u : 0u;
    const uint32_t inv_m = (65536u + (uint32_t)M - 1u) / (uint32_t)M;   // i / M == (i * inv_m) >> 16 for i < 4096
    auto by_m = [&](int i) { return (int)(((uint32_t)i * inv_m) >> 16); };
    auto rms = [&](float ss) { return rsqrtf(ss / (float)D + p.eps); };

    // x of a phase -> shared memory, a warp per (group of 128 k, row), four of them under way at once. One lane of a warp waits for one word
    // first: with every lane asking for its own, the requests for a few hot lines delay everything else (W4, one sequence, four layers of width
    // 1024: 137 us a step, three sequences with one lane asking 108).
    auto stage_x = [&](uint32_t from, int G, uint32_t flag, const unsigned char* ss) {
        const int n = M * G;
        auto word_of = [&](int i) {
            const int grp = by_m(i), row = i - grp * M;
            return ex + from + (uint32_t)(row * G + grp) * 512u + lane * 16;
        };
        // the sums of squares of few rows are the last warps' only task
        const bool apart = ss && M <= 3;
        const int nw = apart ? kWarps - M : kWarps, ss_row = !ss ? M : apart ? (warp >= nw ? warp - nw : M) : warp;
        if (warp < n) {
            if (lane == 0) wait.wait_word(word_of(warp), flag);
            __syncwarp();
        }
        if (warp < nw)
#pragma unroll 1
            for (int i0 = warp; i0 < n; i0 += 4 * nw) {   // past the end: the last one once more
                FlagWords w[4];
                bool found;
#pragma unroll 1
                do {
                    found = true;
#pragma unroll
                    for (int j = 0; j < 4; ++j) w[j] = peek_words(word_of(min(i0 + j * nw, n - 1)));
#pragma unroll
                    for (int j = 0; j < 4; ++j) found = found && has_flag(w[j], flag);
                } while (!found && wait.again());
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int i = min(i0 + j * nw, n - 1);
                    *reinterpret_cast<uint2*>(sm + S.x + (uint32_t)i * 256 + (((lane >> 1) ^ ((i - by_m(i) * M) & 7)) << 4) + (lane & 1) * 8) =
                        make_uint2((uint32_t)w[j].a, (uint32_t)w[j].b);
                }
            }
        if (ss_row < M) {
            const unsigned char* row = ss + (uint32_t)(ss_row * ss_tiles + lane) * 8u;
            if (lane == 0) wait.wait_word(row, flag);
            __syncwarp();
            float s = 0.f;
#pragma unroll 1
            for (int i0 = 0; i0 < ss_tiles; i0 += 192) {
                uint64_t w[6];
                bool found;
#pragma unroll 1
                do {
                    found = true;
#pragma unroll
                    for (int j = 0; j < 6; ++j) w[j] = peek_word(row + min(i0 + 32 * j, ss_tiles - 1 - lane) * 8);
#pragma unroll
                    for (int j = 0; j < 6; ++j) found = found && has_flag(w[j], flag);
                } while (!found && wait.again());
#pragma unroll
                for (int j = 0; j < 6; ++j) s += i0 + 32 * j + lane < ss_tiles ? word_f32(w[j]) : 0.f;
            }
            s = warp_sum(s);
            if (lane == 0) inv[ss_row] = rms(s);
        }
        consumers_sync();
    };

    // ---- the tokens' embeddings: this CTA's columns of the residual stream, and x of the first projection -----------------------------
    auto token_of = [&](int row) { return p.given ? p.token_in[row] : p.token[row]; };
    if (cta == 0 && tid < M && (token_of(tid) < 0 || token_of(tid) >= p.vocab)) atomicExch(p.status, 2);
#pragma unroll 1
    for (int m = 0; m < M; ++m) {
        const int id = token_of(m);
        const bool ok = id >= 0 && id < p.vocab;
#pragma unroll 1
        for (int c = tid; c < h_cols; c += kConsumers) h_own[m * h_cols + c] = ok ? p.tok_emb[(size_t)id * D + t_h0 * 16 + c] : 0.f;
    }
    {
        float* const sums = slots;   // [row][group of 128]
        const int G = D / 128;
        const float* ln = p.layers[0].ln1;
#pragma unroll 1
        for (int i = warp; i < M * G; i += kWarps) {
            const int grp = by_m(i), row = i - grp * M;
            const int id = token_of(row);
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (id >= 0 && id < p.vocab) v = *reinterpret_cast<const float4*>(p.tok_emb + (size_t)id * D + grp * 128 + lane * 4);
            const float4 gn = *reinterpret_cast<const float4*>(ln + grp * 128 + lane * 4);
            *reinterpret_cast<uint2*>(sm + S.x + (uint32_t)i * 256 + (((lane >> 1) ^ (row & 7)) << 4) + (lane & 1) * 8) =
                make_uint2(pack_bf16x2(v.x * gn.x, v.y * gn.y), pack_bf16x2(v.z * gn.z, v.w * gn.w));
            const float s = warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
            if (lane == 0) sums[row * G + grp] = s;
        }
        consumers_sync();
        if (tid < M) {
            float s = 0.f;
#pragma unroll 4
            for (int i = 0; i < G; ++i) s += sums[tid * G + i];
            inv[tid] = rms(s);
        }
        consumers_sync();
    }

    // ---- this CTA's part in attention: a slice of the pages of one kv head of one row ----------------------------------------------------
    const int splits = p.splits, n_tasks = M * p.Hkv * splits;
    const bool attends = cta < n_tasks;
    const int a_row = attends ? cta / (p.Hkv * splits) : 0, a_head = (cta / splits) % p.Hkv, a_split = cta % splits;
    int len = p.ctx[a_row];
    if (len < 1 || len > p.max_len) {
        if (attends && tid == 0) atomicExch(p.status, 2);
        len = len < 1 ? 1 : p.max_len;
    }
    const int pos = len - 1, pages = (len + 15) >> 4, per = (pages + splits - 1) / splits;
    const int pg0 = min(pages, a_split * per), pg1 = min(pages, pg0 + per);
    const int pair = warp % kPairs, half = warp / kPairs;   // the odd warp has half 2: no part in attention
    const int* const page_row = p.page_table + (size_t)p.slot[a_row] * p.max_pages;
    const int first_page = attends && pg0 + pair < pg1 ? page_row[pg0 + pair] : 0;
    uint32_t page_phase = 0;
    bool page_failed = false;
    unsigned char* const my_page = sm + S.x + pair * kPageBytes;
    auto load_page = [&](int layer, int page) {   // one thread of the pair
        fence_proxy_async();
        mbar_expect_tx(page_bar + pair, kPageBytes);
        bulk_g2s(my_page, p.pool + (size_t)layer * p.pool_layer_bytes + ((size_t)page * p.Hkv + a_head) * kPageBytes, kPageBytes, page_bar + pair);
    };
    auto swz = [](int tok, int chunk) { return tok * 256 + ((chunk ^ (tok & 7)) << 4); };

    auto better = [](float& v, int& i, float ov, int oi) { if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; } };
    // the largest logits of this thread's rows 2t, 2t + 1 and their ids: over the slots, which the head does not need
    float4* const best = reinterpret_cast<float4*>(slots) + tid;
    const int QKV = (p.Hq + 2 * p.Hkv) * 128;
    uint32_t flag = p.epoch;

#pragma unroll 1
    for (int phase = 0; phase <= 4 * p.n_layers; ++phase) {
        const int l = min(phase >> 2, p.n_layers - 1), kind = phase == 4 * p.n_layers ? kHead : phase & 3;
        const QuantStepLayer& L = p.layers[l];
        if (kind == kQkv) ++flag;
        if (kind == kOut && attends) {
            // ---- attention ---------------------------------------------------------------------------------------------------------------
            unsigned char* const qs = sm + S.qkv;   // rotated queries [group][128], new key, new value
            const unsigned char* const row_at = ex + E.qkv + (uint32_t)(a_row * QKV) * 4u;
            auto rotate = [](uint32_t& lo, uint32_t& hi, float2 c, float2 s) {   // pairs (channel, channel + 64), f32, rounded once
                const float a0 = bf16_lo(lo), a1 = bf16_hi(lo), b0 = bf16_lo(hi), b1 = bf16_hi(hi);
                lo = pack_bf16x2(a0 * c.x - b0 * s.x, a1 * c.y - b1 * s.y);
                hi = pack_bf16x2(b0 * c.x + a0 * s.x, b1 * c.y + a1 * s.y);
            };
            if (tid < (group + 1) * 16) {   // four channels and their partners
                const int head = tid >> 4, c = (tid & 15) * 4;
                const int col = head < group ? (a_head * group + head) * 128 : (p.Hq + a_head) * 128;
                const unsigned char* at = row_at + (col + c) * 4;
                const float4 cs = *reinterpret_cast<const float4*>(p.cos_table + (size_t)pos * 64 + c);
                const float4 sn = *reinterpret_cast<const float4*>(p.sin_table + (size_t)pos * 64 + c);
                FlagWords w0, w1;
#pragma unroll 1
                do { w0 = peek_words(at); w1 = peek_words(at + 256); } while (!(has_flag(w0, flag) && has_flag(w1, flag)) && wait.again());
                uint2 lo = make_uint2((uint32_t)w0.a, (uint32_t)w0.b), hi = make_uint2((uint32_t)w1.a, (uint32_t)w1.b);
                rotate(lo.x, hi.x, make_float2(cs.x, cs.y), make_float2(sn.x, sn.y));
                rotate(lo.y, hi.y, make_float2(cs.z, cs.w), make_float2(sn.z, sn.w));
                *reinterpret_cast<uint2*>(qs + head * 256 + c * 2) = lo;
                *reinterpret_cast<uint2*>(qs + head * 256 + 128 + c * 2) = hi;
            } else if (tid >= 256 && tid < 288) {
                const FlagWords w = wait.wait_words(row_at + ((p.Hq + p.Hkv + a_head) * 128 + lane * 4) * 4, flag);
                *reinterpret_cast<uint2*>(qs + (group + 1) * 256 + lane * 8) = make_uint2((uint32_t)w.a, (uint32_t)w.b);
            }
            consumers_sync();   // the slots' readers are through as well
            const uint32_t q_at = smem_u32(qs) + (uint32_t)(min(g, group - 1) * 256 + 4 * t);   // rows past the group repeat its last one: nobody reads theirs
            float o[8][4];
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
            float m_run = -INFINITY, l_run = 0.f;
            const uint32_t kb = smem_u32(my_page), vb = kb + kPageBytes / 2;
            const int k_tok = ((lane >> 4) << 3) + (lane & 7), k_half = (lane >> 3) & 1;
            const int v_tok = (((lane >> 3) & 1) << 3) + (lane & 7), v_chunk = lane >> 4;
#pragma unroll 1
            for (int pg = half < 2 ? pg0 + pair : pg1; pg < pg1; pg += kPairs) {
                const int next = pg + kPairs < pg1 ? page_row[pg + kPairs] : 0;
                if (!page_failed && !wait_bounded(page_bar + pair, page_phase)) {
                    page_failed = true;
                    if (lane == 0) atomicExch(p.status, 3);
                }
                page_phase ^= 1u;
                if (pg == pages - 1) {   // the new token's key and value, into this copy of the page and into the pool
                    if (half == 0 && !page_failed) {
                        const int tok = pos & 15, c = lane >> 2, in = (lane & 3) * 4;
                        const uint32_t k_lo = *reinterpret_cast<const uint32_t*>(qs + group * 256 + lane * 4);
                        const uint32_t k_hi = *reinterpret_cast<const uint32_t*>(qs + group * 256 + 128 + lane * 4);
                        const uint2 v_new = *reinterpret_cast<const uint2*>(qs + (group + 1) * 256 + lane * 8);
                        unsigned char* const blk = p.pool + (size_t)l * p.pool_layer_bytes + ((size_t)page_row[pg] * p.Hkv + a_head) * kPageBytes;
                        for (unsigned char* to : {my_page, blk}) {
                            *reinterpret_cast<uint32_t*>(to + swz(tok, c) + in) = k_lo;
                            *reinterpret_cast<uint32_t*>(to + swz(tok, c + 8) + in) = k_hi;
                            *reinterpret_cast<uint2*>(to + kPageBytes / 2 + swz(tok, lane >> 1) + (lane & 1) * 8) = v_new;
                        }
                    }
                    pair_sync(pair);
                }
                float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) {
                    uint32_t b[4];
                    ldmatrix_x4(b, kb + swz(k_tok, 2 * ks + k_half));
                    const uint32_t q0 = lds_32(q_at + ks * 32), q1 = lds_32(q_at + ks * 32 + 16);
                    mma_16816(s[0], q0, 0u, q1, 0u, b[0], b[1]);
                    mma_16816(s[1], q0, 0u, q1, 0u, b[2], b[3]);
                }
                float mx = -INFINITY;
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        s[nt][e] = pg * 16 + nt * 8 + 2 * t + e < len ? s[nt][e] * p.scale_log2 : -INFINITY;
                        mx = fmaxf(mx, s[nt][e]);
                    }
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                const float m_new = fmaxf(m_run, mx);   // finite: a page's first token is visible
                const float alpha = exp2f(m_run - m_new);
                float pr[2][2], psum = 0.f;
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        pr[nt][e] = exp2f(s[nt][e] - m_new);
                        psum += pr[nt][e];
                    }
                l_run = l_run * alpha + psum;
                m_run = m_new;
#pragma unroll
                for (int i = 0; i < 8; ++i) { o[i][0] *= alpha; o[i][1] *= alpha; }
                const uint32_t pa0 = pack_bf16x2(pr[0][0], pr[0][1]), pa2 = pack_bf16x2(pr[1][0], pr[1][1]);
#pragma unroll
                for (int np = 0; np < 4; ++np) {   // 64 value channels of this warp
                    uint32_t b[4];
                    ldmatrix_x4_trans(b, vb + swz(v_tok, half * 8 + 2 * np + v_chunk));
                    mma_16816(o[2 * np], pa0, 0u, pa2, 0u, b[0], b[1]);
                    mma_16816(o[2 * np + 1], pa0, 0u, pa2, 0u, b[2], b[3]);
                }
                if (pg + kPairs < pg1) {
                    pair_sync(pair);
                    if (half == 0 && lane == 0) load_page(l, next);
                }
            }
            if (page_failed) wait_bounded(page_bar + pair, page_phase ^ 1u);
            l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
            l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
            float* const po = slots;   // [pair][query head][132]
            if (g < group && half < 2) {
                float* to = po + (pair * group + g) * kPartStride;
#pragma unroll
                for (int i = 0; i < 8; ++i) *reinterpret_cast<float2*>(to + half * 64 + i * 8 + 2 * t) = make_float2(o[i][0], o[i][1]);
                if (half == 0 && t == 0) { to[128] = m_run; to[129] = l_run; }
            }
            consumers_sync();
#pragma unroll 1
            for (int i = tid; i < group * 32; i += kConsumers) {
                const int r = i >> 5, c = (i & 31) * 4;
                float mx = -INFINITY;
#pragma unroll
                for (int w = 0; w < kPairs; ++w) mx = fmaxf(mx, po[(w * group + r) * kPartStride + 128]);
                float sum = 0.f;
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int w = 0; w < kPairs; ++w) {
                    const float* from = po + (w * group + r) * kPartStride;
                    const float mw = from[128], f = mw == -INFINITY ? 0.f : exp2f(mw - mx);   // a pair that has seen no page
                    sum += from[129] * f;
                    const float4 v = *reinterpret_cast<const float4*>(from + c);
                    a.x += v.x * f; a.y += v.y * f; a.z += v.z * f; a.w += v.w * f;
                }
                unsigned char* part = ex + E.part + (uint32_t)((cta * group + r) * kPartStride) * 8u;
                if (a_split > 0) {
                    put_words(part + c * 8, __float_as_uint(a.x), __float_as_uint(a.y), flag);
                    put_words(part + c * 8 + 16, __float_as_uint(a.z), __float_as_uint(a.w), flag);
                    if (c == 0) put_words(part + 128 * 8, __float_as_uint(mx), __float_as_uint(sum), flag);
                    continue;
                }
#pragma unroll 1
                for (int q = 1; q < splits; ++q) {   // the other slices, in order
                    const unsigned char* from = part + (uint32_t)(q * group * kPartStride) * 8u;
                    FlagWords ml, v0, v1;
#pragma unroll 1
                    do { ml = peek_words(from + 128 * 8); v0 = peek_words(from + c * 8); v1 = peek_words(from + c * 8 + 16); }
                    while (!(has_flag(ml, flag) && has_flag(v0, flag) && has_flag(v1, flag)) && wait.again());
                    const float mq = word_f32(ml.a);
                    if (mq == -INFINITY) continue;   // a slice without pages
                    const float m_new = fmaxf(mx, mq), fa = exp2f(mx - m_new), fb = exp2f(mq - m_new);
                    sum = sum * fa + word_f32(ml.b) * fb;
                    a.x = a.x * fa + word_f32(v0.a) * fb; a.y = a.y * fa + word_f32(v0.b) * fb;
                    a.z = a.z * fa + word_f32(v1.a) * fb; a.w = a.w * fa + word_f32(v1.b) * fb;
                    mx = m_new;
                }
                const float n = 1.f / sum;
                put_words(ex + E.attn + (uint32_t)(a_row * QD + (a_head * group + r) * 128 + c) * 4u, pack_bf16x2(a.x * n, a.y * n), pack_bf16x2(a.z * n, a.w * n), flag);
            }
            // (a barrier of the consumers lies between these reads of the slots and the next writes to them: a projection's x, or the one that
            // a CTA without columns of qkv passes; the pages have been read when the partial outputs are complete)
        }
        const int4 mine = tiles[kind];   // first tile, tiles, groups, all tiles
        const int t0 = mine.x, nt = mine.y, G = mine.z;
        const int items = nt * M * 4;    // four channels of a row of a tile
        const float* gain = kind == kOut ? L.ln2 : l + 1 < p.n_layers ? p.layers[l + 1].ln1 : p.final_gain;   // out, down: of the next norm
        float4 gn = make_float4(0.f, 0.f, 0.f, 0.f);
        if (nt == 0) {
            if (kind == kQkv) consumers_sync();   // x and the slots are free for attention
        } else {
            // what the epilogue reads is asked for before the phase's x has arrived
            if ((kind & 1) && tid < items) gn = *reinterpret_cast<const float4*>(gain + (t0 + by_m(tid >> 2)) * 16 + (tid & 3) * 4);
            const unsigned char* w = kind == kQkv ? L.w_qkv : kind == kOut ? L.w_out : kind == kGateUp ? L.w_gate_up : kind == kDown ? L.w_down : p.w_head;
            const __half2* channel_scales = reinterpret_cast<const __half2*>(w + (size_t)mine.w * G * 2048);   // W8: of the channels g, g + 8 of a tile
            const int4 r = ranges[kind * kWarps + warp];
            int tile = r.z, grp = r.w;
            __half2 cs = BITS == 8 && r.x < r.y ? channel_scales[(t0 + tile) * 8 + g] : __half2();
            if (phase > 0) {
                const bool in = kind == kQkv || kind == kHead;
                stage_x(in ? E.x_in : kind == kOut ? E.attn : kind == kGateUp ? E.x_mid : E.mlp, G, kind == kQkv ? flag - 1u : flag,
                        in ? ex + E.ss_in : kind == kGateUp ? ex + E.ss_mid : nullptr);
            }
            // ---- this warp's units
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            const int m = 2 * t;
            if (kind == kHead) *best = make_float4(-INFINITY, -INFINITY, __int_as_float(0x7fffffff), __int_as_float(0x7fffffff));
#pragma unroll 1
            for (int u = r.x; u < r.y;) {
                const int n = min(kUnits<BITS>, min(r.y - u, G - grp));
                stage_units<BITS>(ring, n, acc, lane_base + grp * lane_stride, lane_stride, lane, p.status);
                grp += n;
                u += n;
                if (grp == G || u == r.y) {
                    if (BITS == 8) {
                        const float lo = __low2float(cs), hi = __high2float(cs);
                        acc[0] *= lo; acc[1] *= lo; acc[2] *= hi; acc[3] *= hi;
                        if (u < r.y) cs = channel_scales[(t0 + tile + 1) * 8 + g];
                    }
                    if (kind == kHead) {   // whole tiles
                        const int n = (t0 + tile) * 16 + g;
                        float* to = p.logits + (size_t)m * p.vocab + n;
                        float4 bst = *best;
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                            if (m + e < M) {
                                const float a = acc[e] * inv[m + e], b = acc[2 + e] * inv[m + e];
                                to[(size_t)e * p.vocab] = a; to[(size_t)e * p.vocab + 8] = b;
                                float& v = e ? bst.y : bst.x;
                                int i = __float_as_int(e ? bst.w : bst.z);
                                better(v, i, a, n);
                                better(v, i, b, n + 8);
                                (e ? bst.w : bst.z) = __int_as_float(i);
                            }
                        *best = bst;
                    } else {
                        float* s = slots + (warp + tile) * kSlotFloats;
                        s[m * 16 + g] = acc[0]; s[(m + 1) * 16 + g] = acc[1];
                        s[m * 16 + g + 8] = acc[2]; s[(m + 1) * 16 + g + 8] = acc[3];
                    }
                    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
                    grp = 0;
                    ++tile;
                }
            }
            if (kind == kHead) break;
            consumers_sync();
        }
        // the projection has read x: the pages of attention may lie over it
        if (kind == kQkv && attends && warp < kPairs && lane == 0 && pg0 + pair < pg1) load_page(l, first_page);
        // ---- the warps' parts in order, and what the projection does with the sums
        const bool sparse = nt * G < kWarps;   // warps without a unit
        const uint32_t starved = p.starve == 1 && phase == 0 && t0 == 0 ? 1u : 0u;
#pragma unroll 1
        for (int i = tid; i < ((items + 31) & ~31); i += kConsumers) {
            const bool live = i < items;
            const int c = (i & 3) * 4, m = live ? (i >> 2) - by_m(i >> 2) * M : 0, tile = live ? by_m(i >> 2) : 0;
            const uchar2 span = spans[kind * 32 + tile];
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
            for (int w = span.x; w <= span.y; w += 4) {
                float4 s[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) s[j] = *reinterpret_cast<const float4*>(slots + (min(w + j, (int)span.y) + tile) * kSlotFloats + m * 16 + c);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (w + j <= span.y && !(sparse && ranges[kind * kWarps + w + j].x == ranges[kind * kWarps + w + j].y)) {
                        v.x += s[j].x; v.y += s[j].y; v.z += s[j].z; v.w += s[j].w;
                    }
            }
            if (kind & 1) {   // out, down: the residual stream, the next norm's input and its sum of squares
                float ss = 0.f;
                if (live) {
                    float4* h = reinterpret_cast<float4*>(h_own + m * h_cols + tile * 16 + c);
                    float4 y = *h;
                    y.x += v.x; y.y += v.y; y.z += v.z; y.w += v.w;
                    *h = y;
                    if (i >= kConsumers) gn = *reinterpret_cast<const float4*>(gain + (t0 + tile) * 16 + c);
                    put_words(ex + (kind == kOut ? E.x_mid : E.x_in) + (uint32_t)(m * D + (t0 + tile) * 16 + c) * 4u, pack_bf16x2(y.x * gn.x, y.y * gn.y),
                         pack_bf16x2(y.z * gn.z, y.w * gn.w), flag);
                    ss = y.x * y.x + y.y * y.y + y.z * y.z + y.w * y.w;
                }
                ss += __shfl_xor_sync(0xffffffffu, ss, 1);
                ss += __shfl_xor_sync(0xffffffffu, ss, 2);
                if (live && c == 0) put_word(ex + (kind == kOut ? E.ss_mid : E.ss_in) + (uint32_t)(m * ss_tiles + t0 + tile) * 8u, __float_as_uint(ss), flag);
            } else {
                const float r = inv[m];
                v.x *= r; v.y *= r; v.z *= r; v.w *= r;
                if (kind == kQkv) {
                    if (live) put_words(ex + E.qkv + (uint32_t)(m * QKV + (t0 + tile) * 16 + c) * 4u, pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w), flag - starved);
                } else {   // a tile: 8 gate channels, then the 8 up channels that go with them
                    float4 up;
                    up.x = __shfl_xor_sync(0xffffffffu, v.x, 2); up.y = __shfl_xor_sync(0xffffffffu, v.y, 2);
                    up.z = __shfl_xor_sync(0xffffffffu, v.z, 2); up.w = __shfl_xor_sync(0xffffffffu, v.w, 2);
                    auto act = [](float a, float b) { return a / (1.f + expf(-a)) * b; };
                    if (live && c < 8)
                        put_words(ex + E.mlp + (uint32_t)(m * FF + (t0 + tile) * 8 + c) * 4u, pack_bf16x2(act(v.x, up.x), act(v.y, up.y)),
                             pack_bf16x2(act(v.z, up.z), act(v.w, up.w)), flag);
                }
            }
        }
    }

    // ---- the greedy pick ----------------------------------------------------------------------------------------------------------------
    const float4 bst = tiles[kHead].y ? *best : make_float4(-INFINITY, -INFINITY, __int_as_float(0x7fffffff), __int_as_float(0x7fffffff));
    float top[2] = {bst.x, bst.y};
    int top_i[2] = {__float_as_int(bst.z), __float_as_int(bst.w)};
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, top[e], off);
            const int oi = __shfl_xor_sync(0xffffffffu, top_i[e], off);
            better(top[e], top_i[e], ov, oi);
        }
    float* const bv = reinterpret_cast<float*>(sm + S.best);   // [warp][8]
    int* const bi = reinterpret_cast<int*>(sm + S.best) + kWarps * 8;
    if (g == 0)
#pragma unroll
        for (int e = 0; e < 2; ++e) { bv[warp * 8 + 2 * t + e] = top[e]; bi[warp * 8 + 2 * t + e] = top_i[e]; }
    consumers_sync();
    if (tid < M) {
        float v = bv[tid];
        int i = bi[tid];
#pragma unroll 1
        for (int w = 1; w < kWarps; ++w) better(v, i, bv[w * 8 + tid], bi[w * 8 + tid]);
        put_words(ex + E.best + (uint32_t)(tid * 256 + cta) * 16u, __float_as_uint(v), (uint32_t)i, flag);
    }
    if (cta == 0 && warp < M) {
        float v = -INFINITY;
        int i = 0x7fffffff;
#pragma unroll 1
        for (int k = lane; k < grid; k += 32) {
            const FlagWords c = wait.wait_words(ex + E.best + (uint32_t)(warp * 256 + k) * 16u, flag);
            better(v, i, word_f32(c.a), (int)(uint32_t)c.b);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, off);
            const int oi = __shfl_xor_sync(0xffffffffu, i, off);
            better(v, i, ov, oi);
        }
        if (lane == 0) {
            p.sampled[warp] = i;
            if (p.advance) {   // every CTA has read its token, position and length by now: its candidate came behind
                const int at = p.pos[warp];
                if (at >= 0 && at < p.context_length) p.history[(size_t)warp * p.context_length + at] = p.given ? p.token_in[warp] : p.token[warp];
                p.token[warp] = i;
                p.pos[warp] = at + 1;
                p.ctx[warp] += 1;
                p.out[warp] = i;
            }
        }
    }
}

constexpr int kSmemLimit = 227 * 1024;

int max_tiles(int D, int FF, int Hq, int Hkv) {
    const int grid = sm_count();
    return std::max({ceil_div(D / 16, grid), ceil_div(FF / 8, grid), ceil_div((Hq + 2 * Hkv) * 8, grid)});
}
StepSmem smem_of(int bits, int rows, int D, int FF, int Hq, int Hkv, int stages) {
    return smem_plan(rows, std::max({D, FF, Hq * 128}), Hq / Hkv, ceil_div(D / 16, sm_count()) * 16, max_tiles(D, FF, Hq, Hkv), stages,
                     bits == 4 ? kStageBytes<4> : kStageBytes<8>);
}
// Stages of every warp's ring beside what `rows` rows need; 0: it does not fit.
int ring_stages(int bits, int rows, int D, int FF, int Hq, int Hkv) {
    for (int s = 12; s >= 2; --s)
        if ((int)smem_of(bits, rows, D, FF, Hq, Hkv, s).total <= kSmemLimit) return s;
    return 0;
}

// Slices that the pages of a row are cut into. A slice takes seven pages at a time (a round, 1.2 to 1.6 us: a pair of warps asks for its next page
// when it has used the last), and the CTA of the first slice adds the others' outputs one by one (0.4 us each): s rounds fewer against s slices
// more meet at the root of three times the rounds that one slice would have. Step of four layers, us, with as many slices: W4 of width 1024, one
// row, 1000 tokens 1: 148, 4: 120, 6: 115, 9: 121; 3000 tokens 4: 137, 9: 129, 24: 146; 8000 tokens 8: 159, 16: 150, 72: 225; 32000 tokens
// 18: 230, 36: 209, 74: 250; W8 of width 2048, eight rows, 215 tokens 1: 201, 2: 193; W4 of width 3072, four rows 206, 201.
int slices(int max_ctx, int rows, int n_kv_heads) {
    const int rounds = ceil_div(ceil_div(max_ctx, 16), kPairs), most = std::min(rounds, std::max(1, sm_count() / (rows * n_kv_heads)));
    int s = 1;
    while (s < most && s * s < 3 * rounds) ++s;
    return s;
}

}  // namespace

int quant_step_max_rows(int bits, int n_layers, int D, int FF, int Hq, int Hkv, int vocab) {
    if (n_layers < 1 || n_layers > kStepMaxLayers || D % 128 || FF % 128 || vocab % 16 || Hq % Hkv || Hq / Hkv > 8 || sm_count() > 256) return 0;
    if (max_tiles(D, FF, Hq, Hkv) > 32) return 0;
    int n = 0;
    // W8 rings of two stages lose against a kernel per projection (width 3072, 7 and 8 rows 376 -> 386, 395 -> 439 us a step of six layers).
    // With three it is the rows of the longest projection that decide, which every CTA reads: 6 x 9216 values lose at every length (four layers,
    // 20 / 300 / 3000 / 12000 tokens, kernel by kernel / here: 264 / 267, 272 / 281, 314 / 332, 488 / 529), 8 x 6144 (196 / 180, 200 / 189,
    // 232 / 231) and 5 x 9216 (264 / 245, 270 / 258; 3000 tokens: quant_step_pays) win.
    const int k_max = std::max({D, FF, Hq * 128}), most_x = bits == 4 ? INT_MAX : 48 * 1024;
    while (n < kStepMaxRows && (n + 1) * Hkv <= sm_count() && (n + 1) * k_max <= most_x && ring_stages(bits, n + 1, D, FF, Hq, Hkv) >= (bits == 4 ? 2 : 3)) ++n;
    return n;
}
// Whether a step is faster here than kernel by kernel: what attention takes longer, in us of a layer, against what the rest is faster (widths 1024,
// 2048 and 3072, 1 to 8 rows: 11.5 in W4; in W8 5.2 while attention there is one kernel, and 7.8 where it has become three). Here it is rounds of pages and slices to add up (see `slices`), and all rows have as
// many CTAs; there long rows have more splits and two pages per warp under way: at least 0.6 us per 1000 tokens of the longest row, or all
// pages at 6.1 TB/s. Four layers, us, kernel by kernel / here: W4 of width 3072, 8 rows at 3000 tokens 409 / 330, 8000 511 / 502, 16000
// 713 / 805; one of 8000 among short ones 364 / 458, of 32000 508 / 1224; 4 rows at 8000 366 / 330, 16000 491 / 496; W4 of width 2048, 8 rows at
// 16000 424 / 423, 32000 574 / 652; W8 of width 2048, 8 rows at 3000 232 / 231, 6000 298 / 275, one of 2000 210 / 211, one of 3000 217 / 224, 4 rows at
// 16000 340 / 281, one of 16000 255 / 270; W8 of width 3072, 5 rows at 1000 278 / 273, 3000 307 / 310, 4 rows at 3000 299 / 289; one row is faster
// here at every length up to 32000 (W4 of width 3072 there 445 / 380, W8 of widths 1024 and 3072 at 3000 146 / 140, 275 / 273).
bool quant_step_pays(int bits, int rows, int n_q_heads, int n_kv_heads, int max_ctx, int64_t all_ctx) {
    const int s = slices(max_ctx, rows, n_kv_heads);
    const double here = 1.5 * ceil_div(ceil_div(max_ctx, 16), kPairs * s) + 0.3 * (s - 1);
    const double there = std::max(1.5 + 0.0006 * max_ctx, (double)all_ctx * n_kv_heads * 512 / 6.1e6);
    return here - there < (bits == 4 ? 11.5 : attention_step_splits(max_ctx, rows, n_q_heads, n_kv_heads) ? 5.2 : 7.8);
}
size_t quant_step_exchange_bytes(int D, int FF, int Hq, int Hkv) { return exchange_layout(D, FF, Hq, Hkv).total; }

int quant_step_launch(int bits, QuantStepParams p, int max_ctx, cudaStream_t st) {
    void (*const kern)(const QuantStepParams) = bits == 4 ? quant_step_kernel<4> : quant_step_kernel<8>;
    static PerDeviceOnce attr_once;
    if (attr_once.first_time()) {
        GPTRS_CUDA_OK(cudaFuncSetAttribute(quant_step_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
        GPTRS_CUDA_OK(cudaFuncSetAttribute(quant_step_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
    }
    const int grid = sm_count();
    p.stages = ring_stages(bits, p.rows, p.D, p.FF, p.Hq, p.Hkv);
    p.ex = exchange_layout(p.D, p.FF, p.Hq, p.Hkv);
    p.sm = smem_of(bits, p.rows, p.D, p.FF, p.Hq, p.Hkv, p.stages);
    p.splits = slices(max_ctx, p.rows, p.Hkv);
    step_wait_limits(&p.ring_polls, &p.flag_polls, &p.starve);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = p.sm.total;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeCooperative;   // all CTAs co-resident: they wait for each other's words
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
    if (e != cudaSuccess) return fail(GPTRS_EXECUTION, std::string("cooperative launch failed: ") + cudaGetErrorString(e));
    return GPTRS_OK;
}

}  // namespace gptrs
