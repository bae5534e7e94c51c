// f32 matmul on the tcgen05 tensor cores: y[M][N] = act(x[M][K] . w[K][N] + bias) + residual for many rows
// (functional::matmul, crates/gpt-rs/src/ops/functional/linalg.rs:109-127; Linear::forward, nn/layers/linear.rs:50-71).
//
// An f32 value of 2^-110 and more is the sum of three bf16 values (8 significant bits each, the remainders exact in f32): v = v1 + v2 + v3. The product
// keeps the six terms of at least 2^-18 of it, w1x1 + (w1x2 + w2x1 + w2x2 + w1x3 + w3x1); what is left out is below 2^-26, less than
// the rounding of one f32 product. Products of bf16 values are exact; what the tensor core loses is in the order of its sums, so the
// leading term w1x1 is summed in tensor memory over 64 k only and then added to f32 registers, and the five small terms, 2^-8 of the
// whole and less, have an accumulator of their own that is read once.
//
// CTA: 128 output channels (M side of the MMA) x BN rows: 128 rows with 16 splitting warps, one CTA per SM; up to 64 rows with 8 and two
// CTAs per SM. Per stage of 32 k the splitting warps load f32 from global memory (ahead, in registers), split, and
// store the planes K-major in the 128-byte swizzle (a row holds 32 k of planes 1 and 2, a second tile plane 3); the last of
// them also issues the 12 MMAs. Stages and two leading accumulators alternate, so that the sums of earlier stages go to registers and the next stage is split
// while the tensor core works. K is split over a cluster where the output tiles do not fill the SMs; the parts meet in the shared memory
// of the CTA that owns the row and are added in the order of the ranks.
//
// Relative error against 64 bits (random operands, K 768 / 3072, N 768, 937 rows): 5.3e-8 / 9.6e-8, plain f32 fused multiply-adds 5.8e-8 / 1.15e-7.
// Operands of one sign do worse, because the tensor core cuts its sums where f32 arithmetic rounds them (magnitudes of random operands,
// N 2304, K 768 / 3072: 64 rows 8.9e-8 / 8.9e-8, 937 rows, whose K is not split, 9.5e-8 / 1.23e-7; the kernel for few rows 4.7e-8 / 4.5e-8,
// a library's f32 matmul 3.7e-7 / 1.5e-7 to 7.4e-7). Sums taken after 32 k instead of 64 would halve the cut and double the additions.
//
// Infinities, NaN and magnitudes from 3.39e38 on, which a bf16 cannot hold, become NaN in the remainders and so in every sum that they
// enter, and a product past the f32 range can be an infinity of one sign in each accumulator: sums that are not finite are computed again
// with plain f32 fused multiply-adds, the others keep what they have. Below 2^-110 the third term, then the second, falls under what a
// bf16 holds: an operand is then off by up to 2^-134, which against the sum's other products counts only where all of them are as small.
#include "split_f32.cuh"
#include "umma_common.cuh"

namespace gptrs {
// umma_matmul.cu: the library's per-device status word, and the polls of a wait and the test switch of gptrs_cuda_debug_matmul_fault
int* matmul_status_word();
void matmul_wait_limits(uint32_t* spin_limit, int* starve);
namespace {

constexpr int kSfBK = 32;
constexpr int kSfTile = 128 * 128;   // bytes of 128 rows of 128

// 8 consecutive k of a row -> three planes
__device__ __forceinline__ void split3(const float (&v)[8], uint4 (&o)[3]) {
    uint32_t p[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float a = v[2 * i], b = v[2 * i + 1];
        p[0][i] = pack_bf16x2(a, b);
        a -= bf16_lo(p[0][i]); b -= bf16_hi(p[0][i]);
        p[1][i] = pack_bf16x2(a, b);
        a -= bf16_lo(p[1][i]); b -= bf16_hi(p[1][i]);
        p[2][i] = pack_bf16x2(a, b);
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) o[j] = make_uint4(p[j][0], p[j][1], p[j][2], p[j][3]);
}

template <int BN>
struct SfShape {
    static constexpr int kWarps = BN == 128 ? 16 : 8;             // 16 per SM, so that each may have 128 registers a thread
    static constexpr int kThreads = 32 * kWarps;
    static constexpr int kStages = BN == 128 ? 3 : 2;
    static constexpr int kStageBytes = 2 * (kSfTile + BN * 128);  // w planes 1 2, w plane 3, x planes 1 2, x plane 3
    static constexpr size_t kSmem = (size_t)kStages * kStageBytes + 1024;
};

// EARLY: the weights were there before the kernel in front began. DEBUG: the wait limits and the test switch of the call (as reads of the
// parameters they cost the others 3 %)
template <int BN, bool EARLY, bool DEBUG = false>
__global__ void __launch_bounds__(SfShape<BN>::kThreads, BN == 128 ? 1 : 2) split_f32_kernel(const SplitF32Params p) {
    using Shape = SfShape<BN>;
    const uint32_t limit = DEBUG ? p.spin_limit : kSpinLimit;
    constexpr int kWarps = Shape::kWarps, kSplitters = 32 * kWarps, STAGES = Shape::kStages, kXTile = BN * 128, kStage = Shape::kStageBytes;
    constexpr uint32_t kCols = BN == 128 ? 512 : BN == 64 ? 256 : 128;
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | (8u << 24);
    constexpr int kWItems = 512 / kSplitters;        // 8-k chunks of weights per thread and stage
    constexpr int kSets = kWItems == 1 ? 2 : 1;      // stages that are loaded ahead
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES];
    __shared__ uint32_t tmem_holder;
    unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b = blockIdx.z / p.m_tiles, m0 = (blockIdx.z % p.m_tiles) * BN, n0 = blockIdx.x * 128;
    const int k_tiles = p.K / kSfBK;
    const int kt0 = (int)((int64_t)k_tiles * blockIdx.y / p.n_split), n_k = (int)((int64_t)k_tiles * (blockIdx.y + 1) / p.n_split) - kt0;
    const float* x = p.x + b * p.x_step;
    const float* w = p.w + (size_t)b * p.K * p.N;
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], kSplitters); mbar_init(&empty[s], 1); }
        mbar_fence_init();
        fence_proxy_async();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_holder)), "r"(kCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_holder;
    pdl_launch_dependents();

    // this thread's share of a stage: channel wn, 8-k chunks wc and (with 8 warps) wc + 2 of the weights; chunk xc of row xr. Channels and
    // rows past the end repeat the last one; their sums are dropped.
    const int wn = tid & 127, wc = tid >> 7, xr = tid >> 2, xc = tid & 3;
    const bool x_has = xr < BN;
    const uint32_t w_row = (uint32_t)p.N * 4, w_stage = w_row * kSfBK;   // bytes; the matrix has less than 2^32
    uint32_t w_at = (uint32_t)kt0 * w_stage + (uint32_t)wc * 8 * w_row + (uint32_t)min(n0 + wn, p.N - 1) * 4;
    const float* x_at = x + (size_t)min(m0 + xr, p.M - 1) * p.ldx + kt0 * kSfBK + xc * 8;
    struct Raw { float w[kWItems][8], x[8]; };
    Raw raw[kSets];
    auto load_w = [&](Raw& to) {
#pragma unroll
        for (int i = 0; i < kWItems; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) to.w[i][j] = __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(w) + (w_at + (uint32_t)(16 * i + j) * w_row)));
        w_at += w_stage;
    };
    auto load_x = [&](Raw& to) {
        if (x_has) {
            const float4 lo = *reinterpret_cast<const float4*>(x_at), hi = *reinterpret_cast<const float4*>(x_at + 4);
            to.x[0] = lo.x; to.x[1] = lo.y; to.x[2] = lo.z; to.x[3] = lo.w; to.x[4] = hi.x; to.x[5] = hi.y; to.x[6] = hi.z; to.x[7] = hi.w;
        }
        x_at += kSfBK;
    };
    bool failed = false;
    float acc[32];
    const int quarter = warp & 3, c_lo = (warp >> 2) * 32;
    const bool sums = warp < BN / 8;   // four warps take the sums of 32 columns (rows of y)
    {
        if constexpr (!EARLY) pdl_wait();   // else the weights travel while the kernel in front still runs
#pragma unroll
        for (int i = 0; i < kSets; ++i)
            if (i < n_k) load_w(raw[i]);
        pdl_wait();
#pragma unroll
        for (int i = 0; i < kSets; ++i)
            if (i < n_k) load_x(raw[i]);
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = 0.f;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c_lo;
        auto add_columns = [&](int at) {
            float v[32];
            tmem_ld_32(lane_base + (uint32_t)at, v);
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[i] += v[i];
        };
        unsigned char* const w_out = smem + wn * 128;
        unsigned char* const x_out = smem + 2 * kSfTile + xr * 128;
        const int w_sw = wn & 7, x_sw = xr & 7;
        // Stages 2c and 2c + 1 share leading accumulator c & 1: it is taken once stage 2c + 1 is complete, before this thread lets
        // stage 2c + 4 begin.
        int taken = 0, buf = 0;
        uint32_t parity = 1;   // of the last use of a stage's buffer
        auto issue = [&](int s, uint32_t st) {
            // K steps of 16 are 2 descriptor units apart; plane 2 lies 4 units behind plane 1
            const uint64_t w12 = make_smem_desc(st), w3 = make_smem_desc(st + kSfTile);
            const uint64_t x12 = make_smem_desc(st + 2 * kSfTile), x3 = make_smem_desc(st + 2 * kSfTile + kXTile);
            const uint32_t lead = tmem + (uint32_t)(((s >> 1) & 1) * BN), rest = tmem + 2u * BN;
#pragma unroll
            for (int k = 0; k < 4; k += 2) {
                umma_bf16(lead, w12 + k, x12 + k, kIdesc, (s & 1) || k > 0 ? 1u : 0u);
                umma_bf16(rest, w3 + k, x12 + k, kIdesc, s > 0 || k > 0 ? 1u : 0u);
                umma_bf16(rest, w12 + k, x3 + k, kIdesc, 1u);
                umma_bf16(rest, w12 + 4 + k, x12 + 4 + k, kIdesc, 1u);
                umma_bf16(rest, w12 + 4 + k, x12 + k, kIdesc, 1u);
                umma_bf16(rest, w12 + k, x12 + 4 + k, kIdesc, 1u);
            }
            umma_commit(&empty[buf]);
        };
        auto step = [&](int s, Raw& r) {
            if (s >= STAGES) {   // the MMAs of stage s - STAGES are complete
                if (!failed && !mbar_wait_relaxed(&empty[buf], parity, limit)) failed = true;
                tc_fence_after();
            }
            if (!(s & 1) && s >= 4) {
                if (sums) add_columns((taken & 1) * BN);
                ++taken;
            }
            const int st = buf * kStage;
#pragma unroll
            for (int i = 0; i < kWItems; ++i) {
                uint4 o[3];
                split3(r.w[i], o);
                const int c = wc + 2 * i;
                *reinterpret_cast<uint4*>(w_out + st + ((c ^ w_sw) << 4)) = o[0];
                *reinterpret_cast<uint4*>(w_out + st + (((c + 4) ^ w_sw) << 4)) = o[1];
                *reinterpret_cast<uint4*>(w_out + st + kSfTile + ((c ^ w_sw) << 4)) = o[2];
            }
            if (s + kSets < n_k) load_w(r);
            if (x_has) {
                uint4 o[3];
                split3(r.x, o);
                *reinterpret_cast<uint4*>(x_out + st + ((xc ^ x_sw) << 4)) = o[0];
                *reinterpret_cast<uint4*>(x_out + st + (((xc + 4) ^ x_sw) << 4)) = o[1];
                *reinterpret_cast<uint4*>(x_out + st + kXTile + ((xc ^ x_sw) << 4)) = o[2];
            }
            if (s + kSets < n_k) load_x(r);
            fence_proxy_async();
            tc_fence_before();
            mbar_arrive(&full[buf]);
            if (warp == kWarps - 1) {
                if (!failed && !mbar_wait_relaxed(&full[buf], parity ^ 1, limit)) failed = true;
                tc_fence_after();
                if (lane == 0 && !failed && !(DEBUG && p.debug_starve && s == 0)) issue(s, smem_u32(smem) + (uint32_t)st);
                __syncwarp();
            }
            if (++buf == STAGES) { buf = 0; parity ^= 1; }
        };
#pragma unroll 1
        for (int s = 0; s < n_k; s += kSets) {
            step(s, raw[0]);
            if constexpr (kSets == 2)
                if (s + 1 < n_k) step(s + 1, raw[kSets - 1]);
        }
        for (int s = max(n_k - STAGES, 0); s < n_k; ++s)
            if (!failed && !mbar_wait_relaxed(&empty[s % STAGES], (uint32_t)(s / STAGES) & 1u, limit)) failed = true;
        tc_fence_after();
        if (sums) {
#pragma unroll 1
            for (; taken < (n_k + 1) / 2; ++taken) add_columns((taken & 1) * BN);
            add_columns(2 * BN);
        }
    }
    if (failed && lane == 0) atomicExch(p.status, 3);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kCols) : "memory");
    // Row r of the tile belongs to rank r % S of the cluster; its receive slots [rank][row / S][128] lie over the stages, so nobody
    // pushes before everybody's MMAs have read theirs.
    const int S = p.n_split, rank = S > 1 ? (int)cluster_ctarank() : 0, rows_max = (BN + S - 1) / S;
    if (S > 1) cluster_sync_all();
    auto push = [&](int r, int col, float v) {
        const uint32_t at = smem_u32(smem) + (uint32_t)(((rank * rows_max + r / S) * 128 + col) * 4);
        if (S > 1) st_cluster_f32(map_to_cta(at, (uint32_t)(r % S)), v);
        else asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(at), "f"(v) : "memory");
    };
    const int col = quarter * 32 + lane;
    if (sums) {
        uint32_t special = 0;   // rows whose sum is not finite
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            push(c_lo + i, col, acc[i]);
            special |= fabsf(acc[i]) < INFINITY ? 0u : 1u << i;
        }
        const int n = n0 + col, k_hi = (kt0 + n_k) * kSfBK;
        for (; special; special &= special - 1) {
            const int r = c_lo + __ffs(special) - 1, m = m0 + r;
            if (m >= p.M || n >= p.N) continue;
            float sum = 0.f;
#pragma unroll 1
            for (int k = kt0 * kSfBK; k < k_hi; ++k) sum = fmaf(x[(size_t)m * p.ldx + k], w[(size_t)k * p.N + n], sum);
            push(r, col, sum);
        }
    }
    if (S > 1) cluster_sync_all();
    else __syncthreads();
    const float* got = reinterpret_cast<const float*>(smem);
#pragma unroll 2
    for (int j = tid; j < rows_max * 128; j += Shape::kThreads) {
        const int local = j >> 7, r = rank + S * local, m = m0 + r, n = n0 + (j & 127);
        if (r >= BN || m >= p.M || n >= p.N) continue;
        float v = got[j];
        for (int q = 1; q < S; ++q) v += got[q * rows_max * 128 + j];
        if (p.bias) v += p.bias[n];
        if (p.act == 1) v = (0.5f * v) * (1.f + erff(v / 1.4142135f));
        if (p.dense.kind || p.dense.softcap > 0.f) v = dense_act(p.dense, v);
        if (p.residual) v += p.residual[(size_t)m * p.N + n];
        p.y[b * p.y_step + (size_t)m * p.ldy + n] = v;
    }
}

// How many CTAs of a cluster size run at one time (clusters leave SMs of a GPC over), asked once per device.
template <int BN>
int64_t slots_of(int cluster) {
    static std::atomic<int> known[kMaxDevices][9];
    std::atomic<int>& slot = known[current_device() & (kMaxDevices - 1)][cluster];
    int n = slot.load(std::memory_order_relaxed);
    if (n == 0) {
        using Shape = SfShape<BN>;
        n = (BN == 128 ? 1 : 2) * sm_count();
        if (cluster > 1) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(1, (unsigned)cluster, 1);
            cfg.blockDim = dim3(Shape::kThreads);
            cfg.dynamicSmemBytes = Shape::kSmem;
            cudaLaunchAttribute attr;
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = 1; attr.val.clusterDim.y = (unsigned)cluster; attr.val.clusterDim.z = 1;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, split_f32_kernel<BN, true>, &cfg) != cudaSuccess) { cudaGetLastError(); clusters = 0; }
            n = clusters > 0 ? clusters * cluster : 1;
        }
        slot.store(n, std::memory_order_relaxed);
    }
    return n;
}

// K parts: as many as make the last CTA end soonest, with the set-up, the reduction and the epilogue of a CTA as so many stages.
template <int BN>
void plan(SplitF32Params& p) {
    p.m_tiles = ceil_div(p.M, BN);
    const int64_t ctas = (int64_t)ceil_div(p.N, 128) * p.m_tiles * p.batch, k_tiles = p.K / kSfBK;
    int64_t best = 1ll << 60;
    for (int s = 1; s <= 8 && s <= k_tiles; ++s) {
        const int64_t slots = slots_of<BN>(s), t = ((ctas * s + slots - 1) / slots) * ((k_tiles + s - 1) / s + 8 + 2 * (s > 1));
        if (t < best) { best = t; p.n_split = s; }
    }
}

template <int BN>
int launch(SplitF32Params p, cudaStream_t st) {
    using Shape = SfShape<BN>;
    static PerDeviceOnce attr_once;
    if (attr_once.first_time())
        for (auto k : {split_f32_kernel<BN, true>, split_f32_kernel<BN, false>, split_f32_kernel<BN, false, true>})
            GPTRS_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape::kSmem));
    plan<BN>(p);
    const int64_t z = (int64_t)p.m_tiles * p.batch;
    if (z > 65535) return fail(GPTRS_UNIMPLEMENTED, "f32 matmul: too many rows in one launch");
    auto kern = p.debug_starve || p.spin_limit != kSpinLimit ? split_f32_kernel<BN, false, true> : p.w_constant ? split_f32_kernel<BN, true> : split_f32_kernel<BN, false>;
    return launch_kernel(kern, dim3((unsigned)ceil_div(p.N, 128), (unsigned)p.n_split, (unsigned)z), dim3(Shape::kThreads), Shape::kSmem, st, p.n_split, p);
}

}  // namespace

// K in whole stages, rows that 16-byte loads can read, weights that a 32-bit byte offset can reach. The line against the kernel for few
// rows: that one makes a CTA of every 8 rows and 128 columns, and is done as fast while those are few (us, it / this one, K 768:
// N 768, 24 rows 9.9 / 11.7, 64 rows 12.7 / 13.2, 100 rows 22.6 / 15.1; N 2304, 16 rows 11.2 / -, 24 rows about 20 / 12.6,
// 937 rows 798 / 44.7; N 3072, 24 rows about 24 / 14.0, 937 rows 1075 / 91; K 3072, N 768, 24 rows 17.8 / 21.1, 100 rows 39 / 27). With a
// small K those CTAs are short (K 32, N 4096, 64 and 300 rows 5.0 / 11.1, 13.7 / 12.8; K 64, N 256, 937 rows 11.9 / 13.7; K 64, N 8192,
// 24 and 64 rows 7.4 / 9.4, 18.6 / 12.3; K 128, N 1024, 64 and 300 rows 6.9 / 10.8, 20.7 / 12.5; K 256, N 1024, 64 rows 16.2 / 10.2): the
// line is at 16384 CTAs x K.
bool split_f32_line(int64_t m, int64_t n, int64_t k) {
    const int64_t few_row_ctas = (int64_t)ceil_div(m, 8) * ceil_div(n, 128);
    return m >= kSplitF32Rows && few_row_ctas > 48 && few_row_ctas * k >= 16384;
}
bool split_f32_takes(const SplitF32Params& p) {
    return split_f32_line(p.M, p.N, p.K) && p.K % kSfBK == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15) == 0 && ((p.ldx | p.x_step) & 3) == 0 &&
           (int64_t)p.K * p.N < (1ll << 30);
}

int split_f32_matmul(SplitF32Params p, cudaStream_t st) {
    if (!p.status) p.status = matmul_status_word();
    if (!p.status) return fail(GPTRS_EXECUTION, "no status word");
    matmul_wait_limits(&p.spin_limit, &p.debug_starve);
    if (p.M <= 32) return launch<32>(p, st);
    if (p.M <= 64) return launch<64>(p, st);
    return launch<128>(p, st);
}

}  // namespace gptrs
