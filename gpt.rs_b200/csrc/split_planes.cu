// y[M][N] = act(x[M][K] . w[K][N] + bias) + residual in f32 on the tcgen05 tensor cores, as split_f32_kernel does it (three bf16 planes per
// operand, the six products of at least 2^-18, the leading one summed in tensor memory over 64 k (in tiles of 32 rows over 16) and then in f32
// registers, the others in an accumulator of their own; sums that are not finite once more in plain f32), for operands whose planes lie in memory: a model's weights split
// once, and the rows of a pass split once per projection instead of once per column tile.
//
// split_f32_kernel splits inside its tiles: 512 threads load, split, store and fence every 32 k, 2900 cycles a stage, of which the MMAs are 770.
// Here a loader warp requests the planes by TMA, one warp issues the MMAs and eight warps add up the leading sums beside them. CTA: 128 output
// channels (M side of the MMA) x BN rows, stages of 64 k in the 128-byte swizzle (two blocks of planes 1 and 2 of 32 k each, one block of plane
// 3). What bounds it: the MMAs, 24 x BN / 2 cycles a stage (0.95 us with 128 rows), and what a CTA does once, 7 to 10 us. The weights' first
// stages are under way before the kernel in front has ended, and the norms and the GELU leave the planes of their rows themselves.
// K is split over a cluster where the output tiles do not fill the SMs, the parts meet in the shared memory of the CTA that owns the row; the
// epilogue then takes four neighbouring channels per thread (a channel per thread and scalar residuals took 10 to 17 us more at 937 rows).
// Tensor cores cut their sums where f32 arithmetic rounds them: operands of one sign, leading sums over 64 k, are off by twice what plain f32
// leaves. With sums of 16 k, one MMA each, nothing is cut but an MMA's own sum, and four of them are added in pairs. Where the kernel for few rows would
// be taken without planes (split_f32_line), such tiles alone are taken. Error against 64 bits over the sum of magnitudes, that kernel / tiles of
// 32 rows over 64 k / over 16 k, 64 rows, N 768: one sign, K 768 4.6e-8 / 8.9e-8 / 4.7e-8, K 3072 4.6e-8 / 8.9e-8 / 4.7e-8; either sign 5.8e-9 / 5.1e-9 /
// 4.3e-9 and 4.2e-9 / - / 2.6e-9. A pass of four layers of width 256, 512, 768 at 24 rows, us, over 64 k / over 16 k: 209 / 214, 237 / 243,
// 299 / 302; without planes 260, 321, 382.
// Pieces of a third of a stage, in rings of 6 to 11, bring nothing: what the loads take is hidden with two stages.
// GPT-2 small, us, split_f32_kernel / this: at 937 rows qkv 47 / 20, attention output 33 / 16, MLP in 96 / 32, MLP out 83 / 32; at 64 rows
// qkv 11 / 7.5, MLP out 16 / 10.
#include "matmul_common.cuh"
#include "split_f32.cuh"
#include "split_planes.cuh"
#include "umma_common.cuh"

namespace gptrs {
// umma_matmul.cu: the library's per-device status word, and the polls of a wait and the test switch of gptrs_cuda_debug_matmul_fault
int* matmul_status_word();
void matmul_wait_limits(uint32_t* spin_limit, int* starve);
namespace {

constexpr int kBlock = 128 * 128;   // bytes of 128 rows of 128

__device__ __forceinline__ void split3(float v, uint32_t (&o)[3]) {   // bf16 bits of the three terms
    float r = v;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const __nv_bfloat16 b = __float2bfloat16_rn(r);
        o[i] = (uint32_t)__bfloat16_as_ushort(b);
        r -= __bfloat162float(b);
    }
}

// four neighbouring k of a row
__device__ __forceinline__ void store_planes(__nv_bfloat16* planes, int rows, int K, int row, int k, const float4& v) {
    uint32_t a[3], b[3], c[3], d[3];
    split3(v.x, a); split3(v.y, b); split3(v.z, c); split3(v.w, d);
    __nv_bfloat16* at = planes + (size_t)row * 2 * K + (k >> 5) * 64 + (k & 31);
    *reinterpret_cast<uint2*>(at) = make_uint2(a[0] | b[0] << 16, c[0] | d[0] << 16);
    *reinterpret_cast<uint2*>(at + 32) = make_uint2(a[1] | b[1] << 16, c[1] | d[1] << 16);
    *reinterpret_cast<uint2*>(planes + (size_t)rows * 2 * K + (size_t)row * K + k) = make_uint2(a[2] | b[2] << 16, c[2] | d[2] << 16);
}

struct SplitParams { const float* src; __nv_bfloat16 *p12, *p3; int rows, K, N; };
// a thread: four neighbouring k of a row
__global__ void __launch_bounds__(256) split_rows_kernel(const SplitParams p) {
    pdl_launch_dependents();
    pdl_wait();
    const int quarter = p.K >> 2;
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= (int64_t)p.rows * quarter) return;
    const int row = (int)(i / quarter), k = (int)(i - (int64_t)row * quarter) * 4;
    store_planes(p.p12, p.rows, p.K, row, k, *reinterpret_cast<const float4*>(p.src + (size_t)row * p.K + k));
}
// w [K][N]: 32 x 32 tiles through shared memory, rows of the planes are the columns of w
__global__ void __launch_bounds__(256) split_weights_kernel(const SplitParams p) {
    __shared__ float tile[32][33];
    const int n0 = blockIdx.x * 32, k0 = blockIdx.y * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int i = ty; i < 32; i += 8) tile[i][tx] = n0 + tx < p.N ? p.src[(size_t)(k0 + i) * p.N + n0 + tx] : 0.f;
    __syncthreads();
    for (int i = ty; i < 32; i += 8) {
        const int n = n0 + i;
        if (n >= p.N) continue;
        uint32_t o[3];
        split3(tile[tx][i], o);
        __nv_bfloat16* at = p.p12 + (size_t)n * 2 * p.K + (k0 >> 5) * 64 + tx;
        at[0] = __ushort_as_bfloat16((unsigned short)o[0]);
        at[32] = __ushort_as_bfloat16((unsigned short)o[1]);
        p.p3[(size_t)n * p.K + k0 + tx] = __ushort_as_bfloat16((unsigned short)o[2]);
    }
}

struct KernelParams {
    CUtensorMap w12, w3, x12, x3;
    PlanesMatmul q;
    int n_split;
    uint32_t spin_limit;
    int starve;         // test switch: the products of the first stage are never begun
};

// 32 lanes x 16 columns of this warp's quarter of the tensor memory
__device__ __forceinline__ void tmem_ld_16(uint32_t at, float (&v)[16]) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                   "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(at));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

constexpr int kThreads = 320;   // warps 0-7 sums and epilogue, 8 loader, 9 MMA + tensor memory
template <int BN> constexpr int kStages = BN >= 128 ? 2 : 3;   // of 64 k
template <int BN> constexpr int kLeads = BN == 32 ? 4 : 1;     // leading sums of a stage (four of 64 rows do not fit beside three stages' others)
template <int BN> constexpr int kStageBytes = 3 * kBlock + 3 * BN * 128;

// DEBUG: the wait limits and the test switch of the call
template <int BN, bool DEBUG = false>
__global__ void __launch_bounds__(kThreads, 1) planes_matmul_kernel(const __grid_constant__ KernelParams kp) {
    const uint32_t limit = DEBUG ? kp.spin_limit : kSpinLimit;
    constexpr int S = kStages<BN>, L = kLeads<BN>, kStage = kStageBytes<BN>, kX = BN * 128, kSumCols = BN >= 64 ? BN / 2 : 32;   // columns of a summing thread
    constexpr int kSumWarps = 4 * (BN / kSumCols);
    constexpr uint32_t kCols = (S * L + 1) * BN > 256 ? 512 : 256;
    static_assert((S * L + 1) * BN <= (int)kCols && (L == 1 || (L == 4 && kSumCols == 32)));
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | (8u << 24);
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[S], done[S], lead_empty[S];
    __shared__ uint32_t tmem_holder;
    unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const PlanesMatmul& p = kp.q;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.x * 128, m0 = blockIdx.z * BN;
    const int k_tiles = p.K / 64;
    const int kt0 = k_tiles * (int)blockIdx.y / kp.n_split, n_k = k_tiles * ((int)blockIdx.y + 1) / kp.n_split - kt0;
    if (tid == 0) {
        for (int s = 0; s < S; ++s) { mbar_init(&full[s], 1); mbar_init(&done[s], 1); mbar_init(&lead_empty[s], 32 * kSumWarps); }
        mbar_fence_init();
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_holder)), "r"(kCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_holder;
    pdl_launch_dependents();
    bool failed = false;
    auto wait = [&](uint64_t* bar, uint32_t parity) {
        if (!failed && !mbar_wait_relaxed(bar, parity, limit)) failed = true;
        failed = __any_sync(0xffffffffu, failed);
        return !failed;
    };
    float acc[kSumCols];
    const int quarter = warp & 3, c_lo = (warp >> 2) * kSumCols;
    const bool sums = warp < kSumWarps;
    if (warp == 8) {
        auto load = [&](int it, bool w, bool x) {   // lane 0; the weights are constant: their first stages travel while the kernel in front still runs
            const int s = it % S, kt = kt0 + it;
            unsigned char* at = smem + s * kStage;
            const uint32_t bar = smem_u32(&full[s]);
            if (w) {
                mbar_expect_tx_addr(bar, kStage);
                tma_load_2d(at, &kp.w12, kt * 128, n0, bar);
                tma_load_2d(at + kBlock, &kp.w12, kt * 128 + 64, n0, bar);
                tma_load_2d(at + 2 * kBlock, &kp.w3, kt * 64, n0, bar);
            }
            if (x) {
                tma_load_2d(at + 3 * kBlock, &kp.x12, kt * 128, m0, bar);
                tma_load_2d(at + 3 * kBlock + kX, &kp.x12, kt * 128 + 64, m0, bar);
                tma_load_2d(at + 3 * kBlock + 2 * kX, &kp.x3, kt * 64, m0, bar);
            }
        };
        if (lane == 0)
            for (int it = 0; it < min(S, n_k); ++it) load(it, true, false);
        pdl_wait();
        if (lane == 0)
            for (int it = 0; it < min(S, n_k); ++it) load(it, false, true);
        __syncwarp();
        int last = min(S, n_k);
        for (int it = S; it < n_k; ++it) {
            if (!wait(&done[it % S], (uint32_t)(it / S - 1) & 1u)) break;
            if (lane == 0) load(it, true, true);
            __syncwarp();
            last = it + 1;
        }
        for (int i = max(last - S, 0); i < last; ++i) mbar_wait_relaxed(&full[i % S], (uint32_t)(i / S) & 1u, limit);   // what is in flight writes this CTA's shared memory
    } else if (warp == 9) {
        // One elected thread waits and issues for the whole loop: with the warp voting at every wait, lane 0 issuing and a commit per consumer, a
        // stage of 128 rows took 1.45 us instead of 0.95, one of 32 rows 1.25 instead of 0.68.
        if (elect_one()) {
            int s = 0;
            uint32_t phase = 0;
            for (int it = 0; it < n_k; ++it) {
                if (it >= S && !mbar_wait_relaxed(&lead_empty[s], phase ^ 1u, limit)) { failed = true; break; }
                if (!mbar_wait_relaxed(&full[s], phase, limit)) { failed = true; break; }
                if (DEBUG && kp.starve) break;
                tc_fence_after();
                const uint32_t at = smem_u32(smem) + (uint32_t)(s * kStage);
                const uint32_t lead = tmem + (uint32_t)(s * L * BN), rest = tmem + (uint32_t)(S * L * BN);
                const uint64_t w3 = make_smem_desc(at + 2 * kBlock), x3 = make_smem_desc(at + 3 * kBlock + 2 * kX);
#pragma unroll
                for (int k = 0; k < 4; ++k) {   // K steps of 16 are 2 descriptor units apart; plane 2 lies 4 units behind plane 1
                    const uint64_t w = make_smem_desc(at + (k >> 1) * kBlock) + (uint64_t)(2 * (k & 1)), x = make_smem_desc(at + 3 * kBlock + (k >> 1) * kX) + (uint64_t)(2 * (k & 1));
                    umma_bf16(lead + k * L / 4 * BN, w, x, kIdesc, k % (4 / L) > 0 ? 1u : 0u);
                    umma_bf16(rest, w3 + 2 * k, x, kIdesc, it > 0 || k > 0 ? 1u : 0u);
                    umma_bf16(rest, w, x3 + 2 * k, kIdesc, 1u);
                    umma_bf16(rest, w + 4, x + 4, kIdesc, 1u);
                    umma_bf16(rest, w + 4, x, kIdesc, 1u);
                    umma_bf16(rest, w, x + 4, kIdesc, 1u);
                }
                umma_commit(&done[s]);
                if (++s == S) { s = 0; phase ^= 1u; }
            }
        }
        __syncwarp();
    } else if (sums) {
#pragma unroll
        for (int i = 0; i < kSumCols; ++i) acc[i] = 0.f;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c_lo;
        auto add = [&](uint32_t at) {
#pragma unroll
            for (int h = 0; h < kSumCols / 32 * 32; h += 32) {
                float v[32];
                tmem_ld_32(lane_base + at + (uint32_t)h, v);
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[h + i] += v[i];
            }
            if constexpr (kSumCols % 32) {
                constexpr int h = kSumCols / 32 * 32;
                float v[16];
                tmem_ld_16(lane_base + at + (uint32_t)h, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[h + i] += v[i];
            }
        };
#pragma unroll 1
        for (int it = 0; it < n_k; ++it) {
            const int b = it % S;
            if (!wait(&done[b], (uint32_t)(it / S) & 1u)) break;
            tc_fence_after();
            if constexpr (L == 4) {   // in pairs: fewer roundings of the long sum
                float v[4][32];
#pragma unroll
                for (int j = 0; j < 4; ++j) tmem_ld_32(lane_base + (uint32_t)((b * 4 + j) * BN), v[j]);
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[i] += (v[0][i] + v[1][i]) + (v[2][i] + v[3][i]);
            } else {
                add((uint32_t)(b * BN));
            }
            tc_fence_before();
            mbar_arrive(&lead_empty[b]);
        }
        tc_fence_after();
        add((uint32_t)(S * L * BN));   // complete with the last stage's leading sums
        pdl_wait();     // what the epilogue reads (residual, x of a repeated sum)
    }
    if (failed) atomicExch(p.status, 3);
    tc_fence_before();
    __syncthreads();
    if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kCols) : "memory");

    const int parts = kp.n_split, rank = parts > 1 ? (int)cluster_ctarank() : 0, rows_max = (BN + parts - 1) / parts;
    // Row r of the tile belongs to rank r % parts of the cluster; its slots [rank][row / parts][128] lie over the stages, so nobody pushes before
    // everybody's MMAs have read theirs.
    if (parts > 1) cluster_sync_all();
    const uint32_t inv = (65536u + (uint32_t)parts - 1u) / (uint32_t)parts;   // r / parts == (r * inv) >> 16 for r < 160
    auto push = [&](int r, int col, float v) {
        const int local = (int)(((uint32_t)r * inv) >> 16);
        const uint32_t at = smem_u32(smem) + (uint32_t)(((rank * rows_max + local) * 128 + col) * 4);
        if (parts > 1) st_cluster_f32(map_to_cta(at, (uint32_t)(r - local * parts)), v);
        else asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(at), "f"(v) : "memory");
    };
    if (sums) {
        const int col = quarter * 32 + lane, n = n0 + col, k_lo = kt0 * 64, k_hi = (kt0 + n_k) * 64;
        uint64_t special = 0, behind = 0;   // rows whose sum is not finite (behind: from the 64th on): once more, in f32
        if (parts == 1) {
            float* at = reinterpret_cast<float*>(smem) + c_lo * 128 + col;
#pragma unroll
            for (int i = 0; i < kSumCols; ++i) at[i * 128] = acc[i];
        } else {
#pragma unroll
            for (int i = 0; i < kSumCols; ++i) push(c_lo + i, col, acc[i]);
        }
#pragma unroll
        for (int i = 0; i < kSumCols; ++i) (i < 64 ? special : behind) |= fabsf(acc[i]) < INFINITY ? 0ull : 1ull << (i & 63);
#pragma unroll 1
        while (special | behind) {
            const int r = c_lo + (special ? __ffsll((long long)special) - 1 : __ffsll((long long)behind) + 63), m = m0 + r;
            if (special) special &= special - 1;
            else behind &= behind - 1;
            if (m >= p.M || n >= p.N) continue;
            float sum = 0.f;
#pragma unroll 1
            for (int k = k_lo; k < k_hi; ++k) sum = fmaf(p.x[(size_t)m * p.K + k], p.w[(size_t)k * p.N + n], sum);
            push(r, col, sum);
        }
    }
    if (parts > 1) cluster_sync_all();
    else __syncthreads();
    const float4* got = reinterpret_cast<const float4*>(smem);   // N is a multiple of four
#pragma unroll 1
    for (int j = tid; j < rows_max * 32; j += kThreads) {
        const int r = rank + parts * (j >> 5), m = m0 + r, n = n0 + (j & 31) * 4;
        if (r >= BN || m >= p.M || n >= p.N) continue;
        float4 v = got[j];
#pragma unroll 1
        for (int q = 1; q < parts; ++q) {
            const float4 u = got[q * rows_max * 32 + j];
            v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
        }
        if (p.bias) {
            const float4 u = __ldg(reinterpret_cast<const float4*>(p.bias + n));
            v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
        }
        if (p.act == 1) {
            auto gelu = [](float z) { return (0.5f * z) * (1.f + erff(z / 1.4142135f)); };
            v.x = gelu(v.x); v.y = gelu(v.y); v.z = gelu(v.z); v.w = gelu(v.w);
        }
        const size_t at = (size_t)m * p.N + n;
        if (p.residual) {
            const float4 u = *reinterpret_cast<const float4*>(p.residual + at);
            v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
        }
        *reinterpret_cast<float4*>(p.y + at) = v;
        if (p.y_planes) store_planes(static_cast<__nv_bfloat16*>(p.y_planes), p.M, p.N, m, n, v);
    }
}

// ---- norms that leave their rows as planes, too -----------------------------------------------------------------------------------------
struct NormParams { const float *x, *gamma, *beta; float* y; void* planes; int rows, K; float eps; };
// A warp per row of up to 2048 elements, the row in registers: LayerNorm (beta may be null) or RMSNorm.
template <bool LN>
__global__ void __launch_bounds__(256) norm_planes_kernel(const NormParams p) {
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5), n = p.K >> 7;   // float4 of a lane
    pdl_wait();
    if (row >= p.rows) return;
    const float4* x = reinterpret_cast<const float4*>(p.x + (size_t)row * p.K);
    float4 v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (j < n) v[j] = x[lane + 32 * j];
    float mean = 0.f;
    if constexpr (LN) {
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (j < n) s += (v[j].x + v[j].y) + (v[j].z + v[j].w);
        mean = warp_sum(s) / (float)p.K;
    }
    float q = 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (j < n) {
            const float a = v[j].x - mean, b = v[j].y - mean, c = v[j].z - mean, d = v[j].w - mean;
            q += (a * a + b * b) + (c * c + d * d);
        }
    const float inv = 1.f / sqrtf(warp_sum(q) / (float)p.K + p.eps);
    __nv_bfloat16* planes = static_cast<__nv_bfloat16*>(p.planes);
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (j < n) {
            const int k = (lane + 32 * j) * 4;
            const float4 g = __ldg(reinterpret_cast<const float4*>(p.gamma + k));
            float4 o = make_float4((v[j].x - mean) * inv * g.x, (v[j].y - mean) * inv * g.y, (v[j].z - mean) * inv * g.z, (v[j].w - mean) * inv * g.w);
            if (LN && p.beta) {
                const float4 b = __ldg(reinterpret_cast<const float4*>(p.beta + k));
                o.x += b.x; o.y += b.y; o.z += b.z; o.w += b.w;
            }
            *reinterpret_cast<float4*>(p.y + (size_t)row * p.K + k) = o;
            store_planes(planes, p.rows, p.K, row, k, o);
        }
}

int make_map(CUtensorMap* map, const void* base, uint64_t inner, uint64_t rows, uint32_t box_rows) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return fail(GPTRS_EXECUTION, "cuTensorMapEncodeTiled is not available");
    const cuuint64_t dims[2] = {inner, rows}, strides[1] = {inner * 2};
    const cuuint32_t box[2] = {64, box_rows}, elem[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(GPTRS_EXECUTION, "cuTensorMapEncodeTiled failed for bf16 planes (" + std::to_string((int)r) + ")");
    return GPTRS_OK;
}

template <int BN> constexpr size_t kSmem = (size_t)kStages<BN> * kStageBytes<BN> + 1024;
template <int BN>
int allow_smem() {
    static PerDeviceOnce once;
    if (once.first_time())
        for (auto k : {planes_matmul_kernel<BN>, planes_matmul_kernel<BN, true>})
            GPTRS_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem<BN>));
    return GPTRS_OK;
}

// How many CTAs of a cluster size run at one time, asked once per device.
template <int BN>
int64_t slots_of(int cluster) {
    static std::atomic<int> known[kMaxDevices][9];
    std::atomic<int>& slot = known[current_device() & (kMaxDevices - 1)][cluster];
    int n = slot.load(std::memory_order_relaxed);
    if (n == 0) {
        n = sm_count();
        if (cluster > 1) {
            allow_smem<BN>();
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(1, (unsigned)cluster, 1);
            cfg.blockDim = dim3(kThreads);
            cfg.dynamicSmemBytes = kSmem<BN>;
            cudaLaunchAttribute attr;
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = 1; attr.val.clusterDim.y = (unsigned)cluster; attr.val.clusterDim.z = 1;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, planes_matmul_kernel<BN>, &cfg) != cudaSuccess) { cudaGetLastError(); clusters = 0; }
            n = clusters > 0 ? clusters * cluster : 1;
        }
        slot.store(n, std::memory_order_relaxed);
    }
    return n;
}

template <int BN>
int launch(const PlanesMatmul& q, int split, cudaStream_t st) {
    if (int rc = allow_smem<BN>()) return rc;
    KernelParams p;
    p.q = q;
    const __nv_bfloat16 *w = static_cast<const __nv_bfloat16*>(q.w_planes), *x = static_cast<const __nv_bfloat16*>(q.x_planes);
    int rc;
    if ((rc = make_map(&p.w12, w, 2 * (uint64_t)q.K, (uint64_t)q.N, 128)) || (rc = make_map(&p.w3, w + (size_t)q.N * 2 * q.K, (uint64_t)q.K, (uint64_t)q.N, 128)) ||
        (rc = make_map(&p.x12, x, 2 * (uint64_t)q.K, (uint64_t)q.M, BN)) || (rc = make_map(&p.x3, x + (size_t)q.M * 2 * q.K, (uint64_t)q.K, (uint64_t)q.M, BN))) return rc;
    p.n_split = split;
    matmul_wait_limits(&p.spin_limit, &p.starve);
    return launch_kernel(p.starve || p.spin_limit != kSpinLimit ? planes_matmul_kernel<BN, true> : planes_matmul_kernel<BN>, dim3((unsigned)ceil_div(q.N, 128), (unsigned)p.n_split, (unsigned)ceil_div(q.M, BN)), dim3(kThreads), kSmem<BN>, st, p.n_split, p);
}

// The rows of a tile and the parts of K that make the last CTA end soonest, in hundredths of a microsecond as measured on GPT-2's projections
// at 32 to 937 rows: a stage of 64 k takes 0.68 / 0.80 / 0.95 / 1.08 us with 32 / 64 / 128 / 160 rows, a CTA's beginning and end 6.4 / 7 / 9 / 10,
// the exchange of the parts 1.5.
struct Tiling { int rows = 0, split = 1; int64_t time = 1ll << 60; };
template <int BN>
void consider(const PlanesMatmul& q, Tiling& best) {
    constexpr int64_t stage = BN == 32 ? 68 : BN == 64 ? 80 : BN == 128 ? 95 : 108, fixed = BN == 32 ? 640 : BN == 64 ? 700 : BN == 128 ? 900 : 1000;
    const int64_t ctas = (int64_t)ceil_div(q.N, 128) * ceil_div(q.M, BN), k_tiles = q.K / 64;
    for (int s = 1; s <= 8 && s <= k_tiles; ++s) {
        const int64_t slots = slots_of<BN>(s), t = ((ctas * s + slots - 1) / slots) * ((k_tiles + s - 1) / s * stage + fixed + (s > 1 ? 150 : 0));
        if (t < best.time) best = {BN, s, t};
    }
}

}  // namespace

int split_weight_planes(const float* w, void* planes, int64_t k, int64_t n, cudaStream_t st) {
    GPTRS_REQUIRE(k > 0 && k % 64 == 0 && n > 0, "planes: K a multiple of 64");
    __nv_bfloat16* at = static_cast<__nv_bfloat16*>(planes);
    const SplitParams p = {w, at, at + (size_t)n * 2 * k, (int)n, (int)k, (int)n};
    split_weights_kernel<<<dim3((unsigned)ceil_div(n, 32), (unsigned)(k / 32)), 256, 0, st>>>(p);
    GPTRS_CUDA_OK(cudaGetLastError());
    return GPTRS_OK;
}
int split_row_planes(const float* x, void* planes, int64_t m, int64_t k, cudaStream_t st) {
    GPTRS_REQUIRE(k > 0 && k % 64 == 0 && m > 0, "planes: K a multiple of 64");
    __nv_bfloat16* at = static_cast<__nv_bfloat16*>(planes);
    const SplitParams p = {x, at, at + (size_t)m * 2 * k, (int)m, (int)k, 0};
    return launch_kernel(split_rows_kernel, dim3((unsigned)ceil_div(m * (k / 4), 256)), dim3(256), 0, st, 1, p);
}
bool norm_planes_takes(int64_t k) { return k % 128 == 0 && k <= 2048; }
int norm_planes(const float* x, const float* gamma, const float* beta, float eps, bool layer_norm, float* y, void* planes, int64_t rows, int64_t k, cudaStream_t st) {
    GPTRS_REQUIRE(norm_planes_takes(k) && rows > 0, "norm with planes: rows of up to 2048, a multiple of 128");
    const NormParams p = {x, gamma, beta, y, planes, (int)rows, (int)k, eps};
    return launch_kernel(layer_norm ? norm_planes_kernel<true> : norm_planes_kernel<false>, dim3((unsigned)ceil_div(rows, 8)), dim3(256), 0, st, 1, p);
}
int planes_matmul(const PlanesMatmul& q, cudaStream_t st) {
    GPTRS_REQUIRE(q.M > 0 && q.N > 0 && q.K > 0 && q.K % 64 == 0 && q.N % 4 == 0 && (!q.y_planes || q.N % 64 == 0), "planes: K (and N of a result that is split) a multiple of 64, N of 4");
    PlanesMatmul p = q;
    if (!p.status) p.status = matmul_status_word();
    if (!p.status) return fail(GPTRS_EXECUTION, "no status word");
    Tiling t;
    consider<32>(p, t);   // alone where plain f32 is the other choice: see above
    if (split_f32_line(p.M, p.N, p.K)) { consider<64>(p, t); consider<128>(p, t); consider<160>(p, t); }
    switch (t.rows) {
        case 32: return launch<32>(p, t.split, st);
        case 64: return launch<64>(p, t.split, st);
        case 128: return launch<128>(p, t.split, st);
        default: return launch<160>(p, t.split, st);
    }
}

}  // namespace gptrs

extern "C" int gptrs_cuda_debug_planes_matmul(const float* d_x, const float* d_w, const float* d_bias, const float* d_residual, float* d_y, int64_t m, int64_t n,
                                              int64_t k, int gelu, void* d_planes, size_t planes_bytes, void* stream) {
    using namespace gptrs;
    GPTRS_REQUIRE(d_x && d_w && d_y && d_planes, "null pointer");
    GPTRS_REQUIRE(m > 0 && n > 0 && k > 0 && m <= INT32_MAX && n <= INT32_MAX && k <= INT32_MAX && k % 64 == 0, "planes: K a multiple of 64");
    const size_t w_bytes = (plane_bytes(n, k) + 255) & ~(size_t)255;
    GPTRS_REQUIRE(planes_bytes >= w_bytes + plane_bytes(m, k) && (reinterpret_cast<uintptr_t>(d_planes) & 255) == 0, "planes: buffer too small or not aligned to 256 bytes");
    cudaStream_t st = as_stream(stream);
    void* const x_planes = static_cast<unsigned char*>(d_planes) + w_bytes;
    struct PdlGuard { int saved = g_use_pdl; PdlGuard() { g_use_pdl = 0; } ~PdlGuard() { g_use_pdl = saved; } } guard;   // these weights are not constant
    int rc;
    if ((rc = split_weight_planes(d_w, d_planes, k, n, st)) || (rc = split_row_planes(d_x, x_planes, m, k, st))) return rc;
    return planes_matmul({d_planes, x_planes, d_x, d_w, d_bias, d_residual, d_y, nullptr, (int)m, (int)n, (int)k, gelu ? 1 : 0, nullptr}, st);
}
