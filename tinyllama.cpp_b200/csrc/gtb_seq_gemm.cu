// gtb_seq_gemm.cu -- bf16 matrix product of the layer-list sequence models on the 5th-generation tensor cores.
//
//     C[M][N] = (acc ? C : 0) + bias + A[M][K] . W[N][K]^T        A, W bf16 (K contiguous), C fp32
//
// Same structure as the batched-prefill product of the TinyLlama path (gtb_prefill.cu), with bf16 operands and a plain fp32
// epilogue: persistent CTAs (one per SM) walk the 128 x BN output tiles; warp 0 is the TMA producer (128-byte swizzled 128 x 64 and
// BN x 64 boxes through a ring of mbarrier stages), one thread of warp 1 issues tcgen05.mma kind::f16 (M128 x N(BN) x K16, fp32
// accumulators in a double-buffered TMEM allocation) and releases stages / publishes accumulators with tcgen05.commit, warps 2-9
// read their 32 TMEM lanes back with tcgen05.ld and write C -- the epilogue of tile i overlaps the main loop of tile i + 1.
// Rows and columns beyond M and N come in as zeros (TMA out-of-bounds fill) and are not stored; K is a multiple of 64 because every
// operand of these models is padded to that.
//
// Every mbarrier wait is bounded: a wait that does not complete raises the CTA's abort flag, every role leaves its loop, the
// TMEM allocation is released and the kernel returns with a status word set that the host reads after the launch.
//
// The fused variant (EPI_GEGLU) takes W = gate rows and up rows interleaved in groups of 32 and writes gelu_tanh(gate) * up as a
// bf16 operand block: the feed-forward activation never exists in fp32 in HBM.
//
// Grouped products (routed experts): the rows of A are sorted into groups that start on multiples of 128 rows, a device table gives
// every M tile its group (or -1: nothing to do), and group g multiplies with rows [g N, (g + 1) N) of W.  EPI_RELU2 writes
// row_w[row] * relu(acc)^2 as a bf16 operand block (the expert's activation, already weighted with the router's score); EPI_GELU writes
// gelu(acc) (erf form), the activation of an ungated feed-forward, the same way.
#include "gtb_seq_gemm.h"

#include <cuda_bf16.h>

#include "gtb_internal.h"
#include "gtb_seq_gemm_plan.h"
#include "gtb_tc.cuh"

namespace gtb {
namespace seq {

constexpr int SQ_BM = 128, SQ_BK = 64, SQ_THREADS = 320, SQ_EPI_THREADS = 256;
enum { SQ_EPI_F32 = 0, SQ_EPI_GEGLU = 1, SQ_EPI_RELU2 = 2, SQ_EPI_GELU = 3 };

template <int BN> struct SqCfg {
    static constexpr int STAGES = (BN == 256) ? 4 : 6;
    static constexpr uint32_t A_BYTES = SQ_BM * SQ_BK * 2;
    static constexpr uint32_t B_BYTES = BN * SQ_BK * 2;
    static constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr uint32_t SMEM = STAGES * STAGE_BYTES + 1024 + 256;
    // kind::f16 instruction descriptor: D fp32 (bit 4), A and B bf16 (format 1 at bits 7-9 and 10-12), both K-major,
    // N >> 3 at bits 17-22, M >> 4 at bits 24-28
    static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(SQ_BM >> 4) << 24);
};

struct SqEpi {
    float* C;
    int ldc;
    const float* bias;
    int accumulate;
    __nv_bfloat16* act;      // EPI_GEGLU: output operand [M][ld_act], written at column act_off + (pair index)
    int ld_act, act_off;
    int* status;
    const int* tile_group;   // grouped product: group of every M tile (-1: skip), or null
    int group_rows;          // rows of W per group
    const float* row_w;      // EPI_RELU2: weight of every row of A; EPI_GEGLU: optional weight of every row
    int act_kind;            // EPI_GEGLU: 0 = gelu_tanh(gate) * up, 1 = silu(gate) * up
    int w_blocks;            // k-blocks of W: A's k-block kb meets W's kb mod w_blocks (split operands hold several pieces of K one after the other)
};

// bounded wait: false when the barrier did not complete (or another role gave up)
__device__ __forceinline__ bool sq_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    for (int it = 0; it < (1 << 24); it++) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 1023) == 1023 && *abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}

// tanh on the special-function unit: relative error ~2^-11, below the bf16 rounding of the value that is stored
__device__ __forceinline__ float sq_gelu(float z) {
    const float c = 0.7978845608028654f;
    float th;
    asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(c * (z + 0.044715f * z * z * z)));
    return 0.5f * z * (1.0f + th);
}

// silu(z) = z / (1 + 2^(-z log2 e)) on the special-function unit; the value is rounded to bf16 right after
__device__ __forceinline__ float sq_silu(float z) { return __fdividef(z, 1.0f + __expf(-z)); }
// gelu(z) = z (1 + erf(z / sqrt 2)) / 2 with erfc from Abramowitz & Stegun, Handbook of Mathematical Functions, 7.1.26 (absolute error
// 1.5e-7): erfc(x) = (a1 t + .. + a5 t^5) exp(-x^2), t = 1 / (1 + p x), x >= 0.  No branch, and a negative z multiplies erfc itself, so its
// small values keep their relative accuracy; the value is rounded to bf16 right after
__device__ __forceinline__ float sq_gelu_erf(float z) {
    const float x = fabsf(z) * 0.70710678118654752f;
    const float t = __fdividef(1.0f, fmaf(0.3275911f, x, 1.0f));
    float q = fmaf(t, 1.061405429f, -1.453152027f);
    q = fmaf(t, q, 1.421413741f);
    q = fmaf(t, q, -0.284496736f);
    q = fmaf(t, q, 0.254829592f);
    q *= t * __expf(-x * x);
    return 0.5f * z * (z < 0.0f ? q : 2.0f - q);
}
__device__ __forceinline__ float sq_gate(float z, int kind) { return kind ? sq_silu(z) : sq_gelu(z); }

// SWAP: 128 rows of W are the M side of the MMA and BN rows of A its N side (tmA is then the map of W, tmB that of A): TMEM lanes are
// output columns, so the fp32 epilogue writes 128 contiguous bytes per warp and row of C (one row per lane otherwise: 32 half-used sectors per
// store).  2048 x 6400 x 2048: 54 us against 65; accumulating into C 58 against 762, so residual updates need no block of their own.
template <int BN, int EPI, bool SWAP>
__global__ void __launch_bounds__(SQ_THREADS, 1)
k_seq_gemm(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int M, int N, int K, const SqEpi ep) {
    using Cfg = SqCfg<BN>;
    constexpr int ST = Cfg::STAGES;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + ST * Cfg::STAGE_BYTES);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * ST + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t smem_base = smem_u32(smem), bar_base = smem_u32(bars);
    auto bar_full = [&](int s) { return bar_base + 8u * s; };
    auto bar_empty = [&](int s) { return bar_base + 8u * (ST + s); };
    auto bar_tfull = [&](int a) { return bar_base + 8u * (2 * ST + a); };
    auto bar_tempty = [&](int a) { return bar_base + 8u * (2 * ST + 2 + a); };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int TM = SWAP ? BN : SQ_BM, TN = SWAP ? SQ_BM : BN;      // rows and columns of C per tile
    const int n_mt = (M + TM - 1) / TM, n_nt = (N + TN - 1) / TN;
    const int n_tiles = n_mt * n_nt, nkb = K / SQ_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; s++) { mbar_init(bar_full(s), 1); mbar_init(bar_empty(s), 1); }
        for (int a = 0; a < 2; a++) { mbar_init(bar_tfull(a), 1); mbar_init(bar_tempty(a), SQ_EPI_THREADS); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 2 * BN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger_and_wait();        // (behind the TMEM allocation)

    if (warp == 0) {
        if (lane == 0) {        // ---------------- TMA producer
            tma_prefetch_desc(&tmA);
            tma_prefetch_desc(&tmB);
            uint32_t s = 0, ph = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < n_tiles; tile += gridDim.x) {
                const int mt = tile % n_mt, nt = tile / n_mt;         // consecutive CTAs share one slice of W
                const int grp = ep.tile_group ? ep.tile_group[mt] : 0;
                if (grp < 0) continue;
                const int arow = mt * TM, wrow = grp * ep.group_rows + nt * TN;
                for (int kb = 0; kb < nkb; kb++) {
                    if (!(ok = sq_wait(bar_empty(s), ph ^ 1, abort_flag))) break;
                    mbar_expect_tx(bar_full(s), Cfg::STAGE_BYTES);
                    const uint32_t sa = smem_base + s * Cfg::STAGE_BYTES;
                    tma_load_2d(sa, &tmA, bar_full(s), (SWAP ? kb % ep.w_blocks : kb) * SQ_BK, SWAP ? wrow : arow);
                    tma_load_2d(sa + Cfg::A_BYTES, &tmB, bar_full(s), kb * SQ_BK, SWAP ? arow : wrow);
                    if (++s == ST) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {        // ---------------- MMA issuer
            uint32_t s = 0, ph = 0;
            int it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < n_tiles; tile += gridDim.x) {
                if (ep.tile_group && ep.tile_group[tile % n_mt] < 0) continue;      // skipped tiles take no accumulator stage
                const int cur = it++, as = cur & 1;
                if (!(ok = sq_wait(bar_tempty(as), ((cur >> 1) & 1) ^ 1, abort_flag))) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(as * BN);
                for (int kb = 0; kb < nkb; kb++) {
                    if (!(ok = sq_wait(bar_full(s), ph, abort_flag))) break;
                    tc_fence_after();
                    const uint32_t sa = smem_base + s * Cfg::STAGE_BYTES, sb = sa + Cfg::A_BYTES;
#pragma unroll
                    for (int k = 0; k < SQ_BK / 16; k++)
                        umma_f16(d_tmem, umma_desc_sw128(sa + k * 32), umma_desc_sw128(sb + k * 32), Cfg::IDESC, (kb | k) != 0);
                    umma_commit(bar_empty(s));
                    if (kb == nkb - 1) umma_commit(bar_tfull(as));
                    if (++s == ST) { s = 0; ph ^= 1; }
                }
            }
        }
        __syncwarp();
    } else {                    // ---------------- epilogue warps
        const int lg = warp & 3;                                    // TMEM lanes 32 * (warp % 4) .. + 31
        const int chalf = (warp - 2) >> 2;                          // which half of the tile's columns
        int it = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < n_tiles; tile += gridDim.x) {
            const int mt = tile % n_mt, nt = tile / n_mt;
            if (ep.tile_group && ep.tile_group[mt] < 0) continue;
            const int cur = it++, as = cur & 1;
            if (!(ok = sq_wait(bar_tfull(as), (cur >> 1) & 1, abort_flag))) break;
            tc_fence_after();
            const int row = mt * SQ_BM + lg * 32 + lane;
            const uint32_t tacc = tmem_base + ((uint32_t)(lg * 32) << 16) + (uint32_t)(as * BN);
            if (EPI == SQ_EPI_F32 && SWAP) {
                const int col = nt * TN + lg * 32 + lane, r0 = mt * TM;
                const float bias = (ep.bias && col < N) ? ep.bias[col] : 0.0f;
#pragma unroll 1
                for (int c = chalf * (BN / 64); c < (chalf + 1) * (BN / 64); c++) {
                    if (r0 + c * 32 >= M) break;
                    float v[32];
                    tmem_ld32(tacc + (uint32_t)(c * 32), v);
                    float* dst = ep.C + (size_t)(r0 + c * 32) * ep.ldc + col;
                    const int nr = col < N ? min(32, M - r0 - c * 32) : 0;
                    if (ep.accumulate) {
                        float p[32];
#pragma unroll
                        for (int j = 0; j < 32; j++) p[j] = j < nr ? dst[(size_t)j * ep.ldc] : 0.0f;
#pragma unroll
                        for (int j = 0; j < 32; j++) v[j] += p[j];
                    }
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (j < nr) dst[(size_t)j * ep.ldc] = v[j] + bias;
                }
            } else if (EPI == SQ_EPI_F32) {                         // grouped products: no bias, nothing to add to
#pragma unroll 1
                for (int c = chalf * (BN / 64); c < (chalf + 1) * (BN / 64); c++) {
                    const int col = nt * BN + c * 32;
                    float v[32];
                    tmem_ld32(tacc + (uint32_t)(c * 32), v);
                    if (row < M && col < N) {
                        float* dst = ep.C + (size_t)row * ep.ldc + col;
                        const int nc = min(32, N - col);
                        if (nc == 32 && ((((uintptr_t)dst) & 15) == 0)) {
#pragma unroll
                            for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; j++)
                                if (j < nc) dst[j] = v[j];
                        }
                    }
                }
            } else if (EPI == SQ_EPI_RELU2 || EPI == SQ_EPI_GELU) {
                const float wt = (EPI == SQ_EPI_RELU2 && row < M) ? ep.row_w[row] : 0.0f;
                auto act = [wt](float a) {
                    if (EPI == SQ_EPI_GELU) return sq_gelu_erf(a);
                    a = fmaxf(a, 0.0f);
                    return wt * a * a;
                };
#pragma unroll 1
                for (int c = chalf * (BN / 64); c < (chalf + 1) * (BN / 64); c++) {
                    const int col = nt * BN + c * 32;
                    float v[32];
                    tmem_ld32(tacc + (uint32_t)(c * 32), v);
                    if (row < M && col < N) {
                        __nv_bfloat16* dst = ep.act + (size_t)row * ep.ld_act + ep.act_off + col;
                        const int nc = min(32, N - col);
                        if (nc == 32 && ((((uintptr_t)dst) & 15) == 0)) {
#pragma unroll
                            for (int j = 0; j < 32; j += 8) {
                                uint32_t w[4];
#pragma unroll
                                for (int q = 0; q < 4; q++) {
                                    const __nv_bfloat162 pr = __floats2bfloat162_rn(act(v[j + 2 * q]), act(v[j + 2 * q + 1]));
                                    w[q] = *reinterpret_cast<const uint32_t*>(&pr);
                                }
                                *reinterpret_cast<uint4*>(dst + j) = make_uint4(w[0], w[1], w[2], w[3]);
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; j++)
                                if (j < nc) dst[j] = __float2bfloat16_rn(act(v[j]));
                        }
                    }
                }
            } else {
                // 64 accumulator columns = 32 gate columns followed by their 32 up columns
                const float wt = (ep.row_w && row < M) ? ep.row_w[row] : 1.0f;
                const int ak = ep.act_kind;
#pragma unroll 1
                for (int c2 = chalf * (BN / 128); c2 < (chalf + 1) * (BN / 128); c2++) {
                    const int col = nt * BN + c2 * 64;
                    float g[32], u[32];
                    tmem_ld32(tacc + (uint32_t)(c2 * 64), g);
                    tmem_ld32(tacc + (uint32_t)(c2 * 64 + 32), u);
                    if (row < M && col < N) {
                        const int c0 = col >> 1;                   // first of the 32 activation channels
                        __nv_bfloat16* dst = ep.act + (size_t)row * ep.ld_act + ep.act_off + c0;
                        const int nc = min(32, (N >> 1) - c0);
                        if (nc == 32 && ((((uintptr_t)dst) & 15) == 0)) {
#pragma unroll
                            for (int j = 0; j < 32; j += 8) {
                                uint32_t w[4];
#pragma unroll
                                for (int q = 0; q < 4; q++) {
                                    const __nv_bfloat162 v = __floats2bfloat162_rn(wt * sq_gate(g[j + 2 * q], ak) * u[j + 2 * q], wt * sq_gate(g[j + 2 * q + 1], ak) * u[j + 2 * q + 1]);
                                    w[q] = *reinterpret_cast<const uint32_t*>(&v);
                                }
                                *reinterpret_cast<uint4*>(dst + j) = make_uint4(w[0], w[1], w[2], w[3]);
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; j++)
                                if (j < nc) dst[j] = __float2bfloat16_rn(wt * sq_gate(g[j], ak) * u[j]);
                        }
                    }
                }
            }
            tc_fence_before();
            mbar_arrive(bar_tempty(as));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag && ep.status) atomicExch(ep.status, 1);
    if (warp == 1) tmem_dealloc(tmem_base, 2 * BN);
}

// ------------------------------------------------------------------------------------------------ few rows: swapped operands, split K
// The same product for passes whose output has too few 128 x BN tiles to occupy the chip (decode batches, short prompts, the head on the
// wanted rows).  Roles are swapped: 128 rows of W are the M side of the MMA and MT rows of A its N side, so a tile costs no padding beyond a
// multiple of 16 rows; K is split over the CTAs of a cluster, whose partial sums meet in distributed shared memory in rank order (the
// result does not depend on timing).  TMEM lanes are output columns, so a warp's partial rows and the final stores are contiguous.
// Bound by the stream of W: 24 rows x 2048 x 2048 in 4.5 us (8.4 MB: 1.9 TB/s) where the FFMA tile kernel took 120 us; 24 rows x 32000 x 2048
// in 28 us (131 MB: 4.7 TB/s).
template <int MT> struct SkCfg {
    static constexpr uint32_t W_BYTES = 128 * SQ_BK * 2;
    static constexpr uint32_t A_BYTES = MT * SQ_BK * 2;
    static constexpr uint32_t STAGE_BYTES = W_BYTES + A_BYTES;
    static constexpr int STAGES = MT <= 32 ? 5 : 4;      // two CTAs per SM
    static constexpr uint32_t SMEM = STAGES * STAGE_BYTES + 1024 + 256;
    static constexpr uint32_t COLS = MT < 32 ? 32 : MT;
    static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(MT >> 3) << 17) | (8u << 24);
    static_assert(MT * 128 * 4 <= STAGES * STAGE_BYTES, "partial sums reuse the stages");
};
constexpr int SK_THREADS = 192;

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr, uint32_t rank) {
    uint32_t a;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int MT, int EPI>
__global__ void __launch_bounds__(SK_THREADS)
k_seq_skinny(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmA, int M, int N, int K, int cs, const SqEpi ep) {
    using Cfg = SkCfg<MT>;
    constexpr int ST = Cfg::STAGES;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + ST * Cfg::STAGE_BYTES);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * ST + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t smem_base = smem_u32(smem), bar_base = smem_u32(bars);
    auto bar_full = [&](int s) { return bar_base + 8u * s; };
    auto bar_empty = [&](int s) { return bar_base + 8u * (ST + s); };
    const uint32_t bar_done = bar_base + 8u * (2 * ST);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x % cs, n0 = (int)blockIdx.x / cs * 128, m0 = (int)blockIdx.y * MT;
    const int nkb = K / SQ_BK, kb0 = (int)((long long)nkb * rank / cs), kb1 = (int)((long long)nkb * (rank + 1) / cs);

    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; s++) { mbar_init(bar_full(s), 1); mbar_init(bar_empty(s), 1); }
        mbar_init(bar_done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), Cfg::COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();                 // (behind the TMEM allocation)
    if (threadIdx.x != 0) pdl_wait();      // the producer thread waits behind its first loads of W

    if (warp == 0) {
        if (lane == 0) {        // ---------------- TMA producer
            // W does not depend on the kernels before: its first stages are on their way while those finish
            const int pre = min(ST, kb1 - kb0);
            for (int i = 0; i < pre; i++) {
                mbar_expect_tx(bar_full(i), Cfg::STAGE_BYTES);
                tma_load_2d(smem_base + i * Cfg::STAGE_BYTES, &tmW, bar_full(i), (kb0 + i) % ep.w_blocks * SQ_BK, n0);
            }
            pdl_wait();
            for (int i = 0; i < pre; i++) tma_load_2d(smem_base + i * Cfg::STAGE_BYTES + Cfg::W_BYTES, &tmA, bar_full(i), (kb0 + i) * SQ_BK, m0);
            uint32_t s = pre % ST, ph = pre == ST ? 1 : 0;
            for (int kb = kb0 + pre; kb < kb1; kb++) {
                if (!sq_wait(bar_empty(s), ph ^ 1, abort_flag)) break;
                mbar_expect_tx(bar_full(s), Cfg::STAGE_BYTES);
                const uint32_t sw = smem_base + s * Cfg::STAGE_BYTES;
                tma_load_2d(sw, &tmW, bar_full(s), kb % ep.w_blocks * SQ_BK, n0);
                tma_load_2d(sw + Cfg::W_BYTES, &tmA, bar_full(s), kb * SQ_BK, m0);
                if (++s == ST) { s = 0; ph ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {        // ---------------- MMA issuer
            uint32_t s = 0, ph = 0;
            bool ok = true;
            for (int kb = kb0; kb < kb1; kb++) {
                if (!(ok = sq_wait(bar_full(s), ph, abort_flag))) break;
                tc_fence_after();
                const uint32_t sw = smem_base + s * Cfg::STAGE_BYTES, sa = sw + Cfg::W_BYTES;
#pragma unroll
                for (int k = 0; k < SQ_BK / 16; k++)
                    umma_f16(tmem_base, umma_desc_sw128(sw + k * 32), umma_desc_sw128(sa + k * 32), Cfg::IDESC, kb > kb0 || k > 0);
                umma_commit(bar_empty(s));
                if (++s == ST) { s = 0; ph ^= 1; }
            }
            if (ok) umma_commit(bar_done);
        }
        __syncwarp();
    } else {                    // ---------------- accumulator -> partial[row of A][128 output columns]
        const bool ok = sq_wait(bar_done, 0, abort_flag);
        tc_fence_after();
        if (ok) {
            const int lg = warp & 3;
            float* part = reinterpret_cast<float*>(smem) + lg * 32 + lane;
#pragma unroll 1
            for (int c = 0; c < MT; c += 16) {
                if (m0 + c >= M) break;
                float v[16];
                tmem_ld16(tmem_base + ((uint32_t)(lg * 32) << 16) + (uint32_t)c, v);
#pragma unroll
                for (int j = 0; j < 16; j++) part[(c + j) * 128] = v[j];
            }
        }
        tc_fence_before();
    }
    if (cs > 1) cluster_sync_all();
    else __syncthreads();
    // every CTA of the cluster finishes its share of the tile's rows
    const int rows = min(MT, M - m0), r0 = rows * rank / cs, r1 = rows * (rank + 1) / cs;
    constexpr int Q = EPI == SQ_EPI_GEGLU ? 16 : 32;       // groups of four outputs per row
    auto sum4 = [&](int m, int n) {
        const uint32_t a = smem_base + (uint32_t)(m * 128 + n) * 4;
        if (cs == 1) return *reinterpret_cast<const float4*>(smem + (size_t)(m * 128 + n) * 4);
        float4 s = ld_cluster_f4(a, 0);
        for (int p = 1; p < cs; p++) { const float4 v = ld_cluster_f4(a, p); s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w; }
        return s;
    };
    for (int i = threadIdx.x; i < (r1 - r0) * Q; i += SK_THREADS) {
        const int m = r0 + i / Q, q = i % Q, row = m0 + m;
        if (EPI == SQ_EPI_F32) {
            const int n = n0 + q * 4;
            if (n >= N) continue;
            float4 o = sum4(m, q * 4);
            float* dst = ep.C + (size_t)row * ep.ldc + n;
            if (n + 4 <= N && (((uintptr_t)dst) & 15) == 0) {
                if (ep.bias) { o.x += ep.bias[n]; o.y += ep.bias[n + 1]; o.z += ep.bias[n + 2]; o.w += ep.bias[n + 3]; }
                if (ep.accumulate) { const float4 p = *reinterpret_cast<const float4*>(dst); o.x += p.x; o.y += p.y; o.z += p.z; o.w += p.w; }
                *reinterpret_cast<float4*>(dst) = o;
            } else {
                const float v[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (n + j < N) dst[j] = v[j] + (ep.bias ? ep.bias[n + j] : 0.0f) + (ep.accumulate ? dst[j] : 0.0f);
            }
        } else {
            // (columns beyond the product's come out as zeros: the operand's padding, as far as the tile reaches, is written too)
            const int c = (EPI == SQ_EPI_GEGLU ? n0 >> 1 : n0) + q * 4, nc = ep.ld_act - ep.act_off;
            if (c >= nc) continue;
            float v[4];
            if (EPI == SQ_EPI_GEGLU) {
                const int g = (q >> 3) * 64 + (q & 7) * 4;                // 32 gate columns, then their 32 up columns
                const float4 a = sum4(m, g), u = sum4(m, g + 32);
                const float wt = ep.row_w ? ep.row_w[row] : 1.0f;
                v[0] = wt * sq_gate(a.x, ep.act_kind) * u.x; v[1] = wt * sq_gate(a.y, ep.act_kind) * u.y;
                v[2] = wt * sq_gate(a.z, ep.act_kind) * u.z; v[3] = wt * sq_gate(a.w, ep.act_kind) * u.w;
            } else {
                const float4 a = sum4(m, q * 4);
                v[0] = sq_gelu_erf(a.x); v[1] = sq_gelu_erf(a.y); v[2] = sq_gelu_erf(a.z); v[3] = sq_gelu_erf(a.w);
            }
            __nv_bfloat16* dst = ep.act + (size_t)row * ep.ld_act + ep.act_off + c;
            if (c + 4 <= nc && (((uintptr_t)dst) & 7) == 0) {
                const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
                *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (c + j < nc) dst[j] = __float2bfloat16_rn(v[j]);
            }
        }
    }
    if (cs > 1) cluster_sync_all();       // a peer may still be reading this CTA's partial sums
    if (threadIdx.x == 0 && *abort_flag && ep.status) atomicExch(ep.status, 1);
    if (warp == 1) tmem_dealloc(tmem_base, Cfg::COLS);
}

// ---------------------------------------------------------------------------------------------------------------- host
int seq_gemm_create(SeqGemmPlan** out) {
    *out = nullptr;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) != cudaSuccess || qres != cudaDriverEntryPointSuccess)
        return fail(GTB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    SeqGemmPlan* g = new SeqGemmPlan();
    g->enc = reinterpret_cast<PFN_tmapEncodeTiled>(p);
    if (cudaMalloc((void**)&g->d_status, sizeof(int)) != cudaSuccess) { delete g; return fail(GTB_ERR_CUDA, "cudaMalloc failed"); }
    cudaMemsetAsync(g->d_status, 0, sizeof(int), ctx().stream);
    *out = g;
    return GTB_OK;
}

void seq_gemm_destroy(SeqGemmPlan* p) {
    if (!p) return;
    if (p->d_status) cudaFree(p->d_status);
    delete p;
}

int seq_gemm_status_async(SeqGemmPlan* p, int* status) {
    GTB_CUDA(cudaMemcpyAsync(status, p->d_status, sizeof(int), cudaMemcpyDeviceToHost, ctx().stream));
    return GTB_OK;
}
int seq_gemm_status(SeqGemmPlan* p, int* status) {
    int rc = seq_gemm_status_async(p, status);
    if (rc) return rc;
    GTB_CUDA(cudaStreamSynchronize(ctx().stream));
    return GTB_OK;
}

static int make_map(SeqGemmPlan* p, CUtensorMap* m, const void* base, int rows, int cols, int ld, int box_rows) {
    const cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t gstr[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)SQ_BK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = p->enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(GTB_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d) for a %d x %d matrix", (int)r, rows, cols);
    return GTB_OK;
}

template <int BN, int EPI, bool SWAP = false>
static int launch(SeqGemmPlan* p, const CUtensorMap& ta, const CUtensorMap& tb, int M, int N, int K, const SqEpi& ep) {
    using Cfg = SqCfg<BN>;
    bool& attr = p->attr[SWAP][BN == 256][EPI];
    if (!attr) {
        GTB_CUDA(cudaFuncSetAttribute(k_seq_gemm<BN, EPI, SWAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM));
        attr = true;
    }
    constexpr int TM = SWAP ? BN : SQ_BM, TN = SWAP ? SQ_BM : BN;
    const int n_tiles = ((M + TM - 1) / TM) * ((N + TN - 1) / TN);
    const int grid = n_tiles < ctx().sm_count ? n_tiles : ctx().sm_count;
    pdl_launch(k_seq_gemm<BN, EPI, SWAP>, grid, SQ_THREADS, Cfg::SMEM, ctx().stream, ta, tb, M, N, K, ep);
    GTB_LAUNCHED();
    return GTB_OK;
}

template <int MT, int EPI>
static int launch_skinny(bool& attr, const CUtensorMap& tw, const CUtensorMap& ta, int M, int N, int K, int cs, const SqEpi& ep) {
    using Cfg = SkCfg<MT>;
    if (!attr) {
        GTB_CUDA(cudaFuncSetAttribute(k_seq_skinny<MT, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM));
        attr = true;
    }
    pdl_launch_cluster(cs, k_seq_skinny<MT, EPI>, dim3((N + 127) / 128 * cs, (M + MT - 1) / MT), SK_THREADS, Cfg::SMEM, ctx().stream, tw, ta, M, N, K, cs, ep);
    GTB_LAUNCHED();
    return GTB_OK;
}
template <int EPI>
static int launch_skinny_mt(SeqGemmPlan* p, int mt, const CUtensorMap& tw, const CUtensorMap& ta, int M, int N, int K, int cs, const SqEpi& ep) {
    if (mt == 16) return launch_skinny<16, EPI>(p->sk_attr[0][EPI], tw, ta, M, N, K, cs, ep);
    if (mt == 32) return launch_skinny<32, EPI>(p->sk_attr[1][EPI], tw, ta, M, N, K, cs, ep);
    return launch_skinny<64, EPI>(p->sk_attr[2][EPI], tw, ta, M, N, K, cs, ep);
}

// Which kernel takes an M x N product.  Few rows mean few tiles, and a CTA streams W at a fixed rate however short its tile is: cutting K is
// what brings the chip's bandwidth to bear, until about two CTAs per SM are resident (beyond that the further clusters wait for a second
// wave) or a CTA's share of K is too short to pay for its start.  So the split-K kernel takes a product as long as K can be cut in two within
// that many CTAs, and every product of up to 64 rows (one tile row: nothing to gain from persistence).  Measured cold, launch included:
// N = K = 2048, 24 rows: 18.5 / 15.3 / 13.2 us for 1 / 2 / 4 cuts; N = 6400, 40 rows: 20.6 / 18.4 / 16.8; N = 32000, 24 rows: 36.8 / 41.1 / 48.5;
// against the persistent kernel with 128 rows (N = K = 2048): 14.9 to 19.2, with 512 rows 19.1 to 20.5, with 800 rows 28.9 to 20.6.
struct SkChoice { int mt = 0, cs = 1; };
static SkChoice skinny_choice(int M, int N, int K) {
    SkChoice c;
    const int nt = (N + 127) / 128, slots = 2 * ctx().sm_count - 40, nkb = K / SQ_BK;
    int mt = M <= 16 ? 16 : M <= 32 ? 32 : 64;
    if (mt == 64 && M <= 64 && nt * 2 <= 64) mt = 32;
    const int tiles = nt * ((M + mt - 1) / mt);
    if (tiles * 2 > slots && M > 64) return c;
    c.mt = mt;
    while (c.cs < 8 && tiles * c.cs * 2 <= slots && nkb >= c.cs * 4) c.cs *= 2;
    return c;
}

// KW: K of W when A holds several pieces of it (fp32 epilogue only)
static int run(SeqGemmPlan* p, int epi, const void* A, int lda, const void* W, int ldw, int M, int N, int K, SqEpi ep, int KW = 0) {
    if (KW == 0) KW = K;
    if (!p || K <= 0 || (KW % SQ_BK) || (K % KW) || (lda % 8) || (ldw % 8) || (((uintptr_t)A | (uintptr_t)W) & 15)) return -1;
    CUtensorMap ta, tb;
    int rc;
    ep.w_blocks = KW / SQ_BK;
    const SkChoice sk = skinny_choice(M, N, K);
    if (sk.mt) {
        rc = make_map(p, &tb, W, N, KW, ldw, 128);
        if (rc) return rc;
        rc = make_map(p, &ta, A, M, K, lda, sk.mt);
        if (rc) return rc;
        if (epi == SQ_EPI_GELU) return launch_skinny_mt<SQ_EPI_GELU>(p, sk.mt, tb, ta, M, N, K, sk.cs, ep);
        if (epi == SQ_EPI_F32) return launch_skinny_mt<SQ_EPI_F32>(p, sk.mt, tb, ta, M, N, K, sk.cs, ep);
        return launch_skinny_mt<SQ_EPI_GEGLU>(p, sk.mt, tb, ta, M, N, K, sk.cs, ep);
    }
    if (epi == SQ_EPI_F32) {
        // 128-row tiles of A while one wave holds them all (half the MMA rate, but twice the SMs) or no second tile is needed, 256-row tiles
        // beyond (N = 5632, K = 1024, cold: 384 rows 16.3 against 17.7 us, 512 rows 21.2 against 17.8)
        const int bn = M <= 128 || ((M + 127) / 128) * ((N + 127) / 128) <= ctx().sm_count ? 128 : 256;
        rc = make_map(p, &tb, W, N, KW, ldw, SQ_BM);
        if (rc) return rc;
        rc = make_map(p, &ta, A, M, K, lda, bn);
        if (rc) return rc;
        return bn == 256 ? launch<256, SQ_EPI_F32, true>(p, tb, ta, M, N, K, ep) : launch<128, SQ_EPI_F32, true>(p, tb, ta, M, N, K, ep);
    }
    // 256-wide tiles when they still give every SM a tile; otherwise 128-wide
    const int mt = (M + SQ_BM - 1) / SQ_BM;
    // (the 128-wide MMA reads as much of A from shared memory per FLOP as the 256-wide one reads of A and W together: it runs at about
    // half the rate, so it only pays when 256-wide tiles would leave most SMs idle)
    const int bn = (N > 128 && mt * ((N + 255) / 256) * 2 >= ctx().sm_count) ? 256 : 128;
    rc = make_map(p, &ta, A, M, K, lda, SQ_BM);
    if (rc) return rc;
    rc = make_map(p, &tb, W, N, K, ldw, bn);
    if (rc) return rc;
    if (epi == SQ_EPI_GELU) return bn == 256 ? launch<256, SQ_EPI_GELU>(p, ta, tb, M, N, K, ep) : launch<128, SQ_EPI_GELU>(p, ta, tb, M, N, K, ep);
    return bn == 256 ? launch<256, SQ_EPI_GEGLU>(p, ta, tb, M, N, K, ep) : launch<128, SQ_EPI_GEGLU>(p, ta, tb, M, N, K, ep);
}

int seq_gemm_bf16(SeqGemmPlan* p, const void* A, int lda, const void* W, int ldw, float* C, int ldc, int M, int N, int K, const float* bias, int accumulate) {
    SqEpi ep{};
    ep.C = C; ep.ldc = ldc; ep.bias = bias; ep.accumulate = accumulate; ep.status = p ? p->d_status : nullptr;
    return run(p, SQ_EPI_F32, A, lda, W, ldw, M, N, K, ep);
}

int seq_gemm_split3(SeqGemmPlan* p, const void* A3, int lda3, const void* W, int ldw, float* C, int ldc, int M, int N, int K, const float* bias, int accumulate) {
    SqEpi ep{};
    ep.C = C; ep.ldc = ldc; ep.bias = bias; ep.accumulate = accumulate; ep.status = p ? p->d_status : nullptr;
    return run(p, SQ_EPI_F32, A3, lda3, W, ldw, M, N, 3 * K, ep, K);
}

int seq_gemm_bf16_gelu(SeqGemmPlan* p, const void* A, int lda, const void* W, int ldw, void* act, int ld_act, int M, int N, int K) {
    SqEpi ep{};
    ep.act = reinterpret_cast<__nv_bfloat16*>(act); ep.ld_act = ld_act; ep.status = p ? p->d_status : nullptr;
    return run(p, SQ_EPI_GELU, A, lda, W, ldw, M, N, K, ep);
}

int seq_gemm_bf16_grouped(SeqGemmPlan* p, const void* A, int lda, const void* W, int ldw, int M_pad, int N, int K, int n_groups, const int* tile_group,
                          float* C, int ldc, void* act, int ld_act, const float* row_w) {
    if (!p || K <= 0 || (K % SQ_BK) || (lda % 8) || (ldw % 8) || (((uintptr_t)A | (uintptr_t)W) & 15) || (M_pad % SQ_BM) || n_groups <= 0) return -1;
    SqEpi ep{};
    ep.C = C; ep.ldc = ldc; ep.act = reinterpret_cast<__nv_bfloat16*>(act); ep.ld_act = ld_act; ep.status = p->d_status;
    ep.tile_group = tile_group; ep.group_rows = N; ep.row_w = row_w;
    const int mt = M_pad / SQ_BM;
    const int bn = (N > 128 && mt * ((N + 255) / 256) * 2 >= ctx().sm_count) ? 256 : 128;
    CUtensorMap ta, tb;
    int rc = make_map(p, &ta, A, M_pad, K, lda, SQ_BM);
    if (rc) return rc;
    rc = make_map(p, &tb, W, n_groups * N, K, ldw, bn);
    if (rc) return rc;
    if (act) return bn == 256 ? launch<256, SQ_EPI_RELU2>(p, ta, tb, M_pad, N, K, ep) : launch<128, SQ_EPI_RELU2>(p, ta, tb, M_pad, N, K, ep);
    return bn == 256 ? launch<256, SQ_EPI_F32>(p, ta, tb, M_pad, N, K, ep) : launch<128, SQ_EPI_F32>(p, ta, tb, M_pad, N, K, ep);
}

int seq_gemm_bf16_geglu(SeqGemmPlan* p, const void* A, int lda, const void* W, int ldw, void* act, int ld_act, int act_off, int M, int N2, int K) {
    return seq_gemm_bf16_gated(p, A, lda, W, ldw, act, ld_act, act_off, M, N2, K, 0, nullptr);
}

int seq_gemm_bf16_gated(SeqGemmPlan* p, const void* A, int lda, const void* W, int ldw, void* act, int ld_act, int act_off, int M, int N2, int K, int act_kind,
                        const float* row_w) {
    if (N2 % 64) return -1;                      // whole (32 gate, 32 up) groups only
    SqEpi ep{};
    ep.act = reinterpret_cast<__nv_bfloat16*>(act); ep.ld_act = ld_act; ep.act_off = act_off; ep.status = p ? p->d_status : nullptr;
    ep.act_kind = act_kind; ep.row_w = row_w;
    return run(p, SQ_EPI_GEGLU, A, lda, W, ldw, M, N2, K, ep);
}

int seq_gemm_bf16_grouped_gated(SeqGemmPlan* p, const void* A, int lda, const void* W, int ldw, int M_pad, int N2, int K, int n_groups, const int* tile_group,
                                void* act, int ld_act, const float* row_w, int act_kind) {
    if (!p || K <= 0 || (K % SQ_BK) || (lda % 8) || (ldw % 8) || (((uintptr_t)A | (uintptr_t)W) & 15) || (M_pad % SQ_BM) || n_groups <= 0 || (N2 % 64) || !act) return -1;
    SqEpi ep{};
    ep.act = reinterpret_cast<__nv_bfloat16*>(act); ep.ld_act = ld_act; ep.status = p->d_status;
    ep.tile_group = tile_group; ep.group_rows = N2; ep.row_w = row_w; ep.act_kind = act_kind;
    const int mt = M_pad / SQ_BM;
    const int bn = (N2 > 128 && mt * ((N2 + 255) / 256) * 2 >= ctx().sm_count) ? 256 : 128;
    CUtensorMap ta, tb;
    int rc = make_map(p, &ta, A, M_pad, K, lda, SQ_BM);
    if (rc) return rc;
    rc = make_map(p, &tb, W, n_groups * N2, K, ldw, bn);
    if (rc) return rc;
    return bn == 256 ? launch<256, SQ_EPI_GEGLU>(p, ta, tb, M_pad, N2, K, ep) : launch<128, SQ_EPI_GEGLU>(p, ta, tb, M_pad, N2, K, ep);
}

}  // namespace seq
}  // namespace gtb
