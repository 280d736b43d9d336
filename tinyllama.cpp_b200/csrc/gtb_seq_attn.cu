// gtb_seq_attn.cu -- attention of prompt portions (bf16 mode) on the 5th-generation tensor cores: softmax attention under a causal, windowed or
// chunked mask with an optional sink, soft cap and distance slope, and sigmoid attention.
//
// A CTA owns 128 consecutive rows of one segment and one query unit; two CTAs share an SM.  Warps 0-3 hold one row per thread (TMEM lane =
// row): scores from TMEM, mask, weights in fp32, bf16 weights back to TMEM.  Warp 4 loads key and value tiles by TMA (128-byte swizzle), one
// thread of warp 5 issues the products:
//     S[128][64] = Q K^T      (Q staged once as bf16 in shared memory, K tile K-major)
//     O[128][VP] += P V       (P bf16 from TMEM, V tile as it lies in the cache: rows of keys, the MN-major B operand)
// There are two score and two weight buffers: while tile j's weights are computed, the scores of tile j + 1 and P V of tile j - 1 run, so the
// weight threads hardly ever wait for a product's latency.
// The softmax keeps its reference maximum until a row's scores exceed it by 2^8 and only then rescales O in TMEM (a rare event, the only one
// that waits for P V; weights up to 2^8 lose nothing in fp32 sums or bf16 operands).  Scores, weights, sums and the output are fp32, the
// weights enter P V as bf16.
//
// Bound: the products' issue -- a 64-wide MMA takes about 90 cycles of the tensor pipe whatever its share of the peak, eight of them per tile of 64
// keys and two CTAs per SM; the weights' exponentials would take 512 cycles per tile, the arithmetic of the products 256.  Two heads per CTA on
// 128-key tiles would need twice the TMEM.  One layer of 2048 rows x 32 heads of 64, causal: 45 us (380 TFLOP/s of its causal half) against 215
// for the mma.sync kernel; sigmoid weights 55 against 199; 128 | 128 latent heads 25 against 80.
//
// Every mbarrier wait is bounded as in gtb_seq_gemm.cu: a wait that does not complete raises the CTA's abort flag, every role leaves, TMEM is
// released and the status word of the plan is set.
#include "gtb_seq_attn.h"

#include <cuda_bf16.h>

#include "gtb_internal.h"
#include "gtb_seq_gemm.h"
#include "gtb_seq_gemm_plan.h"
#include "gtb_tc.cuh"

namespace gtb {
namespace seq {

constexpr int AT_THREADS = 192;

constexpr int AT_KT = 64;                         // keys per tile
template <int DP, int VP> struct AtCfg {
    static constexpr int STAGES = DP + VP == 256 ? 2 : 3;      // (two CTAs per SM)
    static constexpr uint32_t Q_BYTES = 128 * DP * 2, K_BYTES = AT_KT * DP * 2, V_BYTES = AT_KT * VP * 2;
    static constexpr uint32_t SMEM = Q_BYTES + STAGES * (K_BYTES + V_BYTES) + 1024 + 256;
    // TMEM columns: two score buffers, two weight buffers (two weights per column), output.  Values of 128 channels leave no room for weights of
    // their own: there a tile's weights replace its scores
    static constexpr bool P_OWN = VP == 64;
    static constexpr uint32_t COLS = 256, O_COL = P_OWN ? 3 * AT_KT : 2 * AT_KT;
    static __host__ __device__ constexpr uint32_t p_col(int j) { return P_OWN ? 2 * AT_KT + (j & 1) * (AT_KT / 2) : (j & 1) * AT_KT; }
    static_assert(O_COL + VP <= COLS, "TMEM columns");
    static constexpr uint32_t IDESC_S = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(AT_KT >> 3) << 17) | (8u << 24);
    static constexpr uint32_t IDESC_O = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | (8u << 17) | (8u << 24);      // B MN-major, N = 64
};

// D[tmem] (+)= A[tmem] . B[smem]: bf16 A from TMEM (lane = row, two K elements per column)
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, float* v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
        ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr) : "memory");
}
__device__ __forceinline__ float at_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t at_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float at_max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// every lane of the warp gets the same answer
__device__ __forceinline__ bool at_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    bool ok = false;
    for (int it = 0; it < (1 << 24); it++) {
        if (mbar_try_wait(bar, parity)) { ok = true; break; }
        if ((it & 1023) == 1023 && *abort_flag) break;
    }
    if (!ok) *abort_flag = 1;
    return __all_sync(0xffffffffu, ok);
}

template <int DP, int VP, bool SIG>
__global__ void __launch_bounds__(AT_THREADS, 2)
k_attn_tc(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const AttnTc a, int* status) {
    using Cfg = AtCfg<DP, VP>;
    constexpr int KT = AT_KT, AT_STAGES = Cfg::STAGES;
    extern __shared__ unsigned char smem_raw[];
    pdl_wait();
    // the CTA's tile: 128 rows of a segment.  Tiles are the slow grid dimension and a segment's last tiles, which sweep the most keys, come
    // first: every unit's longest tiles start before any shorter one
    int seg = -1, q0 = 0;
    for (int s = 0, idx = blockIdx.y; s < a.S; s++) {
        const int n = (a.seg_len[s] + 127) / 128;
        if (idx < n) { seg = s; q0 = (n - 1 - idx) * 128; break; }
        idx -= n;
    }
    if (seg < 0) return;
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sm_q = smem_u32(smem), sm_k = sm_q + Cfg::Q_BYTES, sm_v = sm_k + AT_STAGES * Cfg::K_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::Q_BYTES + AT_STAGES * (Cfg::K_BYTES + Cfg::V_BYTES));
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4 * AT_STAGES + 7);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t bb = smem_u32(bars);
    auto k_full = [&](int s) { return bb + 8u * s; };
    auto k_empty = [&](int s) { return bb + 8u * (AT_STAGES + s); };
    auto v_full = [&](int s) { return bb + 8u * (2 * AT_STAGES + s); };
    auto v_empty = [&](int s) { return bb + 8u * (3 * AT_STAGES + s); };
    // per score buffer: scores there, weights there, P V done; one for the staged queries
    auto s_bar = [&](int j) { return bb + 8u * (4 * AT_STAGES + (j & 1)); };
    auto p_bar = [&](int j) { return bb + 8u * (4 * AT_STAGES + 2 + (j & 1)); };
    auto o_bar = [&](int j) { return bb + 8u * (4 * AT_STAGES + 4 + (j & 1)); };
    const uint32_t q_bar = bb + 8u * (4 * AT_STAGES + 6);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int u = blockIdx.x, hd = u / a.maps, g = hd / (a.heads / a.kv_heads), ku = g * a.maps + u % a.maps;
    const int slot = a.seg_slot[seg], row0 = a.seg_row0[seg] + q0, nq = min(128, a.seg_len[seg] - q0);
    const int pos0 = a.row_pos[row0], last = pos0 + nq - 1;
    auto first_key = [&](int pos) {
        int lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;
        if (a.chunk > 0) lo = max(lo, pos / a.chunk * a.chunk);
        return lo;
    };
    const int t_lo = first_key(pos0), n_it = (last - t_lo) / KT + 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < 4 * AT_STAGES; s++) mbar_init(bb + 8u * s, 1);
        for (int j = 0; j < 2; j++) { mbar_init(s_bar(j), 1); mbar_init(p_bar(j), 128); mbar_init(o_bar(j), 1); }
        mbar_init(q_bar, 128);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) tmem_alloc(smem_u32(tmem_slot), Cfg::COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = *tmem_slot;
    pdl_trigger();                  // (behind the TMEM allocation)

    if (warp == 4) {
        if (lane == 0) {            // ---------------- TMA producer
            auto wait1 = [&](uint32_t bar, uint32_t parity) {
                for (int it = 0; it < (1 << 24); it++) {
                    if (mbar_try_wait(bar, parity)) return true;
                    if ((it & 1023) == 1023 && *abort_flag) return false;
                }
                *abort_flag = 1;
                return false;
            };
            for (int it = 0; it < n_it; it++) {
                const int s = it % AT_STAGES, ph = (it / AT_STAGES) & 1, y = slot * a.max_ctx + t_lo + it * KT;
                if (!wait1(k_empty(s), ph ^ 1)) break;
                mbar_expect_tx(k_full(s), Cfg::K_BYTES);
#pragma unroll
                for (int c = 0; c < DP / 64; c++) tma_load_2d(sm_k + s * Cfg::K_BYTES + c * (KT * 128), &tmK, k_full(s), ku * DP + c * 64, y);
                if (!wait1(v_empty(s), ph ^ 1)) break;
                mbar_expect_tx(v_full(s), Cfg::V_BYTES);
#pragma unroll
                for (int c = 0; c < VP / 64; c++) tma_load_2d(sm_v + s * Cfg::V_BYTES + c * (KT * 128), &tmV, v_full(s), g * VP + c * 64, y);
            }
        }
        __syncwarp();
    } else if (warp == 5) {         // ---------------- MMA issuer
        auto scores = [&](int j) {
            const int s = j % AT_STAGES;
            if (!at_wait(k_full(s), (j / AT_STAGES) & 1, abort_flag)) return false;
            tc_fence_after();
            if (lane == 0) {
                const uint32_t sk = sm_k + s * Cfg::K_BYTES;
#pragma unroll
                for (int k = 0; k < DP / 16; k++)
                    umma_f16(tm + (j & 1) * KT, umma_desc_sw128(sm_q + (k >> 2) * (128 * 128) + (k & 3) * 32), umma_desc_sw128(sk + (k >> 2) * (KT * 128) + (k & 3) * 32),
                             Cfg::IDESC_S, k > 0);
                umma_commit(k_empty(s));
                umma_commit(s_bar(j));
            }
            __syncwarp();
            return true;
        };
        bool ok = at_wait(q_bar, 0, abort_flag) && scores(0);
        if (ok && n_it > 1) ok = scores(1);
        for (int j = 0; ok && j < n_it; j++) {
            const int s = j % AT_STAGES;
            if (!(ok = at_wait(v_full(s), (j / AT_STAGES) & 1, abort_flag))) break;
            const int nk = last + 1 - (t_lo + j * KT);
            if (nk < KT) {          // rows behind the sequence's last token are whatever the cache held: zero weights must meet zeros
#pragma unroll
                for (int c = 0; c < VP / 64; c++) {
                    uint4* z = reinterpret_cast<uint4*>(smem + (sm_v - sm_q) + s * Cfg::V_BYTES + c * (KT * 128) + nk * 128);
                    for (int e = lane; e < (KT - nk) * 8; e += 32) z[e] = make_uint4(0, 0, 0, 0);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
            }
            if (!(ok = at_wait(p_bar(j), (j >> 1) & 1, abort_flag))) break;
            tc_fence_after();
            if (Cfg::P_OWN && j + 2 < n_it && !(ok = scores(j + 2))) break;      // tile j's scores have been read: the next ones need not wait for P V
            if (lane == 0) {
                const uint32_t sv = sm_v + s * Cfg::V_BYTES;
#pragma unroll
                for (int c = 0; c < VP / 64; c++)
#pragma unroll
                    for (int k = 0; k < KT / 16; k++)
                        umma_f16_ts(tm + Cfg::O_COL + c * 64, tm + Cfg::p_col(j) + k * 8, umma_desc_sw128(sv + c * (KT * 128) + k * 2048), Cfg::IDESC_O, j > 0 || k > 0);
                umma_commit(v_empty(s));
                umma_commit(o_bar(j));
            }
            __syncwarp();
            if (!Cfg::P_OWN && j + 2 < n_it) {     // the next scores replace the weights that this product reads
                if (!(ok = at_wait(o_bar(j), (j >> 1) & 1, abort_flag))) break;
                ok = scores(j + 2);
            }
        }
    } else {                        // ---------------- one row per thread
        // queries -> bf16, 128-byte swizzle, one 64-column tile after the other; the sign of the scale rides on them
        const float sgn = a.scale < 0.0f ? -1.0f : 1.0f;
#pragma unroll
        for (int e0 = 0; e0 < 128 * (DP / 8); e0 += 128 * 8) {
            float v[8][8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int e = e0 + i * 128 + threadIdx.x, r = e / (DP / 8), c8 = e % (DP / 8);
                const float* src = a.Q + (size_t)(row0 + r) * a.ldq + a.q_off + u * DP + c8 * 8;
                if (r < nq && (((uintptr_t)src) & 15) == 0) {
                    const float4 x = *reinterpret_cast<const float4*>(src), y = *reinterpret_cast<const float4*>(src + 4);
                    v[i][0] = x.x; v[i][1] = x.y; v[i][2] = x.z; v[i][3] = x.w; v[i][4] = y.x; v[i][5] = y.y; v[i][6] = y.z; v[i][7] = y.w;
                } else {
#pragma unroll
                    for (int j = 0; j < 8; j++) v[i][j] = r < nq ? src[j] : 0.0f;
                }
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int e = e0 + i * 128 + threadIdx.x, r = e / (DP / 8), c8 = e % (DP / 8);
                *reinterpret_cast<uint4*>(smem + (c8 >> 3) * (128 * 128) + r * 128 + (((c8 & 7) ^ (r & 7)) << 4)) =
                    make_uint4(at_pack(v[i][0] * sgn, v[i][1] * sgn), at_pack(v[i][2] * sgn, v[i][3] * sgn), at_pack(v[i][4] * sgn, v[i][5] * sgn), at_pack(v[i][6] * sgn, v[i][7] * sgn));
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_arrive(q_bar);

        const int r = threadIdx.x, pos = pos0 + r;
        const uint32_t tl = tm + ((uint32_t)(warp * 32) << 16);
        const int k_lo = first_key(pos);                                      // this row sees keys k_lo .. pos
        const int lo_last = first_key(pos0 + 127);
        const float kLog2e = 1.4426950408889634f;
        const bool plain = SIG || (a.softcap <= 0.0f && !a.slope);
        const float scale = fabsf(a.scale), sc2 = plain ? scale * kLog2e : 1.0f;
        const float inv_cap = a.softcap > 0.0f ? 1.0f / a.softcap : 0.0f, slope = a.slope ? a.slope[hd] * kLog2e : 0.0f;
        const float bias = SIG && a.pb ? a.pb[hd] * kLog2e : 0.0f;
        float m = (!SIG && a.sink) ? a.sink[hd] * kLog2e : -INFINITY, l = 0.0f;
        const float sink = m;
        bool ok = true;
        for (int it = 0; it < n_it; it++) {
            const int j0 = t_lo + it * KT;
            const uint32_t ts = tl + (it & 1) * KT;
            if (!(ok = at_wait(s_bar(it), (it >> 1) & 1, abort_flag))) break;
            tc_fence_after();
            float s[KT];
#pragma unroll
            for (int c = 0; c < KT / 32; c++) tmem_ld32_nowait(ts + c * 32, s + c * 32);
            tmem_wait_ld();
            if (!plain) {
#pragma unroll
                for (int k = 0; k < KT; k++) {
                    float v = s[k] * scale;
                    if (a.softcap > 0.0f) {
                        float th;
                        asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(v * inv_cap));
                        v = a.softcap * th;
                    }
                    s[k] = fmaf(v, kLog2e, -slope * (float)(pos - j0 - k));
                }
            }
            if (j0 + KT - 1 > pos0 || j0 < lo_last) {                          // some row of the tile does not see all of its keys
                const int hi = pos - j0, lo = k_lo - j0;
#pragma unroll
                for (int k = 0; k < KT; k++) s[k] = (k <= hi && k >= lo) ? s[k] : -INFINITY;
            }
            if (!SIG) {
                float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
                for (int k = 4; k + 8 <= KT; k += 8)
#pragma unroll
                    for (int i = 0; i < 4; i++) mx[i] = at_max3(mx[i], s[k + 2 * i], s[k + 2 * i + 1]);
                const float mn = fmaxf(m, at_max3(at_max3(mx[0], mx[1], mx[2]), mx[3], at_max3(at_max3(s[KT - 4], s[KT - 3], s[KT - 2]), s[KT - 1], s[KT - 1])) * sc2);
                const bool need = mn - m > 8.0f;
                if (__any_sync(0xffffffffu, need)) {
                    const float corr = need ? (m == -INFINITY ? 0.0f : at_exp2(m - mn)) : 1.0f;
                    if (need) { m = mn; l *= corr; }
                    if (it > 0) {
                        if (!(ok = at_wait(o_bar(it - 1), ((it - 1) >> 1) & 1, abort_flag))) break;      // P V of the tile before has to be in O
                        tc_fence_after();
#pragma unroll 1
                        for (int c = 0; c < VP; c += 16) {
                            float o[16];
                            uint32_t w[16];
                            tmem_ld16(tl + Cfg::O_COL + c, o);
#pragma unroll
                            for (int j = 0; j < 16; j++) w[j] = __float_as_uint(o[j] * corr);
                            tmem_st16(tl + Cfg::O_COL + c, w);
                        }
                    }
                }
            }
            if (Cfg::P_OWN && it > 1 && !(ok = at_wait(o_bar(it), ((it - 2) >> 1) & 1, abort_flag))) break;      // the product that read this weight buffer is done
            const float mu = m == -INFINITY ? 0.0f : m;
            float l0 = 0.0f, l1 = 0.0f;
#pragma unroll
            for (int c = 0; c < KT; c += 32) {
                uint32_t w[16];
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    float p0, p1;
                    if (SIG) {
                        // masked scores are -inf: 1 / (1 + 2^inf) = 0
                        p0 = __fdividef(1.0f, 1.0f + at_exp2(-fmaf(s[c + 2 * j], sc2, bias)));
                        p1 = __fdividef(1.0f, 1.0f + at_exp2(-fmaf(s[c + 2 * j + 1], sc2, bias)));
                    } else {
                        p0 = at_exp2(fmaf(s[c + 2 * j], sc2, -mu));
                        p1 = at_exp2(fmaf(s[c + 2 * j + 1], sc2, -mu));
                        l0 += p0; l1 += p1;
                    }
                    w[j] = at_pack(p0, p1);
                }
                tmem_st16(tl + Cfg::p_col(it) + c / 2, w);
            }
            l += l0 + l1;
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(p_bar(it));
        }
        if (ok && (ok = at_wait(o_bar(n_it - 1), ((n_it - 1) >> 1) & 1, abort_flag))) {
            tc_fence_after();
            float f = 1.0f;
            if (!SIG) {
                if (a.sink) l += at_exp2(sink - m);
                f = 1.0f / l;
            }
            const int row = row0 + r;
            if (!a.out_f) f *= a.out_scale;
            const float* gr = a.gsrc + (size_t)row * a.g_ld + a.g_off;
            if (!a.out_f && a.gate == 3 && r < nq) f *= 1.0f / (1.0f + expf(-gr[hd]));
#pragma unroll 1
            for (int c = 0; c < VP; c += 32) {
                float o[32];
                tmem_ld32(tl + Cfg::O_COL + c, o);
                if (r >= nq) continue;
                if (a.out_f) {
                    float* dst = a.out_f + (size_t)row * a.ld_f + u * VP + c;
#pragma unroll
                    for (int j = 0; j < 32; j++) dst[j] = o[j] * f;
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++) {
                        o[j] *= f;
                        if (a.gate == 1 || a.gate == 2) {
                            const float z = gr[u * VP + c + j], sg = 1.0f / (1.0f + expf(-z));
                            o[j] *= a.gate == 2 ? sg : z * sg;
                        }
                    }
                    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(a.out) + (size_t)row * a.ld_out + a.a_off + u * VP + c;
                    if ((((uintptr_t)dst) & 15) == 0) {
#pragma unroll
                        for (int j = 0; j < 32; j += 8)
                            *reinterpret_cast<uint4*>(dst + j) = make_uint4(at_pack(o[j], o[j + 1]), at_pack(o[j + 2], o[j + 3]), at_pack(o[j + 4], o[j + 5]), at_pack(o[j + 6], o[j + 7]));
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; j++) dst[j] = __float2bfloat16_rn(o[j]);
                    }
                }
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) atomicExch(status, 1);
    if (warp == 5) { tc_fence_after(); tmem_dealloc(tm, Cfg::COLS); }
}

static int map2d(SeqGemmPlan* p, CUtensorMap* m, const void* base, int rows, int cols, int ld, int box_rows) {
    const cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t gstr[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = p->enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(GTB_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d) for a %d x %d cache", (int)r, rows, cols);
    return GTB_OK;
}

template <int DP, int VP, bool SIG>
static int launch(SeqGemmPlan* p, const AttnTc& a, int n_tiles) {
    using Cfg = AtCfg<DP, VP>;
    CUtensorMap tk, tv;
    int rc = map2d(p, &tk, a.kc, a.cache_rows, a.kv_heads * a.maps * DP, a.ld_k, AT_KT);
    if (rc) return rc;
    rc = map2d(p, &tv, a.vc, a.cache_rows, a.kv_heads * VP, a.ld_v, AT_KT);
    if (rc) return rc;
    static bool attr = false;
    if (!attr) { GTB_CUDA(cudaFuncSetAttribute(k_attn_tc<DP, VP, SIG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM)); attr = true; }
    pdl_launch(k_attn_tc<DP, VP, SIG>, dim3(a.heads * a.maps, n_tiles), AT_THREADS, Cfg::SMEM, ctx().stream, tk, tv, a, p->d_status);
    GTB_LAUNCHED();
    return GTB_OK;
}

int seq_attn_tc(SeqGemmPlan* p, const AttnTc& a, int n_tiles) {
    if (!p || (a.dim != 64 && a.dim != 128) || (a.vdim != 64 && a.vdim != 128) || (a.ld_k % 8) || (a.ld_v % 8) || (((uintptr_t)a.kc | (uintptr_t)a.vc) & 15)) return -1;
    if (!(fabsf(a.scale) > 0.0f) || isinf(a.scale)) return -1;      // (masked scores are -inf before they are scaled)
    if (a.sigmoid) {
        if (a.dim == 64) return a.vdim == 64 ? launch<64, 64, true>(p, a, n_tiles) : launch<64, 128, true>(p, a, n_tiles);
        return a.vdim == 64 ? launch<128, 64, true>(p, a, n_tiles) : launch<128, 128, true>(p, a, n_tiles);
    }
    if (a.dim == 64) return a.vdim == 64 ? launch<64, 64, false>(p, a, n_tiles) : launch<64, 128, false>(p, a, n_tiles);
    return a.vdim == 64 ? launch<128, 64, false>(p, a, n_tiles) : launch<128, 128, false>(p, a, n_tiles);
}

}  // namespace seq
}  // namespace gtb
