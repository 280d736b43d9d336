// gtb_seq_attn.h -- attention of prompt portions on the 5th-generation tensor cores (gtb_seq_attn.cu).
#pragma once
#include <stdint.h>

namespace gtb {
namespace seq {

struct SeqGemmPlan;
// One attention branch over the rows of a pass: unit u = head * maps + map of a row attends the keys of its K/V head (and map) and that head's
// values under the row's own mask; see PassTables / SoftAttn for the meaning of the tables and of the shared fields.
struct AttnTc {
    const int *seg_slot, *seg_row0, *seg_len, *row_pos;      // tables of the pass, S segments
    int S;
    const float* Q;              // queries: row r, unit u at Q[r * ldq + q_off + u * dim], fp32
    int ldq, q_off;
    const void *kc, *vc;         // bf16 caches [cache_rows][ld_k | ld_v]; slot s starts at row s * max_ctx
    int ld_k, ld_v, cache_rows, max_ctx;
    int heads, maps, kv_heads, dim, vdim;      // units = heads * maps
    float scale, softcap;
    int window, chunk;
    const float* sink;           // [heads] or null
    const float* slope;          // [heads] or null
    int sigmoid;                 // 1: weight = sigmoid(scale q.k + pb[head]), not normalised
    const float* pb;             // [heads] or null
    void* out;                   // bf16 [row][ld_out], unit u at a_off + u * vdim
    int ld_out, a_off;
    float out_scale;
    int gate;                    // 0: none, 1: silu, 2: logistic, 3: logistic of one number per head
    const float* gsrc;
    int g_ld, g_off;
    float* out_f;                // not null: fp32 [row][ld_f], unit-major, no gate and no weight, instead of out
    int ld_f;
};
// -1 (nothing launched): head sizes, alignments or scale that the kernel does not take
int seq_attn_tc(SeqGemmPlan* p, const AttnTc& a, int n_tiles);

}  // namespace seq
}  // namespace gtb
