// portion_attn.cuh - softmax attention of prompt portions on tcgen05 (portion_attn.cu): its arguments and launch.
#pragma once

#include "row_ops.cuh"

namespace b2 {
namespace row {

struct PortionArgs {
  const __nv_bfloat16* q; int64_t q_tok, q_head; int n_tokens;     // (token t, head h, i) at q[t * q_tok + h * q_head + i]
  // keys: row r has coordinates [0, d1) at k[r * k_row + g * d1 + i] and [d1, d) at k2[r * k2_row + i - d1], shared by the heads; values at
  // v[r * v_row + gv * dv + c].  r is the cache slot of the key (block_tables), or key_start[b] + j without tables; n_rows bounds it
  const __nv_bfloat16* k; int64_t k_row; int d1;
  const __nv_bfloat16* k2; int64_t k2_row;
  const __nv_bfloat16* v; int64_t v_row;
  int64_t n_rows;
  const int32_t* block_tables; int64_t bt_stride; int page;
  const int32_t* key_start;
  const int32_t *seq_start, *seq_pos0, *seq_len;
  const int32_t* cu;                                  // not null: sequence b is tokens cu[b] .. cu[b + 1] - 1 of q, k and v, from position 0 on
  int one_token;                                      // sequences of one token are taken too
  int round_weights;                                  // the weights enter the second product rounded to bf16 once, not as pairs
  const float* sink;                                  // [H] or null
  const __nv_bfloat16* gate; int64_t ldg; int gate_el;
  void* out; int out_f32;                             // [tokens, H * dv]
  int H, G, Gv, d, dv;
  int mask_kind, mask, keep_first;                    // as sink_attn
  float softcap, scale;
  // not null: no softmax, the weight of distance x = position - key is 1 / (1 + exp(r1[h] ln(1 + r2[h] x) - pb[h] - scale score)); a window, nothing kept
  const float *r1, *r2, *pb;
  int n_seqs, max_new;
};

bool portion_attn_applies(const PortionArgs& a);
int launch_portion_attn(const char* what, const PortionArgs& a, cudaStream_t st);

}  // namespace row
}  // namespace b2
