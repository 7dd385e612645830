// prompt_attn.cuh - softmax attention of prompt portions on tcgen05 (prompt_attn_tc.cu): its arguments and launch.
#pragma once

#include "row_ops.cuh"

namespace b2 {
namespace row {

struct PromptAttnArgs {
  const __nv_bfloat16* q; int64_t q_tok, q_head;      // (token t, head h, i) at q[t * q_tok + h * q_head + i]
  // keys: row r has coordinates [0, d1) at k[r * k_row + g * k_head + i] and [d1, d) at k2[r * k2_row + i - d1], shared by the heads;
  // values at v[r * v_row + gv * v_head + c].  r is the cache slot of the key (block_tables), or key_start[b] + j without tables
  const __nv_bfloat16* k; int64_t k_row; int k_head, d1;
  const __nv_bfloat16* k2; int64_t k2_row;
  const __nv_bfloat16* v; int64_t v_row; int v_head;
  const int32_t* block_tables; int64_t bt_stride; int page;
  const int32_t* key_start;
  const int32_t *seq_start, *seq_pos0, *seq_len;
  const float* sink;                                  // [H] or null
  const __nv_bfloat16* gate; int64_t ldg; int gate_el;
  const float* freq; float rot_mult; int rot_dims;    // query coordinates d1 .. d1 + rot_dims - 1 are turned in pairs (2 i, 2 i + 1); 0: none
  void* out; int out_f32;                             // [tokens, H * dv]
  int H, G, Gv, d, dv;
  int mask_kind, mask, keep_first;                    // as sink_attn
  float softcap, scale;
  int split_weights;                                  // the weights enter the second product as a bf16 pair hi + lo (16 bits), or rounded once
  int n_seqs, max_new;
  int box_rows, page_shift, gate_vec;                 // set by the launch
};

bool prompt_attn_applies(const PromptAttnArgs& a);
int launch_prompt_attn(const char* what, const PromptAttnArgs& a, cudaStream_t st);

}  // namespace row
}  // namespace b2
