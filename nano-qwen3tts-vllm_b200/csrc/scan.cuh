// scan.cuh - the arguments of the recurrent scans (recurrent.cu token by token, recurrent_chunk.cu in chunks).
#pragma once

#include <climits>

#include "row_ops.cuh"

namespace b2 {
namespace row {

struct ScanArgs {
  const void* k; int64_t ldk;             // key-like vectors: (row, group g, i) at k[row * ldk + g * d + i]
  const void* q; int64_t ldq;             // query-like vectors, same layout
  const void* v; int64_t ldv;             // values: (row, head h, c) at v[row * ldv + h * dv + c]
  const float* coef;                      // [rows, H, 3] per-token scalars, see scan_kernel (SCAN_GATED: unused); the chunk kernels
                                          // read (decay, write scale, log of the decay)
  const float* head_decay;                // [H] or null: coef = (head_decay[h], 1, 1) for every token (coef itself is then unused)
  int min_len = 1, max_len = INT_MAX;     // only sequences with so many new tokens
  const float* decay; int64_t ldd;        // SCAN_GATED: per key channel, (row, head h, i) at decay[row * ldd + h * d + i]
  const float* skip;                      // [H] or null: out += skip[h] * value
  float* state;                           // [slots, H, d, dv]
  float* out;                             // [rows, H * dv]
  const int32_t* seq_start; const int32_t* seq_pos0; const int32_t* seq_len; const int32_t* seq_slot;
  int H, G, d, dv;
  float qscale;
  float* scores = nullptr;                // what chunks say without the state, formed ahead (chunk_scores_floats(), delta_prep_floats()), or null
  int divide;                             // linear: out = S^T q * qscale / coef[2] instead of S^T q * qscale
};

// bf16 portions in chunks on the tensor cores: which sizes and layouts, the longest portion that is faster token by token, and the
// launches (sequences of min_len tokens and more)
bool scan_chunk_applies(const ScanArgs& a);
int linear_walk_len(const ScanArgs& a, int n_seqs);
int delta_walk_len(const ScanArgs& a, int n_seqs);
int launch_linear_chunk(const char* what, const ScanArgs& a, int n_seqs, int longest, int64_t chunks, cudaStream_t st);
int64_t chunk_scores_floats(int n_tokens, int n_seqs, int G);
int launch_delta_chunk(const char* what, const ScanArgs& a, int n_seqs, int longest, cudaStream_t st);
int64_t delta_prep_floats(int n_tokens, int n_seqs, int H);

}  // namespace row
}  // namespace b2
