// grouped_gemm.cuh - what the grouped products of grouped_gemm.cu and grouped_gemm_tc.cu share.
#pragma once

#include "clamped_gate.cuh"

namespace b2 {

// activations: from GG_CLAMPED on W[e] is [gate; up] and the output has half as many columns
enum { GG_NONE = 0, GG_RELU_SQ = 1, GG_CLAMPED = 2, GG_SILU = 3 };

template <int ACT>
__device__ __forceinline__ float gated_value(float gate, float up, float limit, float alpha) {
  if constexpr (ACT == GG_SILU) return gate / (1.0f + expf(-gate)) * up;
  return clamped_gate(gate, up, limit, alpha);
}

// the tcgen05 kernel's range (w_rows = rows of W per expert), see grouped_gemm_tc.cu
bool grouped_tc_applies(int n_pairs, int experts, int w_rows, int k, bool gated, bool in_by_token, int64_t ldc, const void* c);
// an error, once, when a wait inside an earlier launch has run out
int grouped_tc_check(const char* what);
// `n` = rows of W per expert (twice the output columns from GG_CLAMPED on)
int launch_grouped_tc(const char* what, const void* a, int64_t lda, const void* w, void* c, int64_t ldc, const int32_t* offsets,
                      const int32_t* sorted_pair, int n_pairs, int experts, int n, int k, int top, int in_by_token, int out_by_pair,
                      int act, float limit, float alpha, cudaStream_t st);

}  // namespace b2
