// fused_attn.cuh - what the one-launch decode attention (attention_fused.cu) and the persistent decode step (decode_rows.cu) share, so that both form the
// same sums: tokens per step of the online softmax, the exponential, and into how many splits a context is cut.
#pragma once

#include "common.cuh"

namespace b2 {

constexpr int FA_TILE = 8;

__device__ __forceinline__ float fa_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void fa_unpack8(const uint4& r, float* f) {
  f[0] = bf16lo(r.x); f[1] = bf16hi(r.x); f[2] = bf16lo(r.y); f[3] = bf16hi(r.y);
  f[4] = bf16lo(r.z); f[5] = bf16hi(r.z); f[6] = bf16lo(r.w); f[7] = bf16hi(r.w);
}
int fa_choose_nsplit(int rows, int max_ctx);

}  // namespace b2
