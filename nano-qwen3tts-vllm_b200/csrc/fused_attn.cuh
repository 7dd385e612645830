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
// The same as pairs (2i, 2i + 1), and sixteen products with sums over the even and over the odd ones
__device__ __forceinline__ void fa_pairs8(const uint4& r, uint64_t* f) {
  f[0] = f2_pack(bf16lo(r.x), bf16hi(r.x)); f[1] = f2_pack(bf16lo(r.y), bf16hi(r.y));
  f[2] = f2_pack(bf16lo(r.z), bf16hi(r.z)); f[3] = f2_pack(bf16lo(r.w), bf16hi(r.w));
}
__device__ __forceinline__ float fa_dot16(const uint64_t* q, const uint64_t* k) {
  uint64_t d = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) d = f2_fma(q[i], k[i], d);
  float even, odd;
  f2_unpack(d, even, odd);
  return even + odd;
}
int fa_choose_nsplit(int rows, int max_ctx);

}  // namespace b2
