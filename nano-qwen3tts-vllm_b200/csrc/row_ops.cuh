// row_ops.cuh - helpers shared by the per-row kernels of the hybrid decoders (hybrid_ops.cu, sink_attn.cu, recurrent.cu):
// activation-type conversion, block reductions, and the scalar functions the recurrences evaluate in float.
#pragma once

#include <math.h>

#include "common.cuh"

namespace b2 {
namespace row {

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// sum over the block; every thread gets the result.  `red` holds 33 floats.
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  __syncthreads();                       // red may still be read from a previous call
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float t = lane < nw ? red[lane] : 0.f;
    t = warp_sum(t);
    if (lane == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}

// ln(1 + e^x) without overflow; exact for every float x (no clamp of the result)
__device__ __forceinline__ float softplus_f(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }
// ln(sigmoid(x))
__device__ __forceinline__ float logsigmoid_f(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }

// The same for results that are rounded to bf16, with the approximate reciprocal (one unit in the last place; its argument is between 1 and 2, whatever
// x).  With the exponential's two and three roundings that is within 2^-21 of the result for every x, behind
// which bf16 rounds at 2^-9.  The exact division costs more than the rows it is formed for: layers of a state space 688 us with it, 663 here.
__device__ __forceinline__ float recip_f(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
template <typename T>
__device__ __forceinline__ float sigmoid_for(float x) {
  if constexpr (sizeof(T) == 2) {
    const float e = expf(-fabsf(x));
    return (x < 0.f ? e : 1.0f) * recip_f(1.0f + e);
  } else {
    return sigmoid_f(x);
  }
}
template <typename T>
__device__ __forceinline__ float silu_for(float x) {
  if constexpr (sizeof(T) == 2) {
    const float e = expf(-fabsf(x));
    return (x < 0.f ? x * e : x) * recip_f(1.0f + e);
  } else {
    return silu_f(x);
  }
}

#define B2_ROW_DTYPE_OK(dt) ((dt) == B2TTS_DTYPE_BF16 || (dt) == B2TTS_DTYPE_F32)

}  // namespace row
}  // namespace b2
