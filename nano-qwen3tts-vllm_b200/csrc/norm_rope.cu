// norm_rope.cu - a4/a5 (+a1 fused): RMSNorm, add+RMSNorm, and the fused per-head q/k RMSNorm +
// RoPE + paged KV write that replaces q_norm, k_norm, rotary_emb and store_kvcache as called
// from Qwen3TTSAttention.forward (models/qwen3_tts_share.py:96-106).
//
// All of these are HBM/launch-latency bound element-wise passes: 16-byte (hidden rows) or
// 4-byte-per-lane fully coalesced accesses, fp32 math, rounding points chosen by `rounding`:
//   B2TTS_ROUND_EAGER  layernorm.py:22-27 evaluated op by op: bf16(x*rstd) then bf16(. * w),
//                      rstd = 1/sqrt (correctly rounded, what ATen's CPU rsqrt does);
//   B2TTS_ROUND_FUSED  what torch-inductor emits for the same source on the GPU: fp32 through
//                      to one rounding at the store, rstd = rsqrtf.
// RoPE is never compiled in the reference, so it always keeps the three bf16 roundings of
// `(x*cos) + (rotate_half(x)*sin)` (rotary_embedding.py:33-34) and bf16 cos/sin (:138-139).
#include <stdlib.h>

#include "common.cuh"

namespace b2 {

template <bool EAGER>
__device__ __forceinline__ float rstd_of(float sumsq, int cols, float eps) {
  const float var = sumsq / (float)cols + eps;
  return EAGER ? 1.0f / sqrtf(var) : rsqrtf(var);
}

template <bool EAGER>
__device__ __forceinline__ uint4 norm_eight(const float* f, float rstd, uint4 w) {
  return make_uint4(norm_pair<EAGER>(f[0], f[1], rstd, w.x), norm_pair<EAGER>(f[2], f[3], rstd, w.y), norm_pair<EAGER>(f[4], f[5], rstd, w.z),
                    norm_pair<EAGER>(f[6], f[7], rstd, w.w));
}
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = lane < nw ? red[lane] : 0.f;
  t = warp_sum(t);
  return t;
}

// One CTA per row; every thread keeps up to MAXV 16-byte vectors of the row in registers.
constexpr int RMS_THREADS = 256;
constexpr int RMS_MAXV = 4;       // cols <= 8 * 256 * 4 = 8192

template <bool ADD, bool EAGER>
__global__ void __launch_bounds__(RMS_THREADS)
rmsnorm_kernel(const __nv_bfloat16* __restrict__ x, int64_t x_stride, const __nv_bfloat16* res,
               const __nv_bfloat16* __restrict__ w, __nv_bfloat16* y, __nv_bfloat16* res_out, int cols, float eps,
               int round_sum_first) {
  __shared__ float red[32];
  // programmatic dependent launch: between two GEMMs of a wide batch this kernel must neither drain the chain (the next
  // GEMM's CTAs become resident and stream their first weight tiles while it runs) nor start late itself
  pdl_launch();
  pdl_wait();
  const int row = blockIdx.x;
  const int nvec = cols >> 3;
  const __nv_bfloat16* xr = x + (int64_t)row * x_stride;
  float f[RMS_MAXV][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < RMS_MAXV; ++i) {
    const int v = threadIdx.x + i * RMS_THREADS;
    if (v < nvec) {
      uint4 r = ldg_v4(xr + 8 * v);
      f[i][0] = bf16lo(r.x); f[i][1] = bf16hi(r.x); f[i][2] = bf16lo(r.y); f[i][3] = bf16hi(r.y);
      f[i][4] = bf16lo(r.z); f[i][5] = bf16hi(r.z); f[i][6] = bf16lo(r.w); f[i][7] = bf16hi(r.w);
      if (ADD) {
        uint4 q = ldg_v4(res + (int64_t)row * cols + 8 * v);
        f[i][0] += bf16lo(q.x); f[i][1] += bf16hi(q.x); f[i][2] += bf16lo(q.y); f[i][3] += bf16hi(q.y);
        f[i][4] += bf16lo(q.z); f[i][5] += bf16hi(q.z); f[i][6] += bf16lo(q.w); f[i][7] += bf16hi(q.w);
        uint4 o;
        o.x = pack_bf16(f[i][0], f[i][1]); o.y = pack_bf16(f[i][2], f[i][3]);
        o.z = pack_bf16(f[i][4], f[i][5]); o.w = pack_bf16(f[i][6], f[i][7]);
        stg_v4(res_out + (int64_t)row * cols + 8 * v, o);
        if (round_sum_first) {
          f[i][0] = bf16lo(o.x); f[i][1] = bf16hi(o.x); f[i][2] = bf16lo(o.y); f[i][3] = bf16hi(o.y);
          f[i][4] = bf16lo(o.z); f[i][5] = bf16hi(o.z); f[i][6] = bf16lo(o.w); f[i][7] = bf16hi(o.w);
        }
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) ss = fmaf(f[i][e], f[i][e], ss);
    }
  }
  const float rstd = rstd_of<EAGER>(block_sum(ss, red), cols, eps);
#pragma unroll
  for (int i = 0; i < RMS_MAXV; ++i) {
    const int v = threadIdx.x + i * RMS_THREADS;
    if (v < nvec) {
      stg_v4(y + (int64_t)row * cols + 8 * v, norm_eight<EAGER>(f[i], rstd, ldg_v4(w + 8 * v)));
    }
  }
}

// Narrow rows (cols <= 256, e.g. the per-head norm over 128): one warp per row, 8 rows per CTA.
template <bool EAGER>
__global__ void __launch_bounds__(256)
rmsnorm_narrow_kernel(const __nv_bfloat16* __restrict__ x, int64_t x_stride, const __nv_bfloat16* __restrict__ w,
                      __nv_bfloat16* y, int rows, int cols, float eps) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const int nvec = cols >> 3;                       // <= 32
  const __nv_bfloat16* xr = x + (int64_t)row * x_stride;
  float f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  float ss = 0.f;
  if (lane < nvec) {
    uint4 r = ldg_v4(xr + 8 * lane);
    f[0] = bf16lo(r.x); f[1] = bf16hi(r.x); f[2] = bf16lo(r.y); f[3] = bf16hi(r.y);
    f[4] = bf16lo(r.z); f[5] = bf16hi(r.z); f[6] = bf16lo(r.w); f[7] = bf16hi(r.w);
#pragma unroll
    for (int e = 0; e < 8; ++e) ss = fmaf(f[e], f[e], ss);
  }
  const float rstd = rstd_of<EAGER>(warp_sum(ss), cols, eps);
  if (lane < nvec) {
    stg_v4(y + (int64_t)row * cols + 8 * lane, norm_eight<EAGER>(f, rstd, ldg_v4(w + 8 * lane)));
  }
}

// ------------------------------------------------------------------------------------------
// Fused q/k head-norm + RoPE + KV write.  One CTA per token, 8 warps; a warp owns one head at a
// time (lane l holds dims {2l, 2l+1, 64+2l, 64+2l+1} -> two fully coalesced 128-byte accesses) and walks heads
// warp, warp+8, ...  Cosines and sines are formed once a token, by 128 threads, while the rows of a warp's first four heads
// and of the values are on their way.  For steps of few tokens, see the kernel behind it.
struct QkRopeParams {
  const __nv_bfloat16 *q, *k, *v;
  int64_t q_stride, k_stride, v_stride;
  __nv_bfloat16 *q_out, *k_out;
  const __nv_bfloat16 *q_w, *k_w;
  float eps;
  const int64_t* positions;
  int64_t pos_row_stride;
  const float* inv_freq;
  const int32_t* modality;
  float attention_scaling;
  const int32_t* slot_mapping;
  __nv_bfloat16 *k_cache, *v_cache;
  int num_heads, num_kv_heads;
};

template <bool EAGER>
__global__ void __launch_bounds__(256)
qknorm_rope_kvwrite_kernel(const QkRopeParams p) {
  constexpr int HD = 128;
  const int tok = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kv_dim = p.num_kv_heads * HD;
  const int slot = p.slot_mapping ? __ldg(p.slot_mapping + tok) : -1;

  const int total = p.num_heads + p.num_kv_heads;
  constexpr int AHEAD = 4;                             // heads whose rows are asked for at once
  uint32_t r1[AHEAD], r2[AHEAD];
  auto fetch = [&](int h0) {
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const int hh = h0 + 8 * i;
      r1[i] = r2[i] = 0;
      if (hh < total) {
        const __nv_bfloat16* src = hh >= p.num_heads ? p.k + (int64_t)tok * p.k_stride + (hh - p.num_heads) * HD : p.q + (int64_t)tok * p.q_stride + hh * HD;
        r1[i] = *reinterpret_cast<const uint32_t*>(src + 2 * lane);
        r2[i] = *reinterpret_cast<const uint32_t*>(src + 64 + 2 * lane);
      }
    }
  };
  fetch(warp);
  const bool put_v = slot >= 0 && p.v;                 // V goes to the cache untouched
  uint4 v0 = make_uint4(0, 0, 0, 0);
  if (put_v && threadIdx.x < (kv_dim >> 3)) v0 = ldg_nc_v4(p.v + (int64_t)tok * p.v_stride + 8 * threadIdx.x);
  // cos/sin of columns f (turns[0]) and 64 + f (turns[1]): fp32 angle, fp32 cos/sin, bf16 result.  Both share frequency f but - in the
  // sectioned M-RoPE branch (rotary_embedding.py:73-80) - not necessarily the position row.
  __shared__ __align__(4) __nv_bfloat16 turns[2][2][HD / 2];          // [column half][cosine, sine]
  if (threadIdx.x < HD) {
    const int f = threadIdx.x & 63;
    const int m = p.modality ? __ldg(p.modality + threadIdx.x) : 0;
    const float ang = (float)__ldg(p.positions + (int64_t)m * p.pos_row_stride + tok) * __ldg(p.inv_freq + f);
    turns[threadIdx.x >> 6][0][f] = __float2bfloat16_rn(cosf(ang) * p.attention_scaling);
    turns[threadIdx.x >> 6][1][f] = __float2bfloat16_rn(sinf(ang) * p.attention_scaling);
  }
  __syncthreads();
  const auto pair_of = [&](int half, int part) { return *reinterpret_cast<const uint32_t*>(&turns[half][part][2 * lane]); };
  const uint32_t c1 = pair_of(0, 0), s1 = pair_of(0, 1), c2 = pair_of(1, 0), s2 = pair_of(1, 1);

  for (int h0 = warp; h0 < total; h0 += 8 * AHEAD) {
    if (h0 != warp) fetch(h0);
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const int hh = h0 + 8 * i;
      if (hh >= total) break;
      const bool is_k = hh >= p.num_heads;
      const int h = is_k ? hh - p.num_heads : hh;
      const __nv_bfloat16* w = is_k ? p.k_w : p.q_w;
      uint32_t x1 = r1[i], x2 = r2[i];
      if (w) {
        float ss = bf16lo(x1) * bf16lo(x1);
        ss = fmaf(bf16hi(x1), bf16hi(x1), ss); ss = fmaf(bf16lo(x2), bf16lo(x2), ss); ss = fmaf(bf16hi(x2), bf16hi(x2), ss);
        const float rstd = rstd_of<EAGER>(warp_sum(ss), HD, p.eps);
        x1 = norm_pair<EAGER>(x1, rstd, *reinterpret_cast<const uint32_t*>(w + 2 * lane));
        x2 = norm_pair<EAGER>(x2, rstd, *reinterpret_cast<const uint32_t*>(w + 64 + 2 * lane));
      }
      const uint32_t y1 = turn_first(x1, x2, c1, s1), y2 = turn_second(x1, x2, c2, s2);
      __nv_bfloat16* dst = nullptr;
      if (is_k) {
        if (p.k_out) dst = p.k_out + (int64_t)tok * kv_dim + h * HD;
        if (slot >= 0) {
          __nv_bfloat16* cd = p.k_cache + (int64_t)slot * kv_dim + h * HD;
          *reinterpret_cast<uint32_t*>(cd + 2 * lane) = y1;
          *reinterpret_cast<uint32_t*>(cd + 64 + 2 * lane) = y2;
        }
      } else {
        dst = p.q_out + ((int64_t)tok * p.num_heads + h) * HD;
      }
      if (dst) {
        *reinterpret_cast<uint32_t*>(dst + 2 * lane) = y1;
        *reinterpret_cast<uint32_t*>(dst + 64 + 2 * lane) = y2;
      }
    }
  }
  if (put_v) {
    const __nv_bfloat16* vs = p.v + (int64_t)tok * p.v_stride;
    __nv_bfloat16* vd = p.v_cache + (int64_t)slot * kv_dim;
    if (threadIdx.x < (kv_dim >> 3)) stg_v4(vd + 8 * threadIdx.x, v0);
    for (int i = threadIdx.x + blockDim.x; i < (kv_dim >> 3); i += blockDim.x) stg_v4(vd + 8 * i, ldg_nc_v4(vs + 8 * i));
  }
}

// The same for many tokens: a thread keeps coordinates 4m .. 4m + 3 and 64 + 4m .. of one head (a turn's partners; sixteen threads have a head) over QK_WALK
// consecutive tokens, with its norm weights in registers and the pieces of the next four tokens on their way; the angles of all QK_WALK tokens are formed first, in
// shared memory.  Two tokens share one tree of shuffles and one root, summed in the order of the kernel above: results are the same bits.
// Bound: HBM (14 us at the copy rate without k_out) and instructions.  Tokens of 16 + 8 + 8 heads with k_out in us, above with float arithmetic and a conversion for
// every rounding / above / this one: 5627 35.9 / 29.9 / 23.9, 1184 10.2 / 7.9 / 6.5; 3000 of 32 + 4 + 4 28.0 / 20.9 / 15.7; 1189 of 3 + 1 + 1 5.8 / 5.3 / 4.5.
// Runs of 8 tokens 24.7, 7.0, 16.4, 5.7, of 16 25.0, 9.8, 18.9, 9.5.  Few tokens stay above: 300 of 4 + 2 + 2 heads 3.5, here 4.0.
constexpr int QK_WALK = 4, QK_AHEAD = 2;

template <bool EAGER>
__global__ void __launch_bounds__(256, 4)
qknorm_rope_walk_kernel(const QkRopeParams p, int n_tokens) {
  constexpr int HD = 128;
  __shared__ __align__(16) __nv_bfloat16 turns[QK_WALK][4][HD / 2];  // cosines and sines of the first columns, then (sectioned positions) of the others
  const int t0 = blockIdx.x * QK_WALK, cnt = min(QK_WALK, n_tokens - t0), lane = threadIdx.x & 31;
  const bool put_v = p.slot_mapping != nullptr && p.v != nullptr;
  const int heads = p.num_heads + p.num_kv_heads * (put_v ? 2 : 1), kv_dim = p.num_kv_heads * HD;
  const int i = blockIdx.y * 256 + threadIdx.x, head = i >> 4, col = (i & 15) * 4;
  const bool live = head < heads, is_q = head < p.num_heads, is_k = !is_q && head < p.num_heads + p.num_kv_heads;
  const int h = is_q ? head : is_k ? head - p.num_heads : head - p.num_heads - p.num_kv_heads;
  const __nv_bfloat16* src = (is_q ? p.q : is_k ? p.k : p.v) + h * HD + col;
  const int64_t stride = is_q ? p.q_stride : is_k ? p.k_stride : p.v_stride;
  uint2 x1[QK_WALK], x2[QK_WALK];
  int slot[QK_WALK];
  auto load = [&](int t) {
    x1[t] = x2[t] = make_uint2(0u, 0u);
    slot[t] = -1;
    if (live && t < cnt) {
      x1[t] = ldg_v2(src + (t0 + t) * stride);
      x2[t] = ldg_v2(src + (t0 + t) * stride + HD / 2);
      if (!is_q && p.slot_mapping != nullptr) slot[t] = __ldg(p.slot_mapping + t0 + t);
    }
  };
#pragma unroll
  for (int t = 0; t < QK_AHEAD; ++t) load(t);
  const int planes = p.modality != nullptr ? 2 : 1;
  for (int a = threadIdx.x; a < cnt * planes * (HD / 2); a += 256) {
    const int f = a & 63, t = (a >> 6) / planes, half = (a >> 6) - t * planes;
    const int m = planes == 2 ? __ldg(p.modality + half * 64 + f) : 0;
    const float ang = (float)__ldg(p.positions + (int64_t)m * p.pos_row_stride + t0 + t) * __ldg(p.inv_freq + f);
    turns[t][2 * half][f] = __float2bfloat16_rn(cosf(ang) * p.attention_scaling);
    turns[t][2 * half + 1][f] = __float2bfloat16_rn(sinf(ang) * p.attention_scaling);
  }
  const __nv_bfloat16* w = is_q ? p.q_w : is_k ? p.k_w : nullptr;
  uint32_t w1[2] = {}, w2[2] = {};
  if (live && w != nullptr) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      w1[e] = *reinterpret_cast<const uint32_t*>(w + col + 2 * e);
      w2[e] = *reinterpret_cast<const uint32_t*>(w + HD / 2 + col + 2 * e);
    }
  }
  __syncthreads();
  if (((i & ~31) >> 4) >= heads) return;                  // a warp stays together for the shuffles
#pragma unroll
  for (int t = 0; t < QK_WALK; t += 2) {
    if (t >= cnt) break;
#pragma unroll
    for (int k = QK_AHEAD; k < QK_AHEAD + 2; ++k) if (t + k < QK_WALK) load(t + k);
    float rstd[2] = {1.f, 1.f};
    if (p.q_w != nullptr) {
      float ss[2][2];
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const uint32_t a = e ? x1[t + k].y : x1[t + k].x, b = e ? x2[t + k].y : x2[t + k].x;
          float v = bf16lo(a) * bf16lo(a);
          v = fmaf(bf16hi(a), bf16hi(a), v);
          v = fmaf(bf16lo(b), bf16lo(b), v);
          ss[k][e] = fmaf(bf16hi(b), bf16hi(b), v);
        }
      // upper eight of the sixteen threads go on with the second sums, every other four with the second token
      const bool up = lane & 8, second = lane & 4;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float keep = up ? ss[k][1] : ss[k][0];
        ss[k][0] = keep + __shfl_xor_sync(0xffffffffu, up ? ss[k][0] : ss[k][1], 8);
      }
      float v = second ? ss[1][0] : ss[0][0];
      v += __shfl_xor_sync(0xffffffffu, second ? ss[0][0] : ss[1][0], 4);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 8);
      v = rstd_of<EAGER>(v, HD, p.eps);
      rstd[0] = __shfl_sync(0xffffffffu, v, lane & ~4);
      rstd[1] = __shfl_sync(0xffffffffu, v, lane | 4);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int tok = t0 + t + k;
      uint2 y1 = x1[t + k], y2 = x2[t + k];
      if (is_q || is_k) {
        if (w != nullptr) {
          y1 = make_uint2(norm_pair<EAGER>(y1.x, rstd[k], w1[0]), norm_pair<EAGER>(y1.y, rstd[k], w1[1]));
          y2 = make_uint2(norm_pair<EAGER>(y2.x, rstd[k], w2[0]), norm_pair<EAGER>(y2.y, rstd[k], w2[1]));
        }
        const __nv_bfloat16 *first = &turns[t + k][0][col], *other = first + (planes - 1) * HD;
        const uint2 c1 = ldg_v2(first), s1 = ldg_v2(first + HD / 2), c2 = ldg_v2(other), s2 = ldg_v2(other + HD / 2), a = y1, b = y2;
        y1 = make_uint2(turn_first(a.x, b.x, c1.x, s1.x), turn_first(a.y, b.y, c1.y, s1.y));
        y2 = make_uint2(turn_second(a.x, b.x, c2.x, s2.x), turn_second(a.y, b.y, c2.y, s2.y));
      }
      if (!live || t + k >= cnt) continue;
      auto put = [&](__nv_bfloat16* dst) { stg_v2(dst, y1); stg_v2(dst + HD / 2, y2); };
      if (is_q) {
        put(p.q_out + ((int64_t)tok * p.num_heads + h) * HD + col);
      } else {
        if (is_k && p.k_out) put(p.k_out + (int64_t)tok * kv_dim + h * HD + col);
        if (slot[t + k] >= 0) put((is_k ? p.k_cache : p.v_cache) + (int64_t)slot[t + k] * kv_dim + h * HD + col);
      }
    }
  }
}

}  // namespace b2

extern "C" int b2tts_rmsnorm(const void* x, int64_t x_row_stride, const void* w, void* y,
                             int rows, int cols, float eps, int rounding, void* stream) {
  using namespace b2;
  B2_REQUIRE(rows >= 0 && cols > 0, B2TTS_EINVAL, "rmsnorm: rows=%d cols=%d", rows, cols);
  if (rows == 0) return B2TTS_OK;
  B2_REQUIRE(x && w && y, B2TTS_EINVAL, "rmsnorm: null pointer");
  B2_REQUIRE(cols % 8 == 0 && x_row_stride % 8 == 0 && aligned16(x) && aligned16(w) && aligned16(y), B2TTS_EALIGN,
             "rmsnorm: cols/stride must be multiples of 8 and pointers 16-byte aligned");
  B2_REQUIRE(cols <= 8 * RMS_THREADS * RMS_MAXV, B2TTS_EUNSUPPORTED, "rmsnorm: cols %d > %d", cols,
             8 * RMS_THREADS * RMS_MAXV);
  B2_REQUIRE(rounding == B2TTS_ROUND_EAGER || rounding == B2TTS_ROUND_FUSED, B2TTS_EINVAL, "rmsnorm: rounding %d", rounding);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto xp = static_cast<const __nv_bfloat16*>(x);
  auto wp = static_cast<const __nv_bfloat16*>(w);
  auto yp = static_cast<__nv_bfloat16*>(y);
  if (cols <= 256) {
    const int grid = (rows + 7) / 8;
    if (rounding == B2TTS_ROUND_EAGER) rmsnorm_narrow_kernel<true><<<grid, 256, 0, st>>>(xp, x_row_stride, wp, yp, rows, cols, eps);
    else rmsnorm_narrow_kernel<false><<<grid, 256, 0, st>>>(xp, x_row_stride, wp, yp, rows, cols, eps);
  } else {
    // launched as a programmatic dependent (B2TTS_PDL_NORM=0: a plain launch); correct after any kernel - one that never
    // executes griddepcontrol.launch_dependents releases its dependents when it completes
    static const bool pdl = [] { const char* e = getenv("B2TTS_PDL_NORM"); return !(e && e[0] == '0'); }();
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(rows, 1, 1);
    cfg.blockDim = dim3(RMS_THREADS, 1, 1);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    const __nv_bfloat16* nores = nullptr;
    __nv_bfloat16* noout = nullptr;
    cudaError_t e = rounding == B2TTS_ROUND_EAGER
        ? cudaLaunchKernelEx(&cfg, rmsnorm_kernel<false, true>, xp, x_row_stride, nores, wp, yp, noout, cols, eps, 0)
        : cudaLaunchKernelEx(&cfg, rmsnorm_kernel<false, false>, xp, x_row_stride, nores, wp, yp, noout, cols, eps, 0);
    if (e != cudaSuccess) return cuda_fail(e, "rmsnorm");
  }
  B2_CHECK_LAUNCH("rmsnorm");
  return B2TTS_OK;
}

extern "C" int b2tts_add_rmsnorm(const void* x, const void* res, const void* w, void* y, void* res_out,
                                 int rows, int cols, float eps, int rounding, int round_sum_first,
                                 void* stream) {
  using namespace b2;
  B2_REQUIRE(rows >= 0 && cols > 0, B2TTS_EINVAL, "add_rmsnorm: rows=%d cols=%d", rows, cols);
  if (rows == 0) return B2TTS_OK;
  B2_REQUIRE(x && res && w && y && res_out, B2TTS_EINVAL, "add_rmsnorm: null pointer");
  B2_REQUIRE(cols % 8 == 0 && aligned16(x) && aligned16(res) && aligned16(w) && aligned16(y) && aligned16(res_out),
             B2TTS_EALIGN, "add_rmsnorm: cols must be a multiple of 8 and pointers 16-byte aligned");
  B2_REQUIRE(cols <= 8 * RMS_THREADS * RMS_MAXV, B2TTS_EUNSUPPORTED, "add_rmsnorm: cols %d > %d", cols,
             8 * RMS_THREADS * RMS_MAXV);
  B2_REQUIRE(rounding == B2TTS_ROUND_EAGER || rounding == B2TTS_ROUND_FUSED, B2TTS_EINVAL, "add_rmsnorm: rounding %d", rounding);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto xp = static_cast<const __nv_bfloat16*>(x);
  auto rp = static_cast<const __nv_bfloat16*>(res);
  auto wp = static_cast<const __nv_bfloat16*>(w);
  auto yp = static_cast<__nv_bfloat16*>(y);
  auto op = static_cast<__nv_bfloat16*>(res_out);
  if (rounding == B2TTS_ROUND_EAGER)
    rmsnorm_kernel<true, true><<<rows, RMS_THREADS, 0, st>>>(xp, cols, rp, wp, yp, op, cols, eps, round_sum_first);
  else
    rmsnorm_kernel<true, false><<<rows, RMS_THREADS, 0, st>>>(xp, cols, rp, wp, yp, op, cols, eps, round_sum_first);
  B2_CHECK_LAUNCH("add_rmsnorm");
  return B2TTS_OK;
}

extern "C" int b2tts_qknorm_rope_kvwrite(const void* q, int64_t q_row_stride,
                                         const void* k, int64_t k_row_stride,
                                         const void* v, int64_t v_row_stride,
                                         void* q_out, void* k_out,
                                         const void* q_weight, const void* k_weight, float eps,
                                         const int64_t* positions, int64_t pos_row_stride,
                                         const float* inv_freq, const int32_t* modality,
                                         float attention_scaling,
                                         const int32_t* slot_mapping, void* k_cache, void* v_cache,
                                         int n_tokens, int num_heads, int num_kv_heads, int head_dim,
                                         int rounding, void* stream) {
  using namespace b2;
  const char* what = "qknorm_rope_kvwrite";
  B2_REQUIRE(n_tokens >= 0 && num_heads > 0 && num_kv_heads > 0, B2TTS_EINVAL, "%s: n=%d heads=%d kv=%d", what,
             n_tokens, num_heads, num_kv_heads);
  if (n_tokens == 0) return B2TTS_OK;
  B2_REQUIRE(head_dim == 128, B2TTS_EUNSUPPORTED, "%s: head_dim %d unsupported (128)", what, head_dim);
  B2_REQUIRE(q && k && q_out && positions && inv_freq, B2TTS_EINVAL, "%s: null pointer", what);
  B2_REQUIRE((q_weight == nullptr) == (k_weight == nullptr), B2TTS_EINVAL, "%s: q/k weights must both be set or both NULL", what);
  if (slot_mapping) B2_REQUIRE(k_cache && v_cache && v, B2TTS_EINVAL, "%s: slot_mapping needs v, k_cache, v_cache", what);
  B2_REQUIRE(q_row_stride % 8 == 0 && k_row_stride % 8 == 0 && v_row_stride % 8 == 0 && aligned16(q) && aligned16(k) &&
                 aligned16(v) && aligned16(q_out) && aligned16(k_out) && aligned16(k_cache) && aligned16(v_cache),
             B2TTS_EALIGN, "%s: strides must be multiples of 8 and pointers 16-byte aligned", what);
  B2_REQUIRE(rounding == B2TTS_ROUND_EAGER || rounding == B2TTS_ROUND_FUSED, B2TTS_EINVAL, "%s: rounding %d", what, rounding);
  QkRopeParams p{};
  p.q = static_cast<const __nv_bfloat16*>(q); p.k = static_cast<const __nv_bfloat16*>(k);
  p.v = static_cast<const __nv_bfloat16*>(v);
  p.q_stride = q_row_stride; p.k_stride = k_row_stride; p.v_stride = v_row_stride;
  p.q_out = static_cast<__nv_bfloat16*>(q_out); p.k_out = static_cast<__nv_bfloat16*>(k_out);
  p.q_w = static_cast<const __nv_bfloat16*>(q_weight); p.k_w = static_cast<const __nv_bfloat16*>(k_weight);
  p.eps = eps; p.positions = positions; p.pos_row_stride = pos_row_stride;
  p.inv_freq = inv_freq; p.modality = modality; p.attention_scaling = attention_scaling;
  p.slot_mapping = slot_mapping;
  p.k_cache = static_cast<__nv_bfloat16*>(k_cache); p.v_cache = static_cast<__nv_bfloat16*>(v_cache);
  p.num_heads = num_heads; p.num_kv_heads = num_kv_heads;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (n_tokens >= 8 * sm_count()) {                       // enough runs of tokens for every multiprocessor
    const int heads = num_heads + num_kv_heads * (slot_mapping && v ? 2 : 1);
    const dim3 grid((n_tokens + QK_WALK - 1) / QK_WALK, (heads * 16 + 255) / 256);
    if (rounding == B2TTS_ROUND_EAGER) qknorm_rope_walk_kernel<true><<<grid, 256, 0, st>>>(p, n_tokens);
    else qknorm_rope_walk_kernel<false><<<grid, 256, 0, st>>>(p, n_tokens);
  } else if (rounding == B2TTS_ROUND_EAGER) qknorm_rope_kvwrite_kernel<true><<<n_tokens, 256, 0, st>>>(p);
  else qknorm_rope_kvwrite_kernel<false><<<n_tokens, 256, 0, st>>>(p);
  B2_CHECK_LAUNCH(what);
  return B2TTS_OK;
}
