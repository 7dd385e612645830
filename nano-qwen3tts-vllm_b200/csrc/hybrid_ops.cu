// hybrid_ops.cu - per-row kernels of decoders that keep several copies of the residual stream ("streams", mixed by small
// learned matrices around every sublayer) and pair an attention branch with a recurrent branch in one mixer:
//   token + hashed-bigram embedding into all streams; the stream update after a sublayer fused with the read-out and
//   RMS norm in front of the next one; the final sum of the streams with its norm on gathered rows; the preparation of an
//   attention step (biases, RMS norm over a whole projection, half-split rotation, paged K/V write, values that are the
//   raw keys); a short causal convolution over time with an activation and its carried state; the gate and grouped RMS
//   norm on a recurrent branch's output.
//
// Activations are `T` = bf16 (serving) or float (the all-32-bit mode).  The streams, every norm, angle and gate are float
// in both.  Nothing allocates or synchronises; every launch is graph-capturable.
#include <algorithm>

#include "row_ops.cuh"

namespace b2 {
namespace row {

constexpr int ROW_THREADS = 256;
constexpr int MAX_STREAMS = 8;

// ------------------------------------------------------------------ embedding: token row + bigram row -> every stream
template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
embed_bigram_kernel(const int32_t* __restrict__ tokens, const int32_t* __restrict__ prev_tokens, const T* __restrict__ embed,
                    const T* __restrict__ bigram, float* __restrict__ xs, int cols, int streams, int vocab, int buckets,
                    int mul_prev, int mul_cur) {
  const int r = blockIdx.x;
  int tok = tokens[r];
  const int prev = prev_tokens[r];
  const T* br = nullptr;
  if (bigram != nullptr) {
    long long h = buckets;                                                   // a sequence's first token: the extra row
    if (prev >= 0) h = (static_cast<long long>(prev) * mul_prev + static_cast<long long>(tok) * mul_cur) % buckets;
    br = bigram + static_cast<size_t>(h) * cols;
  }
  tok = min(max(tok, 0), vocab - 1);
  const T* er = embed + static_cast<size_t>(tok) * cols;
  float* xr = xs + static_cast<size_t>(r) * streams * cols;
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    float v = to_f(er[c]);
    if (br != nullptr) v += to_f(br[c]);
    for (int s = 0; s < streams; ++s) xr[static_cast<size_t>(s) * cols + c] = v;
  }
}

// ------------------------------------------------------------------ stream update + read-out + norm
// Row r holds `streams` copies x_0 .. x_(s-1) of `cols` floats.  If y1 is given, all copies are replaced at once from
// the old ones: x_t <- sum_s mix[s, t] x_s + out_w[t] * (c1 * y1 + c2 * y2).  Then, if h is given, the read-out
// u = sum_s in_w[s] x_s (in_w null: the plain sum) is RMS-normed with norm_w into h.
template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
stream_mix_norm_kernel(float* __restrict__ xs, const T* __restrict__ y1, const T* __restrict__ y2, float c1, float c2,
                       const float* __restrict__ mix, const float* __restrict__ out_w, const float* __restrict__ in_w,
                       const float* __restrict__ norm_w, T* __restrict__ h, int cols, int streams, float eps) {
  __shared__ float red[33];
  __shared__ float s_mix[MAX_STREAMS * MAX_STREAMS], s_out[MAX_STREAMS], s_in[MAX_STREAMS];
  if (threadIdx.x < streams * streams && y1 != nullptr) s_mix[threadIdx.x] = mix[threadIdx.x];
  if (threadIdx.x < streams) {
    s_out[threadIdx.x] = y1 != nullptr ? out_w[threadIdx.x] : 0.f;
    s_in[threadIdx.x] = in_w != nullptr ? in_w[threadIdx.x] : 1.f;
  }
  __syncthreads();
  const size_t r = blockIdx.x;
  float* xr = xs + r * streams * cols;
  float ssq = 0.f;
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    float x[MAX_STREAMS];
#pragma unroll
    for (int s = 0; s < MAX_STREAMS; ++s) x[s] = s < streams ? xr[static_cast<size_t>(s) * cols + c] : 0.f;
    float u = 0.f;
    if (y1 != nullptr) {
      float y = c1 * to_f(y1[r * cols + c]);
      if (y2 != nullptr) y += c2 * to_f(y2[r * cols + c]);
#pragma unroll
      for (int t = 0; t < MAX_STREAMS; ++t) {
        if (t < streams) {
          float acc = 0.f;
#pragma unroll
          for (int s = 0; s < MAX_STREAMS; ++s) if (s < streams) acc += s_mix[s * streams + t] * x[s];
          acc += s_out[t] * y;
          xr[static_cast<size_t>(t) * cols + c] = acc;
          u += s_in[t] * acc;
        }
      }
    } else {
#pragma unroll
      for (int t = 0; t < MAX_STREAMS; ++t) if (t < streams) u += s_in[t] * x[t];
    }
    ssq += u * u;
  }
  if (h == nullptr) return;
  const float tot = block_sum(ssq, red);
  const float inv = 1.0f / sqrtf(tot / static_cast<float>(cols) + eps);
  T* hr = h + r * cols;
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {             // the same thread wrote these columns above
    float u = 0.f;
    for (int t = 0; t < streams; ++t) u += s_in[t] * xr[static_cast<size_t>(t) * cols + c];
    hr[c] = from_f<T>(u * inv * norm_w[c]);
  }
}

// four consecutive activations <-> floats (16-byte loads for float, 8-byte for bf16); p must be aligned accordingly
template <typename T> __device__ __forceinline__ float4 load4(const T* p);
template <> __device__ __forceinline__ float4 load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint2 r = ldg_v2(p);
  return make_float4(bf16lo(r.x), bf16hi(r.x), bf16lo(r.y), bf16hi(r.y));
}
template <typename T> __device__ __forceinline__ void store4(T* p, float4 v);
template <> __device__ __forceinline__ void store4<float>(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
template <> __device__ __forceinline__ void store4<__nv_bfloat16>(__nv_bfloat16* p, float4 v) {
  stg_v2(p, make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w)));
}

// The same update and read-out for rows of cols % 4 == 0 and cols <= 4 * SMV_KEEP * ROW_THREADS: a thread owns groups of
// four consecutive columns, moves them as vectors and keeps its read-out values in registers for the norm, so the
// streams are read once and written once.
constexpr int SMV_KEEP = 4;

template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
stream_mix_norm_vec4_kernel(float* __restrict__ xs, const T* __restrict__ y1, const T* __restrict__ y2, float c1, float c2,
                            const float* __restrict__ mix, const float* __restrict__ out_w, const float* __restrict__ in_w,
                            const float* __restrict__ norm_w, T* __restrict__ h, int cols, int streams, float eps) {
  __shared__ float red[33];
  __shared__ float s_mix[MAX_STREAMS * MAX_STREAMS], s_out[MAX_STREAMS], s_in[MAX_STREAMS];
  if (threadIdx.x < streams * streams && y1 != nullptr) s_mix[threadIdx.x] = mix[threadIdx.x];
  if (threadIdx.x < streams) {
    s_out[threadIdx.x] = y1 != nullptr ? out_w[threadIdx.x] : 0.f;
    s_in[threadIdx.x] = in_w != nullptr ? in_w[threadIdx.x] : 1.f;
  }
  __syncthreads();
  const size_t r = blockIdx.x;
  float* xr = xs + r * streams * cols;
  float4 keep[SMV_KEEP];
  float ssq = 0.f;
#pragma unroll
  for (int it = 0; it < SMV_KEEP; ++it) {
    const int c = (threadIdx.x + it * ROW_THREADS) * 4;
    keep[it] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c >= cols) continue;
    float4 x[MAX_STREAMS];
#pragma unroll
    for (int s = 0; s < MAX_STREAMS; ++s)
      if (s < streams) x[s] = *reinterpret_cast<const float4*>(xr + static_cast<size_t>(s) * cols + c);
    float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
    if (y1 != nullptr) {
      float4 y = load4<T>(y1 + r * cols + c);
      y.x *= c1; y.y *= c1; y.z *= c1; y.w *= c1;
      if (y2 != nullptr) {
        const float4 z = load4<T>(y2 + r * cols + c);
        y.x += c2 * z.x; y.y += c2 * z.y; y.z += c2 * z.z; y.w += c2 * z.w;
      }
#pragma unroll
      for (int t = 0; t < MAX_STREAMS; ++t) {
        if (t < streams) {
          float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int s = 0; s < MAX_STREAMS; ++s) {
            if (s < streams) {
              const float m = s_mix[s * streams + t];
              acc.x += m * x[s].x; acc.y += m * x[s].y; acc.z += m * x[s].z; acc.w += m * x[s].w;
            }
          }
          const float ow = s_out[t], iw = s_in[t];
          acc.x += ow * y.x; acc.y += ow * y.y; acc.z += ow * y.z; acc.w += ow * y.w;
          *reinterpret_cast<float4*>(xr + static_cast<size_t>(t) * cols + c) = acc;
          u.x += iw * acc.x; u.y += iw * acc.y; u.z += iw * acc.z; u.w += iw * acc.w;
        }
      }
    } else {
#pragma unroll
      for (int t = 0; t < MAX_STREAMS; ++t) {
        if (t < streams) {
          const float iw = s_in[t];
          u.x += iw * x[t].x; u.y += iw * x[t].y; u.z += iw * x[t].z; u.w += iw * x[t].w;
        }
      }
    }
    keep[it] = u;
    ssq += u.x * u.x + u.y * u.y + u.z * u.z + u.w * u.w;
  }
  if (h == nullptr) return;
  const float tot = block_sum(ssq, red);
  const float inv = 1.0f / sqrtf(tot / static_cast<float>(cols) + eps);
  T* hr = h + r * cols;
#pragma unroll
  for (int it = 0; it < SMV_KEEP; ++it) {
    const int c = (threadIdx.x + it * ROW_THREADS) * 4;
    if (c >= cols) continue;
    const float4 w = *reinterpret_cast<const float4*>(norm_w + c);
    const float4 u = keep[it];
    store4<T>(hr + c, make_float4(u.x * inv * w.x, u.y * inv * w.y, u.z * inv * w.z, u.w * inv * w.w));
  }
}

// out[i] = rms_norm(sum_s in_w[s] x_s of row rows_idx[i]) * norm_w
template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
stream_gather_norm_kernel(const float* __restrict__ xs, const int32_t* __restrict__ rows_idx, const float* __restrict__ in_w,
                          const float* __restrict__ norm_w, T* __restrict__ out, int cols, int streams, float eps) {
  __shared__ float red[33];
  const size_t r = rows_idx != nullptr ? static_cast<size_t>(rows_idx[blockIdx.x]) : blockIdx.x;
  const float* xr = xs + r * streams * cols;
  float ssq = 0.f;
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    float u = 0.f;
    for (int t = 0; t < streams; ++t) u += (in_w != nullptr ? in_w[t] : 1.f) * xr[static_cast<size_t>(t) * cols + c];
    ssq += u * u;
  }
  const float tot = block_sum(ssq, red);
  const float inv = 1.0f / sqrtf(tot / static_cast<float>(cols) + eps);
  T* o = out + static_cast<size_t>(blockIdx.x) * cols;
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    float u = 0.f;
    for (int t = 0; t < streams; ++t) u += (in_w != nullptr ? in_w[t] : 1.f) * xr[static_cast<size_t>(t) * cols + c];
    o[c] = from_f<T>(u * inv * norm_w[c]);
  }
}

// ------------------------------------------------------------------ attention step preparation
// One block per token.  q = u[q_off : +H*d] + q_bias, k = u[k_off : +G*d] + k_bias, v = u[v_off : +G*dv] + v_bias, or,
// with v_off < 0, v = k as it stands here (before norm and rotation).  With norm weights, q and k are each divided by
// the root mean square of their WHOLE projection and multiplied by the weight.  With rot_dims > 0, coordinate
// i < rot_dims/2 of every head is paired with i + rot_dims/2 (or, `interleaved`, coordinate 2i with 2i + 1) and the pair
// turned by position * freq[i].  Without caches (a layer that reads another layer's keys and values) only q is made.
template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
attn_prep_kernel(const T* __restrict__ u, int64_t ldu, int q_off, int k_off, int v_off, const float* __restrict__ q_bias,
                 const float* __restrict__ k_bias, const float* __restrict__ v_bias, const float* __restrict__ q_norm_w,
                 const float* __restrict__ k_norm_w, const float* __restrict__ freq, int rot_dims,
                 const int32_t* __restrict__ positions, const int32_t* __restrict__ slot_mapping, T* __restrict__ q_out,
                 T* __restrict__ k_cache, T* __restrict__ v_cache, int H, int G, int Gv, int d, int dv, float eps, int interleaved) {
  __shared__ float red[33];
  const size_t t = blockIdx.x;
  const int slot = slot_mapping[t];
  if (slot < 0) return;                                   // padding row (uniform over the block)
  const T* ur = u + t * ldu;
  const int nq = H * d, nk = G * d, nv = Gv * dv;
  const float pos = static_cast<float>(positions[t]);
  // values
  T* vr = v_cache + static_cast<size_t>(slot) * nv;
  for (int c = threadIdx.x; c < nv && v_cache != nullptr; c += blockDim.x) {
    float v;
    if (v_off >= 0) v = to_f(ur[v_off + c]) + (v_bias != nullptr ? v_bias[c] : 0.f);
    else v = to_f(ur[k_off + c]) + (k_bias != nullptr ? k_bias[c] : 0.f);
    vr[c] = from_f<T>(v);
  }
  float inv_q = 1.f, inv_k = 1.f;
  if (q_norm_w != nullptr) {
    float sq = 0.f, sk = 0.f;
    for (int c = threadIdx.x; c < nq; c += blockDim.x) {
      const float v = to_f(ur[q_off + c]) + (q_bias != nullptr ? q_bias[c] : 0.f);
      sq += v * v;
    }
    for (int c = threadIdx.x; c < nk; c += blockDim.x) {
      const float v = to_f(ur[k_off + c]) + (k_bias != nullptr ? k_bias[c] : 0.f);
      sk += v * v;
    }
    inv_q = 1.0f / sqrtf(block_sum(sq, red) / static_cast<float>(nq) + eps);
    inv_k = 1.0f / sqrtf(block_sum(sk, red) / static_cast<float>(nk) + eps);
  }
  const int half = rot_dims / 2;
  // a work item is one coordinate that passes unchanged, or one pair of rotated coordinates (owned by its first half)
  for (int part = 0; part < (k_cache != nullptr ? 2 : 1); ++part) {
    const int n = part == 0 ? nq : nk, off = part == 0 ? q_off : k_off;
    const float* bias = part == 0 ? q_bias : k_bias;
    const float* nw = part == 0 ? q_norm_w : k_norm_w;
    const float inv = part == 0 ? inv_q : inv_k;
    T* dst = part == 0 ? q_out + t * nq : k_cache + static_cast<size_t>(slot) * nk;
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
      const int i = c % d;
      const bool rotated = i < rot_dims;
      if (rotated && (interleaved ? (i & 1) : i >= half)) continue;     // second of a pair: written by its partner
      float a = to_f(ur[off + c]) + (bias != nullptr ? bias[c] : 0.f);
      if (nw != nullptr) a = a * inv * nw[c];
      if (rotated) {
        const int c2 = interleaved ? c + 1 : c + half;
        float b = to_f(ur[off + c2]) + (bias != nullptr ? bias[c2] : 0.f);
        if (nw != nullptr) b = b * inv * nw[c2];
        float sn, cs;
        sincosf(pos * freq[interleaved ? i >> 1 : i], &sn, &cs);
        dst[c] = from_f<T>(a * cs - b * sn);
        dst[c2] = from_f<T>(b * cs + a * sn);
      } else {
        dst[c] = from_f<T>(a);
      }
    }
  }
}

// The preparation of heads that are normed ONE BY ONE: v' = N_head(v + bias) * w (w of `dim` numbers, shared by the heads), then
// the rotation by the step's table `rot` [n, rot_dims] (cosines, then sines).  Work items are (token run, head): heads 0 .. H-1
// are queries, then G key heads, then G value heads (bias and cache write only).
struct HeadPrepArgs {
  const void* u; int64_t ldu; int q_off, k_off, v_off;
  const float *q_bias, *k_bias, *v_bias, *q_norm_w, *k_norm_w;
  const float* rot; int rot_dims, interleaved;
  const int32_t* slot_mapping;
  void *q_out, *k_cache, *v_cache;
  int n_tokens, H, G, d, dv;
  float eps;
};

template <typename T>
struct HeadSlice {                                        // what a head reads and writes
  const T* src; const float* bias; const float* nw; T* dst;
  int64_t dst_row; int width; bool cached, qk;
  __device__ __forceinline__ HeadSlice(const HeadPrepArgs& p, int head) {
    const T* u = static_cast<const T*>(p.u);
    if (head < p.H) {
      src = u + p.q_off + head * p.d; bias = p.q_bias ? p.q_bias + head * p.d : nullptr; nw = p.q_norm_w;
      dst = static_cast<T*>(p.q_out) + head * p.d; dst_row = static_cast<int64_t>(p.H) * p.d; width = p.d; cached = false; qk = true;
    } else if (head < p.H + p.G) {
      const int g = head - p.H;
      src = u + p.k_off + g * p.d; bias = p.k_bias ? p.k_bias + g * p.d : nullptr; nw = p.k_norm_w;
      dst = static_cast<T*>(p.k_cache) + g * p.d; dst_row = static_cast<int64_t>(p.G) * p.d; width = p.d; cached = true; qk = true;
    } else {
      const int g = head - p.H - p.G;
      src = u + p.v_off + g * p.dv; bias = p.v_bias ? p.v_bias + g * p.dv : nullptr; nw = nullptr;
      dst = static_cast<T*>(p.v_cache) + g * p.dv; dst_row = static_cast<int64_t>(p.G) * p.dv; width = p.dv; cached = true; qk = false;
    }
  }
};

constexpr int HP_WARPS = 8;

// Any head size, either pairing: one warp per (token, head).
template <typename T>
__global__ void __launch_bounds__(HP_WARPS * 32)
head_prep_kernel(const HeadPrepArgs p) {
  const int heads = p.H + 2 * p.G, lane = threadIdx.x & 31;
  const int64_t item = static_cast<int64_t>(blockIdx.x) * HP_WARPS + (threadIdx.x >> 5);
  if (item >= static_cast<int64_t>(p.n_tokens) * heads) return;
  const size_t t = item / heads;
  const HeadSlice<T> s(p, static_cast<int>(item % heads));
  const int slot = p.slot_mapping[t];
  if (slot < 0) return;                                   // padding row
  const T* src = s.src + t * p.ldu;
  T* dst = s.dst + (s.cached ? static_cast<int64_t>(slot) : static_cast<int64_t>(t)) * s.dst_row;
  auto val = [&](int c) { return to_f(src[c]) + (s.bias != nullptr ? s.bias[c] : 0.f); };
  float inv = 1.f;
  if (s.nw != nullptr) {
    float ssq = 0.f;
    for (int c = lane; c < s.width; c += 32) { const float v = val(c); ssq += v * v; }
    inv = 1.0f / sqrtf(warp_sum(ssq) / static_cast<float>(s.width) + p.eps);
  }
  const int rd = s.qk ? p.rot_dims : 0, half = rd / 2;
  for (int c = lane; c < s.width; c += 32) {
    if (c < rd && (p.interleaved ? (c & 1) : c >= half)) continue;        // second of a pair: written with the first
    float a = val(c) * inv * (s.nw != nullptr ? s.nw[c] : 1.f);
    if (c < rd) {
      const int c2 = p.interleaved ? c + 1 : c + half, i = p.interleaved ? c >> 1 : c;
      const float b = val(c2) * inv * (s.nw != nullptr ? s.nw[c2] : 1.f);
      const float cs = p.rot[t * rd + i], sn = p.rot[t * rd + half + i];
      dst[c] = from_f<T>(a * cs - b * sn);
      dst[c2] = from_f<T>(b * cs + a * sn);
    } else {
      dst[c] = from_f<T>(a);
    }
  }
}

template <typename T> __device__ __forceinline__ void load4_f(const T* p, float* f);
template <> __device__ __forceinline__ void load4_f<float>(const float* p, float* f) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
}
template <> __device__ __forceinline__ void load4_f<__nv_bfloat16>(const __nv_bfloat16* p, float* f) {
  const uint2 r = ldg_v2(p);
  f[0] = bf16lo(r.x); f[1] = bf16hi(r.x); f[2] = bf16lo(r.y); f[3] = bf16hi(r.y);
}

// Pairs (2i, 2i + 1) or no rotation, sizes and offsets multiples of 4: LPH lanes share a head, four neighbouring coordinates
// (two whole pairs) per lane and chunk, so 32 / LPH heads run in a warp and nothing but the sum of squares crosses lanes.  A lane
// group walks TOK tokens of its head with bias and norm weight in registers; the rows of all TOK tokens are asked for first.
template <typename T, int LPH, int NCH, int TOK>
__global__ void __launch_bounds__(HP_WARPS * 32)
head_prep_vec4_kernel(const HeadPrepArgs p) {
  const int heads = p.H + 2 * p.G, sub = threadIdx.x % LPH;
  const int64_t item = (static_cast<int64_t>(blockIdx.x) * (HP_WARPS * 32) + threadIdx.x) / LPH;
  const int64_t n_items = static_cast<int64_t>((p.n_tokens + TOK - 1) / TOK) * heads;
  const bool live = item < n_items;                       // every lane stays for the shuffles
  const int t0 = live ? static_cast<int>(item / heads) * TOK : 0;
  const HeadSlice<T> s(p, live ? static_cast<int>(item % heads) : 0);
  const int rd = s.qk ? p.rot_dims : 0;
  float x[TOK][NCH][4], bias[NCH][4], w[NCH][4];
  int slot[TOK];
#pragma unroll
  for (int t = 0; t < TOK; ++t) slot[t] = live && t0 + t < p.n_tokens ? p.slot_mapping[t0 + t] : -1;
#pragma unroll
  for (int k = 0; k < NCH; ++k) {
    const int c = (k * LPH + sub) * 4;
#pragma unroll
    for (int e = 0; e < 4; ++e) { bias[k][e] = 0.f; w[k][e] = 1.f; }
#pragma unroll
    for (int t = 0; t < TOK; ++t) {
#pragma unroll
      for (int e = 0; e < 4; ++e) x[t][k][e] = 0.f;
      if (c < s.width && slot[t] >= 0) load4_f<T>(s.src + static_cast<int64_t>(t0 + t) * p.ldu + c, x[t][k]);
    }
    if (c < s.width) {
      if (s.bias != nullptr) load4_f<float>(s.bias + c, bias[k]);
      if (s.nw != nullptr) load4_f<float>(s.nw + c, w[k]);
    }
  }
#pragma unroll
  for (int t = 0; t < TOK; ++t) {
    float ssq = 0.f;
#pragma unroll
    for (int k = 0; k < NCH; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e) { x[t][k][e] += bias[k][e]; ssq += x[t][k][e] * x[t][k][e]; }
#pragma unroll
    for (int o = LPH / 2; o > 0; o >>= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, o);
    if (slot[t] < 0) continue;
    const float inv = s.nw != nullptr ? 1.0f / sqrtf(ssq / static_cast<float>(s.width) + p.eps) : 1.f;
    T* dst = s.dst + (s.cached ? static_cast<int64_t>(slot[t]) : static_cast<int64_t>(t0 + t)) * s.dst_row;
    const float* rot = p.rot + static_cast<int64_t>(t0 + t) * rd;
#pragma unroll
    for (int k = 0; k < NCH; ++k) {
      const int c = (k * LPH + sub) * 4;
      if (c >= s.width) continue;
      float v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = x[t][k][e] * inv * w[k][e];
      if (c < rd) {                                       // rot_dims is a multiple of 4: both pairs turn, or neither
        const float2 cs = *reinterpret_cast<const float2*>(rot + c / 2), sn = *reinterpret_cast<const float2*>(rot + rd / 2 + c / 2);
        const float a0 = v[0], a1 = v[2];
        v[0] = a0 * cs.x - v[1] * sn.x; v[1] = v[1] * cs.x + a0 * sn.x;
        v[2] = a1 * cs.y - v[3] * sn.y; v[3] = v[3] * cs.y + a1 * sn.y;
      }
      if constexpr (sizeof(T) == 4) *reinterpret_cast<float4*>(dst + c) = make_float4(v[0], v[1], v[2], v[3]);
      else stg_v2(dst + c, make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3])));
    }
  }
}

template <typename T>
static void launch_head_prep(const HeadPrepArgs& p, cudaStream_t st) {
  const int heads = p.H + 2 * p.G, wide = std::max(p.d, p.dv);
  const bool vec = p.d % 4 == 0 && p.dv % 4 == 0 && p.ldu % 4 == 0 && p.q_off % 4 == 0 && p.k_off % 4 == 0 && p.v_off % 4 == 0 &&
                   wide <= 256 && (p.rot_dims == 0 || (p.interleaved && p.rot_dims % 4 == 0 && aligned16(p.rot))) && aligned16(p.u) &&
                   aligned16(p.q_out) && aligned16(p.k_cache) && aligned16(p.v_cache) && (!p.q_bias || aligned16(p.q_bias)) &&
                   (!p.k_bias || aligned16(p.k_bias)) && (!p.v_bias || aligned16(p.v_bias)) && (!p.q_norm_w || aligned16(p.q_norm_w)) &&
                   (!p.k_norm_w || aligned16(p.k_norm_w));
  if (!vec) {
    const int64_t items = static_cast<int64_t>(p.n_tokens) * heads;
    head_prep_kernel<T><<<static_cast<unsigned>((items + HP_WARPS - 1) / HP_WARPS), HP_WARPS * 32, 0, st>>>(p);
    return;
  }
  const bool many = static_cast<int64_t>(p.n_tokens) * heads > static_cast<int64_t>(sm_count()) * 256;
#define HP_GO_T(LPH, NCH, TOK) do { \
    const int64_t threads = static_cast<int64_t>((p.n_tokens + TOK - 1) / TOK) * heads * LPH; \
    head_prep_vec4_kernel<T, LPH, NCH, TOK><<<static_cast<unsigned>((threads + HP_WARPS * 32 - 1) / (HP_WARPS * 32)), HP_WARPS * 32, 0, st>>>(p); } while (0)
#define HP_GO(LPH, NCH) do { if (many) HP_GO_T(LPH, NCH, 4); else HP_GO_T(LPH, NCH, 1); } while (0)
  if (wide <= 32) HP_GO(8, 1);
  else if (wide <= 64) HP_GO(16, 1);
  else if (wide <= 128) HP_GO(32, 1);
  else HP_GO(32, 2);
#undef HP_GO
#undef HP_GO_T
}

// Both preparations for bf16 rows in 16-byte pieces: a CTA takes TOK tokens, forms (or copies) their angles once for all heads, and a thread
// takes eight coordinates of one head of all of them, with bias and norm weight in registers and the TOK pieces asked for before the first
// is used.  d / 8 neighbouring lanes hold a head: they sum its squares, and hand each other the partners i, i + rot_dims / 2.
// Bound: HBM (u read, queries and cache rows written once) where nothing is normed, issue and latency of the norms else.  16 + 8 + 8 heads of
// 128, 8192 tokens (20 us at the copy rate), kernels above / this one in us: plain 93 / 31, 64 coordinates turned 116 / 37, whole norms and
// turns 131 / 74, head norms and a table 65 / 45 (pairs) and 122 / 58 (halves); 64 tokens 6.9 / 2.5, 9.1 / 3.0, 12.9 / 5.4.  One number a
// thread and step, and angles formed again for every head, were what the first three cost.  Two tokens a CTA: four take 124 registers
// and are slower where norms are formed (head norms 51, whole norms 106 us), as fast where not.
struct PrepArgs {
  const __nv_bfloat16* u; int64_t ldu; int q_off, k_off, v_off;              // v_off < 0: the values are the keys before norm and rotation
  const float *q_bias, *k_bias, *v_bias, *q_norm_w, *k_norm_w;
  int norm;                                                                  // 0: none, 1: over the whole projection, 2: head by head
  const float *rot, *freq; const int32_t* positions; int rot_dims, interleaved;   // a table [n, rot_dims] or frequencies
  const int32_t* slot_mapping;
  __nv_bfloat16 *q_out, *k_cache, *v_cache;
  int n_tokens, H, G, Gv, d, dv;
  float eps;
};
constexpr int PREP_MAX_ROT = 512;

__device__ __forceinline__ void unpack8(const uint4& x, float* f) {
  f[0] = bf16lo(x.x); f[1] = bf16hi(x.x); f[2] = bf16lo(x.y); f[3] = bf16hi(x.y);
  f[4] = bf16lo(x.z); f[5] = bf16hi(x.z); f[6] = bf16lo(x.w); f[7] = bf16hi(x.w);
}
__device__ __forceinline__ void load8_f(const float* p, float* f) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

// From a head's sums of squares of two tokens to the reciprocals of its roots (1 where !normed).  The first exchange leaves each half of the head's lanes with one
// of the tokens: one tree and one root for both, in the order of a tree for each.
template <int LPH>
__device__ __forceinline__ void both_inverses(float (&inv)[2], int lane, bool normed, float eps) {
  const bool second = lane & (LPH / 2);
  float v = second ? inv[1] : inv[0];
  v += __shfl_xor_sync(0xffffffffu, second ? inv[0] : inv[1], LPH / 2);
#pragma unroll
  for (int o = LPH / 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  v = normed ? 1.0f / sqrtf(v / static_cast<float>(LPH * 8) + eps) : 1.f;
  inv[0] = __shfl_sync(0xffffffffu, v, lane & ~(LPH / 2));
  inv[1] = __shfl_sync(0xffffffffu, v, lane | (LPH / 2));
}
__device__ __forceinline__ void turn_pair(float& a, float& b, float co, float si) {
  const float first = a;
  a = first * co - b * si;
  b = b * co + first * si;
}

template <int TOK, int LPH>
__global__ void __launch_bounds__(ROW_THREADS)
prep_vec8_kernel(const PrepArgs p) {
  extern __shared__ __align__(16) float2 turn[];                        // [TOK][rot_dims / 2]: cosine, sine
  __shared__ float red[33], inv_s[2][TOK];
  const int t0 = blockIdx.x * TOK, tid = threadIdx.x, half = p.rot_dims / 2;
  const int nq = p.H * p.d, nk = p.G * p.d, nv = p.Gv * p.dv;
  int slot[TOK];
#pragma unroll
  for (int t = 0; t < TOK; ++t) slot[t] = t0 + t < p.n_tokens ? p.slot_mapping[t0 + t] : -1;      // -1: padding row, or behind the last token
  const int q8 = nq / 8, k8 = p.k_cache != nullptr ? nk / 8 : 0, v8 = p.v_cache != nullptr ? nv / 8 : 0, items = q8 + k8 + v8;
  const int lane = tid & 31;                              // LPH lanes have a head
  constexpr int DIM = LPH * 8;
  static_assert(TOK <= 2, "one exchange shares out the tokens");
  uint4 x[TOK], ahead[TOK];                               // a thread's pieces, and those of its next turn
  auto load = [&](int i) {
    const bool is_q = i < q8, is_k = !is_q && i < q8 + k8;
    const int c = (is_q ? i : is_k ? i - q8 : i - q8 - k8) * 8, off = is_q ? p.q_off : is_k || p.v_off < 0 ? p.k_off : p.v_off;
#pragma unroll
    for (int t = 0; t < TOK; ++t) {
      ahead[t] = make_uint4(0u, 0u, 0u, 0u);
      if (i < items && t0 + t < p.n_tokens) ahead[t] = ldg_v4(p.u + static_cast<int64_t>(t0 + t) * p.ldu + off + c);   // a padding row too: its slot is not waited for
    }
  };
  load(tid);
  for (int i = tid; i < TOK * half; i += ROW_THREADS) {
    const int t = i / half, c = i - t * half;
    if (t0 + t >= p.n_tokens) break;
    float2 cs;
    if (p.rot != nullptr) {
      const float* row = p.rot + static_cast<int64_t>(t0 + t) * p.rot_dims;
      cs = make_float2(row[c], row[half + c]);
    } else {
      sincosf(static_cast<float>(p.positions[t0 + t]) * p.freq[c], &cs.y, &cs.x);
    }
    turn[i] = cs;
  }
  if (p.norm == 1) {
    for (int t = 0; t < TOK; ++t) {
      if (slot[t] < 0) continue;                          // uniform over the block
      const __nv_bfloat16* ur = p.u + static_cast<int64_t>(t0 + t) * p.ldu;
      for (int side = 0; side < 2; ++side) {
        const int n = side ? nk : nq;
        const float* bias = side ? p.k_bias : p.q_bias;
        float ss = 0.f;
        for (int c = tid * 8; c < n; c += ROW_THREADS * 8) {
          float f[8], b[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
          unpack8(ldg_v4(ur + (side ? p.k_off : p.q_off) + c), f);
          if (bias != nullptr) load8_f(bias + c, b);
#pragma unroll
          for (int e = 0; e < 8; ++e) { const float v = f[e] + b[e]; ss += v * v; }
        }
        const float sum = block_sum(ss, red);
        if (tid == 0) inv_s[side][t] = 1.0f / sqrtf(sum / static_cast<float>(n) + p.eps);
      }
    }
  }
  __syncthreads();
  for (int base = tid & ~31; base < items; base += ROW_THREADS) {              // a warp stays together for the shuffles
    const int i = base + lane;
    const bool live = i < items, is_q = i < q8, is_k = !is_q && i < q8 + k8;
    const int c = (is_q ? i : is_k ? i - q8 : i - q8 - k8) * 8;
    const float* bias = is_q ? p.q_bias : is_k || p.v_off < 0 ? p.k_bias : p.v_bias;
#pragma unroll
    for (int t = 0; t < TOK; ++t) x[t] = ahead[t];
    load(i + ROW_THREADS);
    float b[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, w[8] = {1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f};
    if (live && bias != nullptr) load8_f(bias + c, b);
    const bool qk = live && (is_q || is_k);
    const int ci = qk ? c & (DIM - 1) : DIM;              // the piece's first coordinate in its head
    if (qk && p.norm != 0) load8_f((is_q ? p.q_norm_w : p.k_norm_w) + (p.norm == 2 ? ci : c), w);
    const bool turned = qk && ci < p.rot_dims;
    uint64_t y[TOK][4];
#pragma unroll
    for (int t = 0; t < TOK; ++t) {
      const uint32_t word[4] = {x[t].x, x[t].y, x[t].z, x[t].w};
#pragma unroll
      for (int h = 0; h < 4; ++h) y[t][h] = f2_add(f2_pack(bf16lo(word[h]), bf16hi(word[h])), f2_pack(b[2 * h], b[2 * h + 1]));
    }
    float inv[TOK];
#pragma unroll
    for (int t = 0; t < TOK; ++t) inv[t] = 1.f;
    if (p.norm == 2) {
#pragma unroll
      for (int t = 0; t < TOK; ++t) {
        inv[t] = 0.f;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          float lo, hi;
          f2_unpack(y[t][h], lo, hi);
          inv[t] += lo * lo;
          inv[t] += hi * hi;
        }
      }
      if constexpr (TOK == 2) {
        both_inverses<LPH>(inv, lane, qk, p.eps);
      } else {
#pragma unroll
        for (int o = LPH / 2; o > 0; o >>= 1) inv[0] += __shfl_xor_sync(0xffffffffu, inv[0], o);
        inv[0] = qk ? 1.0f / sqrtf(inv[0] / static_cast<float>(DIM) + p.eps) : 1.f;
      }
    } else if (p.norm == 1 && qk) {
#pragma unroll
      for (int t = 0; t < TOK; ++t) inv[t] = inv_s[is_k][t];
    }
#pragma unroll
    for (int t = 0; t < TOK; ++t) {
      float f[8];
#pragma unroll
      for (int h = 0; h < 4; ++h)
        f2_unpack(f2_mul(f2_mul(y[t][h], f2_pack(inv[t], inv[t])), f2_pack(w[2 * h], w[2 * h + 1])), f[2 * h], f[2 * h + 1]);
      if (p.rot_dims > 0 && p.interleaved) {
        if (turned) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float4 cs = reinterpret_cast<const float4*>(turn + t * half + ci / 2)[e];
            turn_pair(f[4 * e], f[4 * e + 1], cs.x, cs.y);
            turn_pair(f[4 * e + 2], f[4 * e + 3], cs.z, cs.w);
          }
        }
      } else if (p.rot_dims > 0) {
        const bool second = ci >= half;
        const int from = turned ? lane + (second ? -half / 8 : half / 8) : lane;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float other = __shfl_sync(0xffffffffu, f[e], from);
          if (turned) {
            const float2 cs = turn[t * half + (second ? ci - half : ci) + e];
            const float x1 = second ? other : f[e], x2 = second ? f[e] * cs.x : -(other * cs.y);
            f[e] = fmaf(x1, second ? cs.y : cs.x, x2);   // the product of the head's first half joins the sum unrounded
          }
        }
      }
      if (live && slot[t] >= 0) {
        __nv_bfloat16* dst = is_q ? p.q_out + static_cast<int64_t>(t0 + t) * nq : is_k ? p.k_cache + static_cast<int64_t>(slot[t]) * nk
                                                                                       : p.v_cache + static_cast<int64_t>(slot[t]) * nv;
        stg_v4(dst + c, make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7])));
      }
    }
  }
}

// The same for many tokens where heads are normed one by one or not at all (one pass over a row): a thread keeps its piece of the row - bias, norm weights, source and
// destination - and walks WALK consecutive tokens two at a time, with the pieces of the next four on their way and the angles of all WALK in shared memory.  Above,
// every two tokens paid for their own indexes, weights, angles and barrier.
// Bound: HBM where nothing is turned, the turns' instructions beside it else.  16 + 8 + 8 heads of 128, 8192 / 4856 ragged tokens in us, above / this one: plain
// 31.5 / 24.5 and 18.0 / 11.4, 64 coordinates turned by frequencies 37.4 / 28.2 and 20.8 / 14.5, head norms 37.4 / 25.5 and 22.1 / 13.8, head norms and a table
// 45.1 / 31.4 and 26.0 / 17.5 (pairs), 57.8 / 39.0 and 34.3 / 22.3 (halves; 38.0 and 22.0 where each coordinate's own
// product joins the sum unrounded, which gives other bits than above).  Angles read from the table by every thread 52 us, cosines beside sines in shared memory 32
// and 51; WALK of 4 30.8 and 18.5, of 16 31.2 and 19.4; two pieces on their way 32.2 and 19.3.  Fewer than 8 tokens a multiprocessor stay above, a token a CTA.
constexpr int WALK = 8, AHEAD = 4;

template <int LPH, bool PAIRS>
__global__ void __launch_bounds__(ROW_THREADS, 3)
prep_walk_kernel(const PrepArgs p) {
  extern __shared__ __align__(16) float turns[];          // [WALK][rot_dims]: the tokens' rows of the table, cosines and then sines
  constexpr int DIM = LPH * 8;
  const int nq = p.H * p.d, nk = p.G * p.d, nv = p.Gv * p.dv, half = p.rot_dims / 2;
  const int q8 = nq / 8, k8 = p.k_cache != nullptr ? nk / 8 : 0, v8 = p.v_cache != nullptr ? nv / 8 : 0, items = q8 + k8 + v8;
  const int i = blockIdx.y * ROW_THREADS + threadIdx.x, lane = threadIdx.x & 31;
  const bool live = i < items, is_q = i < q8, is_k = !is_q && i < q8 + k8, qk = live && (is_q || is_k);
  const int c = live ? (is_q ? i : is_k ? i - q8 : i - q8 - k8) * 8 : 0;
  const __nv_bfloat16* src = p.u + (is_q ? p.q_off : is_k || p.v_off < 0 ? p.k_off : p.v_off) + c;
  __nv_bfloat16* dst = (is_q ? p.q_out : is_k ? p.k_cache : p.v_cache) + c;
  const int64_t dst_row = is_q ? nq : is_k ? nk : nv;
  const int t0 = blockIdx.x * WALK, cnt = min(WALK, p.n_tokens - t0);
  uint4 x[WALK];
  int slot[WALK];                                         // -1: padding row, or behind the last token
  auto load = [&](int t) {
    x[t] = make_uint4(0u, 0u, 0u, 0u);
    slot[t] = -1;
    if (live && t < cnt) {
      x[t] = ldg_v4(src + static_cast<int64_t>(t0 + t) * p.ldu);
      slot[t] = p.slot_mapping[t0 + t];
    }
  };
#pragma unroll
  for (int t = 0; t < AHEAD; ++t) load(t);
  if (p.rot != nullptr) {
    for (int a = threadIdx.x * 4; a < cnt * p.rot_dims; a += ROW_THREADS * 4)
      *reinterpret_cast<float4*>(turns + a) = *reinterpret_cast<const float4*>(p.rot + static_cast<int64_t>(t0) * p.rot_dims + a);
  } else {
    for (int a = threadIdx.x; a < cnt * half; a += ROW_THREADS) {
      const int t = a / half, k = a - t * half;
      float* row = turns + t * p.rot_dims;
      sincosf(static_cast<float>(p.positions[t0 + t]) * p.freq[k], row + half + k, row + k);
    }
  }
  const float* bias = is_q ? p.q_bias : is_k || p.v_off < 0 ? p.k_bias : p.v_bias;
  float b[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, w[8] = {1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f};
  if (live && bias != nullptr) load8_f(bias + c, b);
  const int ci = qk ? c & (DIM - 1) : DIM;                // the piece's first coordinate in its head
  if (qk && p.norm != 0) load8_f((is_q ? p.q_norm_w : p.k_norm_w) + ci, w);
  const bool turned = qk && ci < p.rot_dims, second = !PAIRS && ci >= half;
  const int angle = PAIRS ? ci / 2 : second ? ci - half : ci;      // the first angle of the piece
  if (p.rot_dims > 0) __syncthreads();
  if ((i & ~31) >= items) return;                         // a warp stays together for the shuffles
  const int from = !turned ? lane : second ? lane - half / 8 : lane + half / 8;
#pragma unroll
  for (int t = 0; t < WALK; t += 2) {
    if (t >= cnt) break;
#pragma unroll
    for (int k = AHEAD; k < AHEAD + 2; ++k) if (t + k < WALK) load(t + k);
    uint64_t y[2][4];
    float inv[2] = {1.f, 1.f};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint32_t word[4] = {x[t + k].x, x[t + k].y, x[t + k].z, x[t + k].w};
#pragma unroll
      for (int h = 0; h < 4; ++h) y[k][h] = f2_add(f2_pack(bf16lo(word[h]), bf16hi(word[h])), f2_pack(b[2 * h], b[2 * h + 1]));
    }
    if (p.norm == 2) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        inv[k] = 0.f;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          float lo, hi;
          f2_unpack(y[k][h], lo, hi);
          inv[k] += lo * lo;
          inv[k] += hi * hi;
        }
      }
      both_inverses<LPH>(inv, lane, qk, p.eps);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int row = t0 + t + k;
      float f[8];
#pragma unroll
      for (int h = 0; h < 4; ++h)
        f2_unpack(f2_mul(f2_mul(y[k][h], f2_pack(inv[k], inv[k])), f2_pack(w[2 * h], w[2 * h + 1])), f[2 * h], f[2 * h + 1]);
      if (p.rot_dims > 0) {
        const float* cs = turns + (t + k) * p.rot_dims + angle;
        if constexpr (PAIRS) {
          if (turned) {
            const float4 co = *reinterpret_cast<const float4*>(cs), si = *reinterpret_cast<const float4*>(cs + half);
            turn_pair(f[0], f[1], co.x, si.x);
            turn_pair(f[2], f[3], co.y, si.y);
            turn_pair(f[4], f[5], co.z, si.z);
            turn_pair(f[6], f[7], co.w, si.w);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 8; e += 4) {
            float a1[4] = {1.f, 1.f, 1.f, 1.f}, a2[4] = {0.f, 0.f, 0.f, 0.f}, other[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) other[m] = __shfl_sync(0xffffffffu, f[e + m], from);
            if (turned) {
              load4_f<float>(cs + (second ? half : 0) + e, a1);
              load4_f<float>(cs + (second ? 0 : half) + e, a2);
#pragma unroll
              for (int m = 0; m < 4; ++m) {              // as above, with the cosines and sines of a second half changed over
                const float x1 = second ? other[m] : f[e + m], x2 = (second ? f[e + m] : -other[m]) * a2[m];
                f[e + m] = fmaf(x1, a1[m], x2);
              }
            }
          }
        }
      }
      if (slot[t + k] >= 0)
        stg_v4(dst + (is_q ? row : slot[t + k]) * dst_row, make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7])));
    }
  }
}

// Whole 16-byte pieces everywhere, and a head's lanes a power of two, so that heads never straddle warps; the kernels above take the rest.
static bool prep_vec8_applies(const PrepArgs& p) {
  const int lanes = p.d / 8;
  auto ok = [](const void* x) { return x == nullptr || aligned16(x); };
  return p.d % 8 == 0 && (lanes == 4 || lanes == 8 || lanes == 16 || lanes == 32) && p.dv % 8 == 0 && p.ldu % 8 == 0 && p.q_off % 8 == 0 && p.k_off % 8 == 0 &&
         (p.v_off < 0 || p.v_off % 8 == 0) && p.rot_dims % 8 == 0 && (p.interleaved || p.rot_dims % 16 == 0) && p.rot_dims <= PREP_MAX_ROT &&
         // few tokens with head norms: a warp per head has more of them in flight (64 tokens 2.8 / 3.5 us, 300 tokens 4.4 / 4.3)
         (p.norm != 2 || p.n_tokens >= 2 * sm_count()) &&
         ok(p.u) && ok(p.q_bias) && ok(p.k_bias) && ok(p.v_bias) && ok(p.q_norm_w) && ok(p.k_norm_w) && ok(p.q_out) && ok(p.k_cache) && ok(p.v_cache);
}

template <int LPH>
static void go_prep_vec8(const PrepArgs& p, cudaStream_t st) {
  const size_t turn = static_cast<size_t>(p.rot_dims / 2) * sizeof(float2);
  if (p.n_tokens >= 8 * sm_count() && p.norm != 1 && aligned16(p.rot)) {
    const int items = (p.H * p.d + (p.k_cache != nullptr ? p.G * p.d : 0) + (p.v_cache != nullptr ? p.Gv * p.dv : 0)) / 8;
    const dim3 grid((p.n_tokens + WALK - 1) / WALK, (items + ROW_THREADS - 1) / ROW_THREADS);
    if (p.interleaved) prep_walk_kernel<LPH, true><<<grid, ROW_THREADS, WALK * turn, st>>>(p);
    else prep_walk_kernel<LPH, false><<<grid, ROW_THREADS, WALK * turn, st>>>(p);
    return;
  }
  if (p.n_tokens >= 8 * sm_count()) prep_vec8_kernel<2, LPH><<<(p.n_tokens + 1) / 2, ROW_THREADS, 2 * turn, st>>>(p);
  else prep_vec8_kernel<1, LPH><<<p.n_tokens, ROW_THREADS, turn, st>>>(p);
}
static void launch_prep_vec8(const PrepArgs& p, cudaStream_t st) {
  switch (p.d / 8) {
    case 4: return go_prep_vec8<4>(p, st);
    case 8: return go_prep_vec8<8>(p, st);
    case 16: return go_prep_vec8<16>(p, st);
    default: return go_prep_vec8<32>(p, st);
  }
}

// ------------------------------------------------------------------ short causal convolution + activation
// y[t, c] = act(bias[c] + sum_j w[c, j] * u(position(t) - taps + 1 + j)[c]) over the C columns of u from c_off on.  An
// earlier position comes from this step's rows when it lies in the step's portion, from the sequence's carried state
// (its last taps - 1 rows, oldest first) when it came before, and is zero before the sequence's start.
constexpr int CONV_MAX_TAPS = 8;

template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
short_conv_act_kernel(const T* __restrict__ u, int64_t ldu, const float* __restrict__ w, const float* __restrict__ bias,
                      const T* __restrict__ state, const int32_t* __restrict__ tok_seq, const int32_t* __restrict__ positions,
                      const int32_t* __restrict__ seq_start, const int32_t* __restrict__ seq_pos0,
                      const int32_t* __restrict__ seq_len, const int32_t* __restrict__ seq_slot, T* __restrict__ out,
                      int64_t ldo, int C, int taps, int act) {
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  const size_t t = blockIdx.x;
  if (c >= C) return;
  const int b = tok_seq[t];
  if (seq_len[b] <= 0) return;                            // padding row
  const int p = positions[t], pos0 = seq_pos0[b], start = seq_start[b], R = taps - 1;
  const T* st = state + static_cast<size_t>(seq_slot[b]) * R * C;
  float acc = bias != nullptr ? bias[c] : 0.f;
#pragma unroll
  for (int j = 0; j < CONV_MAX_TAPS; ++j) {
    if (j < taps) {
      const int pj = p - R + j;
      float v = 0.f;
      if (pj >= pos0) v = to_f(u[static_cast<int64_t>(start + pj - pos0) * ldu + c]);
      else if (pj >= 0) v = to_f(st[static_cast<size_t>(pj - (pos0 - R)) * C + c]);   // entry r holds position pos0 - R + r
      acc += w[c * taps + j] * v;
    }
  }
  if (act == 1) acc = silu_f(acc);
  out[t * ldo + c] = from_f<T>(acc);
}

// The same convolution for TAPS known at compile time: a thread owns four consecutive channels and walks CONV_RUN consecutive tokens of one
// sequence with its filters in registers, so that every row is read once (channels and row strides multiples of 16 bytes; u, state, out 16-byte
// aligned).
// What bounds it is the instructions of its elements (25 of them, 17 for the activation) while enough warps are there to hide the rows' way: every row
// of the run is asked for before the first is used and kept as it lies in memory, products are formed two at a time.
// 4 x 2048 tokens of 4352 channels with the state's advance: 60 -> 47 us (eight channels a thread, 127 registers and half of the issue slots empty, before), 300 tokens
// 8.7 -> 7.3; runs of 4 tokens 52 and 7.0, of 16 47 and 7.9.
constexpr int CONV_RUN = 8;

template <typename T, int TAPS>
__global__ void __launch_bounds__(128)
short_conv_act_run_kernel(const T* __restrict__ u, int64_t ldu, const float* __restrict__ w, const float* __restrict__ bias,
                          const T* __restrict__ state, const int32_t* __restrict__ seq_start, const int32_t* __restrict__ seq_pos0,
                          const int32_t* __restrict__ seq_len, const int32_t* __restrict__ seq_slot, T* __restrict__ out,
                          int64_t ldo, int C, int act) {
  using Q = Quad<T>;
  constexpr int R = TAPS - 1;
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
  const int b = blockIdx.z, t0 = blockIdx.x * CONV_RUN;
  const int len = seq_len[b], pos0 = seq_pos0[b], start = seq_start[b], slot = seq_slot[b];
  if (c >= C || t0 >= len) return;
  const int cnt = min(CONV_RUN, len - t0);
  const T* rows = u + static_cast<int64_t>(start + t0) * ldu + c;
  typename Q::Raw raw[CONV_RUN + R];                       // raw[j]: the row of token t0 - R + j
#pragma unroll
  for (int i = 0; i < CONV_RUN; ++i) raw[R + i] = i < cnt ? Q::load(rows + i * ldu) : Q::zero();
#pragma unroll
  for (int j = 0; j < R; ++j) {                            // the rows before the run's first token
    const int pj = pos0 + t0 - R + j;
    raw[j] = Q::zero();
    if (pj >= pos0) raw[j] = Q::load(rows - static_cast<int64_t>(R - j) * ldu);
    else if (pj >= 0) raw[j] = Q::load(state + (static_cast<size_t>(slot) * R + (pj - (pos0 - R))) * C + c);
  }
  float flat[4 * TAPS], bs[4];                             // the filters of four channels lie one behind another
  const float* wc = w + static_cast<size_t>(c) * TAPS;
  if ((reinterpret_cast<uintptr_t>(w) & 15) == 0) {
#pragma unroll
    for (int i = 0; i < 4 * TAPS; i += 4) *reinterpret_cast<float4*>(flat + i) = __ldg(reinterpret_cast<const float4*>(wc + i));
  } else {
#pragma unroll
    for (int i = 0; i < 4 * TAPS; ++i) flat[i] = wc[i];
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) bs[e] = bias != nullptr ? bias[c + e] : 0.f;
  uint64_t wt[TAPS][2], first[2] = {f2_pack(bs[0], bs[1]), f2_pack(bs[2], bs[3])}, win[TAPS][2];
#pragma unroll
  for (int j = 0; j < TAPS; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) wt[j][h] = f2_pack(flat[2 * h * TAPS + j], flat[(2 * h + 1) * TAPS + j]);
#pragma unroll
  for (int j = 0; j < R; ++j) Q::pairs(raw[j], win[j]);
  T* o = out + static_cast<int64_t>(start + t0) * ldo + c;
#pragma unroll
  for (int i = 0; i < CONV_RUN; ++i) {
    if (i >= cnt) break;
    Q::pairs(raw[R + i], win[R]);
    float acc[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint64_t a = first[h];
#pragma unroll
      for (int j = 0; j < TAPS; ++j) a = f2_fma(wt[j][h], win[j][h], a);
      f2_unpack(a, acc[2 * h], acc[2 * h + 1]);
    }
    if (act == 1) {
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] = silu_for<T>(acc[e]);
    }
    store4<T>(o + i * ldo, make_float4(acc[0], acc[1], acc[2], acc[3]));
#pragma unroll
    for (int j = 0; j < R; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) win[j][h] = win[j + 1][h];
  }
}

// The carried state after the step: entry r holds the row of position end - R + r (end = pos0 + new tokens).  One thread
// per (sequence, column) reads its old entries before it writes any, so the shift is safe in place.
template <typename T>
__global__ void conv_state_advance_kernel(const T* __restrict__ u, int64_t ldu, T* __restrict__ state,
                                          const int32_t* __restrict__ seq_start, const int32_t* __restrict__ seq_pos0,
                                          const int32_t* __restrict__ seq_len, const int32_t* __restrict__ seq_slot, int C,
                                          int taps) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (c >= C) return;
  const int len = seq_len[b];
  if (len <= 0) return;
  const int R = taps - 1, pos0 = seq_pos0[b], start = seq_start[b];
  T* st = state + static_cast<size_t>(seq_slot[b]) * R * C + c;
  T old[CONV_MAX_TAPS];
#pragma unroll
  for (int r = 0; r < CONV_MAX_TAPS; ++r) if (r < R) old[r] = st[static_cast<size_t>(r) * C];
  const int end = pos0 + len;
#pragma unroll
  for (int r = 0; r < CONV_MAX_TAPS; ++r) {
    if (r < R) {
      const int pj = end - R + r;
      T v = from_f<T>(0.f);
      if (pj >= pos0) v = u[static_cast<int64_t>(start + pj - pos0) * ldu + c];
      else if (pj >= 0 && pj - (pos0 - R) >= 0) v = old[pj - (pos0 - R)];
      st[static_cast<size_t>(r) * C] = v;
    }
  }
}

// ------------------------------------------------------------------ gate + grouped RMS norm on a branch output
// One block per (row, group): the row y [cols] (float) is cut into `groups` equal consecutive parts; each part is divided
// by its own root mean square and multiplied by w[c mod w_len] (w null: by one); the gate act(gate[r, c]) multiplies y before the norm
// (gate_first) or the normed result.  act 0: sigmoid, 1: SiLU.
template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
gated_group_norm_kernel(const float* __restrict__ y, const T* __restrict__ gate, int64_t ldg, const float* __restrict__ w,
                        int w_len, int groups, int act, int gate_first, float eps, T* __restrict__ out, int cols) {
  __shared__ float red[33];
  const size_t r = blockIdx.x;
  const int gs = cols / groups, c0 = blockIdx.y * gs;
  const float* yr = y + r * cols + c0;
  const T* gr = gate != nullptr ? gate + r * ldg + c0 : nullptr;
  float ssq = 0.f;
  for (int c = threadIdx.x; c < gs; c += blockDim.x) {
    float v = yr[c];
    if (gr != nullptr && gate_first) {
      const float g = to_f(gr[c]);
      v *= act == 0 ? sigmoid_f(g) : silu_f(g);
    }
    ssq += v * v;
  }
  const float inv = 1.0f / sqrtf(block_sum(ssq, red) / static_cast<float>(gs) + eps);
  T* o = out + r * cols + c0;
  for (int c = threadIdx.x; c < gs; c += blockDim.x) {
    float v = yr[c];
    float g = 1.f;
    if (gr != nullptr) {
      g = to_f(gr[c]);
      g = act == 0 ? sigmoid_f(g) : silu_f(g);
    }
    const float ww = w != nullptr ? w[(c0 + c) % w_len] : 1.f;
    if (gate_first) v = v * g * inv * ww;
    else v = v * inv * ww * g;
    o[c] = from_f<T>(v);
  }
}

// The same for groups of a size that is a multiple of four (y 16-byte aligned rows, gate and out 8- / 16-byte aligned).
template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
gated_group_norm_vec4_kernel(const float* __restrict__ y, const T* __restrict__ gate, int64_t ldg, const float* __restrict__ w,
                             int w_len, int groups, int act, int gate_first, float eps, T* __restrict__ out, int cols) {
  __shared__ float red[33];
  const size_t r = blockIdx.x;
  const int gs = cols / groups, c0 = blockIdx.y * gs;
  const float* yr = y + r * cols + c0;
  const T* gr = gate != nullptr ? gate + r * ldg + c0 : nullptr;
  auto fetch = [&](int c, float4& v, float4& z) {
    v = *reinterpret_cast<const float4*>(yr + c);
    z = gr != nullptr ? load4<T>(gr + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  auto gated = [&](float4& v, float4& g) {                 // g comes in as the gate's argument
    if (gr == nullptr) g = make_float4(1.f, 1.f, 1.f, 1.f);
    else if (act == 0) g = make_float4(sigmoid_for<T>(g.x), sigmoid_for<T>(g.y), sigmoid_for<T>(g.z), sigmoid_for<T>(g.w));
    else g = make_float4(silu_for<T>(g.x), silu_for<T>(g.y), silu_for<T>(g.z), silu_for<T>(g.w));
    if (gate_first) { v.x *= g.x; v.y *= g.y; v.z *= g.z; v.w *= g.w; }
  };
  // a group of up to GN_KEEP vectors per thread stays in registers between the sum of squares and the scaled write; all of them are
  // asked for before the first gate is formed (8192 rows of 4096: 89 -> 71 us, with the
  // approximate reciprocal of the gates 55; behind each other's gates the loads came one at a time)
  constexpr int GN_KEEP = 4;
  const bool keep = gs <= 4 * GN_KEEP * static_cast<int>(blockDim.x);
  float4 kv[GN_KEEP], kg[GN_KEEP];
  float ssq = 0.f;
  if (keep) {
#pragma unroll
    for (int it = 0; it < GN_KEEP; ++it) {
      const int c = (threadIdx.x + it * blockDim.x) * 4;
      kv[it] = make_float4(0.f, 0.f, 0.f, 0.f);
      kg[it] = kv[it];
      if (c < gs) fetch(c, kv[it], kg[it]);
    }
#pragma unroll
    for (int it = 0; it < GN_KEEP; ++it) {
      if (static_cast<int>(threadIdx.x + it * blockDim.x) * 4 < gs) {
        gated(kv[it], kg[it]);
        ssq += kv[it].x * kv[it].x + kv[it].y * kv[it].y + kv[it].z * kv[it].z + kv[it].w * kv[it].w;
      }
    }
  } else {
    for (int c = threadIdx.x * 4; c < gs; c += blockDim.x * 4) {
      float4 v, g;
      fetch(c, v, g);
      gated(v, g);
      ssq += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
  }
  const float inv = 1.0f / sqrtf(block_sum(ssq, red) / static_cast<float>(gs) + eps);
  T* o = out + r * cols + c0;
  auto emit = [&](int c, const float4& v, const float4& g) {
    const int wc = w_len >= cols ? c0 + c : (c0 + c) % w_len;                              // w_len is a multiple of four here
    const float4 ww = w != nullptr ? *reinterpret_cast<const float4*>(w + wc) : make_float4(1.f, 1.f, 1.f, 1.f);
    float4 res = make_float4(v.x * inv * ww.x, v.y * inv * ww.y, v.z * inv * ww.z, v.w * inv * ww.w);
    if (!gate_first) { res.x *= g.x; res.y *= g.y; res.z *= g.z; res.w *= g.w; }
    store4<T>(o + c, res);
  };
  if (keep) {
#pragma unroll
    for (int it = 0; it < GN_KEEP; ++it) {
      const int c = (threadIdx.x + it * blockDim.x) * 4;
      if (c < gs) emit(c, kv[it], kg[it]);
    }
  } else {
    for (int c = threadIdx.x * 4; c < gs; c += blockDim.x * 4) {
      float4 v, g;
      fetch(c, v, g);
      gated(v, g);
      emit(c, v, g);
    }
  }
}

// Small groups (a head each): one CTA per row, a warp per group in turn, the group's values in registers, no barrier.
constexpr int GNW_KEEP = 4;                                // groups of up to 4 * GNW_KEEP * 32 = 512 values

template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
gated_group_norm_warp_kernel(const float* __restrict__ y, const T* __restrict__ gate, int64_t ldg, const float* __restrict__ w,
                             int w_len, int groups, int act, int gate_first, float eps, T* __restrict__ out, int cols) {
  const size_t r = blockIdx.x;
  const int gs = cols / groups, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int grp = threadIdx.x >> 5; grp < groups; grp += nw) {
    const int c0 = grp * gs;
    const float* yr = y + r * cols + c0;
    const T* gr = gate != nullptr ? gate + r * ldg + c0 : nullptr;
    float4 kv[GNW_KEEP], kg[GNW_KEEP];
    float ssq = 0.f;
#pragma unroll
    for (int it = 0; it < GNW_KEEP; ++it) {
      const int c = (lane + it * 32) * 4;
      kv[it] = make_float4(0.f, 0.f, 0.f, 0.f);
      kg[it] = make_float4(1.f, 1.f, 1.f, 1.f);
      if (c < gs) {
        kv[it] = *reinterpret_cast<const float4*>(yr + c);
        if (gr != nullptr) {
          const float4 z = load4<T>(gr + c);
          if (act == 0) kg[it] = make_float4(sigmoid_for<T>(z.x), sigmoid_for<T>(z.y), sigmoid_for<T>(z.z), sigmoid_for<T>(z.w));
          else kg[it] = make_float4(silu_for<T>(z.x), silu_for<T>(z.y), silu_for<T>(z.z), silu_for<T>(z.w));
        }
        if (gate_first) { kv[it].x *= kg[it].x; kv[it].y *= kg[it].y; kv[it].z *= kg[it].z; kv[it].w *= kg[it].w; }
        ssq += kv[it].x * kv[it].x + kv[it].y * kv[it].y + kv[it].z * kv[it].z + kv[it].w * kv[it].w;
      }
    }
    const float inv = 1.0f / sqrtf(warp_sum(ssq) / static_cast<float>(gs) + eps);
    T* o = out + r * cols + c0;
#pragma unroll
    for (int it = 0; it < GNW_KEEP; ++it) {
      const int c = (lane + it * 32) * 4;
      if (c < gs) {
        const float4 ww = w != nullptr ? *reinterpret_cast<const float4*>(w + (c0 + c) % w_len) : make_float4(1.f, 1.f, 1.f, 1.f);
        float4 res = make_float4(kv[it].x * inv * ww.x, kv[it].y * inv * ww.y, kv[it].z * inv * ww.z, kv[it].w * inv * ww.w);
        if (!gate_first) { res.x *= kg[it].x; res.y *= kg[it].y; res.z *= kg[it].z; res.w *= kg[it].w; }
        store4<T>(o + c, res);
      }
    }
  }
}

}  // namespace row
}  // namespace b2

// =================================================================================================== C ABI
using namespace b2;
using namespace b2::row;

extern "C" int b2tts_embed_bigram_streams(const int32_t* tokens, const int32_t* prev_tokens, const void* embed,
                                          const void* bigram, float* xs, int rows, int cols, int streams, int vocab,
                                          int buckets, int mul_prev, int mul_cur, int dtype, void* stream) {
  B2_REQUIRE(rows >= 0 && cols > 0 && vocab > 0 && streams >= 1 && streams <= MAX_STREAMS, B2TTS_EINVAL,
             "embed_bigram_streams: rows=%d cols=%d streams=%d (at most %d)", rows, cols, streams, MAX_STREAMS);
  B2_REQUIRE(B2_ROW_DTYPE_OK(dtype), B2TTS_EINVAL, "embed_bigram_streams: dtype %d", dtype);
  B2_REQUIRE(!bigram || buckets > 0, B2TTS_EINVAL, "embed_bigram_streams: buckets=%d", buckets);
  if (rows == 0) return B2TTS_OK;
  B2_REQUIRE(tokens && prev_tokens && embed && xs, B2TTS_EINVAL, "embed_bigram_streams: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == B2TTS_DTYPE_BF16)
    embed_bigram_kernel<__nv_bfloat16><<<rows, ROW_THREADS, 0, st>>>(tokens, prev_tokens, static_cast<const __nv_bfloat16*>(embed),
        static_cast<const __nv_bfloat16*>(bigram), xs, cols, streams, vocab, buckets, mul_prev, mul_cur);
  else
    embed_bigram_kernel<float><<<rows, ROW_THREADS, 0, st>>>(tokens, prev_tokens, static_cast<const float*>(embed),
        static_cast<const float*>(bigram), xs, cols, streams, vocab, buckets, mul_prev, mul_cur);
  B2_CHECK_LAUNCH("embed_bigram_streams");
  return B2TTS_OK;
}

extern "C" int b2tts_stream_mix_norm(float* xs, const void* y1, const void* y2, float c1, float c2, const float* mix,
                                     const float* out_w, const float* in_w, const float* norm_w, void* h, int rows, int cols,
                                     int streams, float eps, int dtype, void* stream) {
  B2_REQUIRE(rows >= 0 && cols > 0 && streams >= 1 && streams <= MAX_STREAMS, B2TTS_EINVAL,
             "stream_mix_norm: rows=%d cols=%d streams=%d (at most %d)", rows, cols, streams, MAX_STREAMS);
  B2_REQUIRE(B2_ROW_DTYPE_OK(dtype), B2TTS_EINVAL, "stream_mix_norm: dtype %d", dtype);
  if (rows == 0) return B2TTS_OK;
  B2_REQUIRE(xs && (!y1 || (mix && out_w)) && (y1 || !y2) && (!h || norm_w), B2TTS_EINVAL, "stream_mix_norm: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool vec4 = cols % 4 == 0 && cols <= 4 * SMV_KEEP * ROW_THREADS && aligned16(xs) && aligned16(norm_w) &&
                    (!y1 || aligned16(y1)) && (!y2 || aligned16(y2)) && (!h || aligned16(h));
  if (vec4 && dtype == B2TTS_DTYPE_BF16)
    stream_mix_norm_vec4_kernel<__nv_bfloat16><<<rows, ROW_THREADS, 0, st>>>(xs, static_cast<const __nv_bfloat16*>(y1),
        static_cast<const __nv_bfloat16*>(y2), c1, c2, mix, out_w, in_w, norm_w, static_cast<__nv_bfloat16*>(h), cols, streams, eps);
  else if (vec4)
    stream_mix_norm_vec4_kernel<float><<<rows, ROW_THREADS, 0, st>>>(xs, static_cast<const float*>(y1), static_cast<const float*>(y2),
        c1, c2, mix, out_w, in_w, norm_w, static_cast<float*>(h), cols, streams, eps);
  else if (dtype == B2TTS_DTYPE_BF16)
    stream_mix_norm_kernel<__nv_bfloat16><<<rows, ROW_THREADS, 0, st>>>(xs, static_cast<const __nv_bfloat16*>(y1),
        static_cast<const __nv_bfloat16*>(y2), c1, c2, mix, out_w, in_w, norm_w, static_cast<__nv_bfloat16*>(h), cols, streams, eps);
  else
    stream_mix_norm_kernel<float><<<rows, ROW_THREADS, 0, st>>>(xs, static_cast<const float*>(y1), static_cast<const float*>(y2),
        c1, c2, mix, out_w, in_w, norm_w, static_cast<float*>(h), cols, streams, eps);
  B2_CHECK_LAUNCH("stream_mix_norm");
  return B2TTS_OK;
}

extern "C" int b2tts_stream_gather_norm(const float* xs, const int32_t* rows_idx, const float* in_w, const float* norm_w,
                                        void* out, int rows, int cols, int streams, float eps, int dtype, void* stream) {
  B2_REQUIRE(rows >= 0 && cols > 0 && streams >= 1, B2TTS_EINVAL, "stream_gather_norm: rows=%d cols=%d streams=%d", rows, cols, streams);
  B2_REQUIRE(B2_ROW_DTYPE_OK(dtype), B2TTS_EINVAL, "stream_gather_norm: dtype %d", dtype);
  if (rows == 0) return B2TTS_OK;
  B2_REQUIRE(xs && norm_w && out, B2TTS_EINVAL, "stream_gather_norm: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == B2TTS_DTYPE_BF16)
    stream_gather_norm_kernel<__nv_bfloat16><<<rows, ROW_THREADS, 0, st>>>(xs, rows_idx, in_w, norm_w, static_cast<__nv_bfloat16*>(out), cols, streams, eps);
  else
    stream_gather_norm_kernel<float><<<rows, ROW_THREADS, 0, st>>>(xs, rows_idx, in_w, norm_w, static_cast<float*>(out), cols, streams, eps);
  B2_CHECK_LAUNCH("stream_gather_norm");
  return B2TTS_OK;
}

extern "C" int b2tts_attn_prep(const void* u, int64_t ldu, int q_off, int k_off, int v_off, const float* q_bias,
                               const float* k_bias, const float* v_bias, const float* q_norm_w, const float* k_norm_w,
                               const float* freq, int rot_dims, const int32_t* positions, const int32_t* slot_mapping,
                               void* q_out, void* k_cache, void* v_cache, int n_tokens, int heads, int kv_heads, int dim,
                               int vdim, float eps, int interleaved, int v_heads, int dtype, void* stream) {
  B2_REQUIRE(v_heads > 0 && (v_off >= 0 || v_heads == kv_heads), B2TTS_EINVAL, "attn_prep: %d value heads", v_heads);
  B2_REQUIRE(n_tokens >= 0 && heads > 0 && kv_heads > 0 && dim > 0 && vdim > 0 && q_off >= 0 && k_off >= 0, B2TTS_EINVAL,
             "attn_prep: bad sizes");
  B2_REQUIRE((k_cache == nullptr) == (v_cache == nullptr), B2TTS_EINVAL, "attn_prep: both caches, or neither");
  B2_REQUIRE(rot_dims >= 0 && rot_dims % 2 == 0 && rot_dims <= dim, B2TTS_EINVAL, "attn_prep: %d rotated of %d coordinates", rot_dims, dim);
  B2_REQUIRE(v_off >= 0 || vdim == dim, B2TTS_EINVAL, "attn_prep: values that are the keys need vdim == dim");
  B2_REQUIRE((q_norm_w == nullptr) == (k_norm_w == nullptr), B2TTS_EINVAL, "attn_prep: norm weights for q and k, or neither");
  B2_REQUIRE(B2_ROW_DTYPE_OK(dtype), B2TTS_EINVAL, "attn_prep: dtype %d", dtype);
  if (n_tokens == 0) return B2TTS_OK;
  B2_REQUIRE(u && positions && slot_mapping && q_out && (rot_dims == 0 || freq), B2TTS_EINVAL, "attn_prep: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  using B = __nv_bfloat16;
  const PrepArgs p{static_cast<const B*>(u), ldu, q_off, k_off, v_off, q_bias, k_bias, v_bias, q_norm_w, k_norm_w, q_norm_w != nullptr ? 1 : 0,
                   nullptr, freq, positions, rot_dims, interleaved, slot_mapping, static_cast<B*>(q_out), static_cast<B*>(k_cache),
                   static_cast<B*>(v_cache), n_tokens, heads, kv_heads, v_heads, dim, vdim, eps};
  if (dtype == B2TTS_DTYPE_BF16 && prep_vec8_applies(p))
    launch_prep_vec8(p, st);
  else if (dtype == B2TTS_DTYPE_BF16)
    attn_prep_kernel<__nv_bfloat16><<<n_tokens, ROW_THREADS, 0, st>>>(static_cast<const __nv_bfloat16*>(u), ldu, q_off, k_off, v_off,
        q_bias, k_bias, v_bias, q_norm_w, k_norm_w, freq, rot_dims, positions, slot_mapping, static_cast<__nv_bfloat16*>(q_out),
        static_cast<__nv_bfloat16*>(k_cache), static_cast<__nv_bfloat16*>(v_cache), heads, kv_heads, v_heads, dim, vdim, eps, interleaved);
  else
    attn_prep_kernel<float><<<n_tokens, ROW_THREADS, 0, st>>>(static_cast<const float*>(u), ldu, q_off, k_off, v_off, q_bias, k_bias,
        v_bias, q_norm_w, k_norm_w, freq, rot_dims, positions, slot_mapping, static_cast<float*>(q_out),
        static_cast<float*>(k_cache), static_cast<float*>(v_cache), heads, kv_heads, v_heads, dim, vdim, eps, interleaved);
  B2_CHECK_LAUNCH("attn_prep");
  return B2TTS_OK;
}

extern "C" int b2tts_attn_head_prep(const void* u, int64_t ldu, int q_off, int k_off, int v_off, const float* q_bias, const float* k_bias,
                                    const float* v_bias, const float* q_norm_w, const float* k_norm_w, const float* rot, int rot_dims,
                                    int interleaved, const int32_t* slot_mapping, void* q_out, void* k_cache, void* v_cache,
                                    int n_tokens, int heads, int kv_heads, int dim, int vdim, float eps, int dtype, void* stream) {
  B2_REQUIRE(n_tokens >= 0 && heads > 0 && kv_heads > 0 && dim > 0 && vdim > 0 && q_off >= 0 && k_off >= 0 && v_off >= 0, B2TTS_EINVAL,
             "attn_head_prep: bad sizes");
  B2_REQUIRE(rot_dims >= 0 && rot_dims % 2 == 0 && rot_dims <= dim, B2TTS_EINVAL, "attn_head_prep: %d rotated of %d coordinates", rot_dims, dim);
  B2_REQUIRE((q_norm_w == nullptr) == (k_norm_w == nullptr), B2TTS_EINVAL, "attn_head_prep: norm weights for q and k, or neither");
  B2_REQUIRE(B2_ROW_DTYPE_OK(dtype), B2TTS_EINVAL, "attn_head_prep: dtype %d", dtype);
  if (n_tokens == 0) return B2TTS_OK;
  B2_REQUIRE(u && slot_mapping && q_out && k_cache && v_cache && (rot_dims == 0 || rot), B2TTS_EINVAL, "attn_head_prep: null pointer");
  using B = __nv_bfloat16;
  const PrepArgs v{static_cast<const B*>(u), ldu, q_off, k_off, v_off, q_bias, k_bias, v_bias, q_norm_w, k_norm_w, q_norm_w != nullptr ? 2 : 0,
                   rot, nullptr, nullptr, rot_dims, interleaved, slot_mapping, static_cast<B*>(q_out), static_cast<B*>(k_cache),
                   static_cast<B*>(v_cache), n_tokens, heads, kv_heads, kv_heads, dim, vdim, eps};
  const HeadPrepArgs p{u, ldu, q_off, k_off, v_off, q_bias, k_bias, v_bias, q_norm_w, k_norm_w, rot, rot_dims, interleaved, slot_mapping,
                       q_out, k_cache, v_cache, n_tokens, heads, kv_heads, dim, vdim, eps};
  if (dtype == B2TTS_DTYPE_BF16 && prep_vec8_applies(v)) launch_prep_vec8(v, static_cast<cudaStream_t>(stream));
  else if (dtype == B2TTS_DTYPE_BF16) launch_head_prep<__nv_bfloat16>(p, static_cast<cudaStream_t>(stream));
  else launch_head_prep<float>(p, static_cast<cudaStream_t>(stream));
  B2_CHECK_LAUNCH("attn_head_prep");
  return B2TTS_OK;
}

template <typename T>
static void launch_conv_act(cudaStream_t st, const void* u, int64_t ldu, int c_off, const float* w, const float* bias, void* state,
                            const int32_t* tok_seq, const int32_t* positions, const int32_t* seq_start, const int32_t* seq_pos0,
                            const int32_t* seq_len, const int32_t* seq_slot, void* out, int64_t ldo, int n_tokens, int n_seqs,
                            int max_new, int C, int taps, int act) {
  const T* uu = static_cast<const T*>(u) + c_off;
  constexpr int VEC = 16 / static_cast<int>(sizeof(T));
  const bool vec = taps >= 2 && taps <= 4 && max_new > 0 && C % VEC == 0 && ldu % VEC == 0 && ldo % VEC == 0 && aligned16(uu) &&
                   aligned16(out) && aligned16(state) && n_seqs <= 65535;
  if (vec) {
    const int threads = std::min(128, (C / 4 + 31) / 32 * 32);
    const dim3 grid((max_new + CONV_RUN - 1) / CONV_RUN, (C / 4 + threads - 1) / threads, n_seqs);
#define CONV_RUN_GO(TP) short_conv_act_run_kernel<T, TP><<<grid, threads, 0, st>>>(uu, ldu, w, bias, static_cast<const T*>(state), seq_start, \
        seq_pos0, seq_len, seq_slot, static_cast<T*>(out), ldo, C, act)
    if (taps == 4) CONV_RUN_GO(4);
    else if (taps == 3) CONV_RUN_GO(3);
    else CONV_RUN_GO(2);
#undef CONV_RUN_GO
  } else {
    short_conv_act_kernel<T><<<dim3(n_tokens, (C + ROW_THREADS - 1) / ROW_THREADS), ROW_THREADS, 0, st>>>(
        uu, ldu, w, bias, static_cast<const T*>(state), tok_seq, positions, seq_start, seq_pos0, seq_len, seq_slot,
        static_cast<T*>(out), ldo, C, taps, act);
  }
  if (taps > 1)
    conv_state_advance_kernel<T><<<dim3((C + 127) / 128, n_seqs), 128, 0, st>>>(uu, ldu, static_cast<T*>(state), seq_start, seq_pos0,
                                                                               seq_len, seq_slot, C, taps);
}

extern "C" int b2tts_short_conv_act(const void* u, int64_t ldu, int c_off, const float* w, const float* bias, void* state,
                                    const int32_t* tok_seq, const int32_t* positions, const int32_t* seq_start,
                                    const int32_t* seq_pos0, const int32_t* seq_len, const int32_t* seq_slot, void* out,
                                    int64_t ldo, int n_tokens, int n_seqs, int max_new, int channels, int taps, int act,
                                    int dtype, void* stream) {
  B2_REQUIRE(n_tokens >= 0 && n_seqs >= 0 && channels > 0 && c_off >= 0, B2TTS_EINVAL, "short_conv_act: bad sizes");
  B2_REQUIRE(taps >= 1 && taps <= CONV_MAX_TAPS, B2TTS_EUNSUPPORTED, "short_conv_act: taps %d not in 1..%d", taps, CONV_MAX_TAPS);
  B2_REQUIRE(act == 0 || act == 1, B2TTS_EINVAL, "short_conv_act: act %d", act);
  B2_REQUIRE(B2_ROW_DTYPE_OK(dtype), B2TTS_EINVAL, "short_conv_act: dtype %d", dtype);
  if (n_tokens == 0 || n_seqs == 0) return B2TTS_OK;
  B2_REQUIRE(u && w && (state || taps == 1) && tok_seq && positions && seq_start && seq_pos0 && seq_len && seq_slot && out,
             B2TTS_EINVAL, "short_conv_act: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == B2TTS_DTYPE_BF16)
    launch_conv_act<__nv_bfloat16>(st, u, ldu, c_off, w, bias, state, tok_seq, positions, seq_start, seq_pos0, seq_len, seq_slot, out,
                                   ldo, n_tokens, n_seqs, max_new, channels, taps, act);
  else
    launch_conv_act<float>(st, u, ldu, c_off, w, bias, state, tok_seq, positions, seq_start, seq_pos0, seq_len, seq_slot, out, ldo,
                           n_tokens, n_seqs, max_new, channels, taps, act);
  B2_CHECK_LAUNCH("short_conv_act");
  return B2TTS_OK;
}

extern "C" int b2tts_gated_group_norm(const float* y, const void* gate, int64_t ldg, const float* w, int w_len, int groups,
                                      int gate_act, int gate_first, float eps, void* out, int rows, int cols, int dtype,
                                      void* stream) {
  B2_REQUIRE(rows >= 0 && cols > 0 && groups > 0 && cols % groups == 0 && (!w || w_len > 0), B2TTS_EINVAL,
             "gated_group_norm: rows=%d cols=%d groups=%d", rows, cols, groups);
  B2_REQUIRE(gate_act == 0 || gate_act == 1, B2TTS_EINVAL, "gated_group_norm: gate_act %d", gate_act);
  B2_REQUIRE(B2_ROW_DTYPE_OK(dtype), B2TTS_EINVAL, "gated_group_norm: dtype %d", dtype);
  if (rows == 0) return B2TTS_OK;
  B2_REQUIRE(y && out, B2TTS_EINVAL, "gated_group_norm: null pointer");
  if (w == nullptr) w_len = 4;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int gs = cols / groups;
  const dim3 grid(rows, groups);
  const bool vec4 = gs % 4 == 0 && w_len % 4 == 0 && ldg % 4 == 0 && aligned16(y) && (!w || aligned16(w)) && aligned16(out) &&
                    (!gate || aligned16(gate));
  if (vec4 && groups > 1 && gs <= 4 * GNW_KEEP * 32) {
    const int threads = 32 * std::min(groups, ROW_THREADS / 32);
    if (dtype == B2TTS_DTYPE_BF16)
      gated_group_norm_warp_kernel<__nv_bfloat16><<<rows, threads, 0, st>>>(y, static_cast<const __nv_bfloat16*>(gate), ldg, w, w_len,
          groups, gate_act, gate_first, eps, static_cast<__nv_bfloat16*>(out), cols);
    else
      gated_group_norm_warp_kernel<float><<<rows, threads, 0, st>>>(y, static_cast<const float*>(gate), ldg, w, w_len, groups, gate_act,
                                                                   gate_first, eps, static_cast<float*>(out), cols);
    B2_CHECK_LAUNCH("gated_group_norm");
    return B2TTS_OK;
  }
  if (vec4) {
    const int threads = std::min(ROW_THREADS, (gs / 4 + 31) / 32 * 32);
    if (dtype == B2TTS_DTYPE_BF16)
      gated_group_norm_vec4_kernel<__nv_bfloat16><<<grid, threads, 0, st>>>(y, static_cast<const __nv_bfloat16*>(gate), ldg, w, w_len,
          groups, gate_act, gate_first, eps, static_cast<__nv_bfloat16*>(out), cols);
    else
      gated_group_norm_vec4_kernel<float><<<grid, threads, 0, st>>>(y, static_cast<const float*>(gate), ldg, w, w_len, groups, gate_act,
                                                                   gate_first, eps, static_cast<float*>(out), cols);
    B2_CHECK_LAUNCH("gated_group_norm");
    return B2TTS_OK;
  }
  const int threads = std::min(ROW_THREADS, (gs + 31) / 32 * 32);
  if (dtype == B2TTS_DTYPE_BF16)
    gated_group_norm_kernel<__nv_bfloat16><<<grid, threads, 0, st>>>(y, static_cast<const __nv_bfloat16*>(gate), ldg, w, w_len, groups,
                                                                    gate_act, gate_first, eps, static_cast<__nv_bfloat16*>(out), cols);
  else
    gated_group_norm_kernel<float><<<grid, threads, 0, st>>>(y, static_cast<const float*>(gate), ldg, w, w_len, groups, gate_act,
                                                            gate_first, eps, static_cast<float*>(out), cols);
  B2_CHECK_LAUNCH("gated_group_norm");
  return B2TTS_OK;
}
