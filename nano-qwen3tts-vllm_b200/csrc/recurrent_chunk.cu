// recurrent_chunk.cu - prompt portions of the recurrences of recurrent.cu in chunks of 64 tokens on the tensor cores (bf16
// activations; state, decays, weights and sums in float).
//
// State space (any head: S <- e^l S + k (w v)^T, o = S^T q * scale + skip v).  With c_i the sum of the log decays l up to token i
// of a chunk of L tokens and S the state in front of it,
//
//   o_i = e^(c_i) S^T q_i + sum_(j <= i) e^(c_i - c_j) w_j (q_i . k_j) v_j        S <- e^(c_L) S + sum_j e^(c_L - c_j) w_j k_j v_j^T
//
// One CTA of four warps per (sequence, head, 64 value columns).  A warp owns 16 value columns: their part of the state lives
// TRANSPOSED in its accumulators (columns of S x key channels) across the chunks, where it is at once the A operand of S^T q and the
// accumulator of the update, so that the state never crosses shared memory and warps only meet over the chunk's weights.
//
// No precision is given up against the token-by-token kernel: q, k and v are bf16 and enter their products exactly; the state, the
// weights and the weighted values are floats and enter as THREE bf16 parts (24 bits), one MMA each, the small parts first (the
// tensor core truncates its sums: what is added while they are small costs nothing), the large ones summed outside; c is summed in
// double.
// Numbers that the split could not represent (not finite, or so large that a product might overflow) send their chunk through a
// token-by-token walk over the same registers, so that an infinity reaches the outputs it reaches there and no others.
//
// Bound: the chain of chunks (about 510 m16n8k16 per warp and chunk, each waiting for its fragments; the tensor pipe is 19 % busy).
// 4 sequences x 2048 tokens, 64 heads of 64 values x 128 channels: 527 us, token by token 3392 us; one sequence of 300 tokens with
// convolution and norm 100 / 229 us, of 24 tokens 70 / 73 us, of 2 tokens 93 / 95 us (launches), so every portion takes this path.
// Error of the outputs against 64 bits over 1024 tokens 8.8e-8 of their norm, token by token 8.4e-8 (plain chains of MMAs
// and scalars formed in float: 2.0e-7).
#include "scan.cuh"

namespace b2 {
namespace row {

constexpr int CK_L = 64, CK_P = 64, CK_THREADS = 128;

// x, y -> three bf16 pairs whose sums are x and y to 24 bits
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16(x, y);
  x -= bf16lo(hi); y -= bf16hi(hi);
  mid = pack_bf16(x, y);
  lo = pack_bf16(x - bf16lo(mid), y - bf16hi(mid));
}
// byte offset of 16-byte piece `ch` of row `r` in a tile of rows of `row_bytes`: pieces are permuted so that the eight rows of an
// ldmatrix phase lie in different banks
__device__ __forceinline__ uint32_t tile_off(int r, int ch, int row_bytes) { return r * row_bytes + ((ch ^ (r & 7)) << 4); }
__device__ __forceinline__ void ldsm4(uint32_t* f, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4t(uint32_t* f, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3]) : "r"(addr));
}

// c += a b with the sum of the 16 products rounded by itself and then added to nearest: the tensor core truncates when it adds to a
// running sum, and a chain of such steps leans towards zero
__device__ __forceinline__ void mma_add(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  float t[4] = {0.f, 0.f, 0.f, 0.f};
  mma_bf16_16816(t, a, b0, b1);
#pragma unroll
  for (int e = 0; e < 4; ++e) c[e] += t[e];
}

template <int D> struct ChunkTiles {
  __nv_bfloat16 q[2][CK_L * D], k[2][CK_L * D], v[2][CK_L * CK_P];
  __nv_bfloat16 m[3][CK_L * CK_L];          // the chunk's weights [i][j] in three parts
  double cum[2][CK_L];                      // sums of the log decays
  float ecum[2][CK_L], w[2][CK_L], wl[2][CK_L];   // e^(c_i); write scales; e^(c_L - c_j) w_j
  int wild[2];                              // a scalar of the chunk is out of the split's range
};

// e^x for a sum of log decays: x leaves double as a float and a remainder
__device__ __forceinline__ float exp_sum(double x) {
  const float hi = static_cast<float>(x), e = expf(hi);
  return fmaf(e, static_cast<float>(x - hi), e);
}

// Scalars of the chunk that starts at token t0, by one warp: lane l holds tokens 2 l, 2 l + 1.
template <int D>
__device__ __forceinline__ void chunk_scalars(ChunkTiles<D>& sm, int s, const float* cp, int H, int t0, int len, int lane) {
  float l[2] = {0.f, 0.f}, w[2] = {0.f, 0.f};
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int t = t0 + 2 * lane + e;
    if (t < len) { w[e] = cp[static_cast<size_t>(t) * H * 3 + 1]; l[e] = cp[static_cast<size_t>(t) * H * 3 + 2]; }
  }
  const bool fine = fabsf(l[0]) < 1e30f && fabsf(l[1]) < 1e30f && fabsf(w[0]) < 1e6f && fabsf(w[1]) < 1e6f;
  double c1 = static_cast<double>(l[0]) + l[1], x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    x = __shfl_up_sync(0xffffffffu, c1, o);
    if (lane >= o) c1 += x;
  }
  double c0 = __shfl_up_sync(0xffffffffu, c1, 1);
  c0 = (lane == 0 ? 0.0 : c0) + l[0];
  const double cl = __shfl_sync(0xffffffffu, c1, 31);
  sm.cum[s][2 * lane] = c0; sm.cum[s][2 * lane + 1] = c1;
  sm.ecum[s][2 * lane] = exp_sum(c0); sm.ecum[s][2 * lane + 1] = exp_sum(c1);
  sm.w[s][2 * lane] = w[0]; sm.w[s][2 * lane + 1] = w[1];
  sm.wl[s][2 * lane] = exp_sum(cl - c0) * w[0]; sm.wl[s][2 * lane + 1] = exp_sum(cl - c1) * w[1];
  const bool all = __all_sync(0xffffffffu, fine);
  if (lane == 0) sm.wild[s] = !all;
}

// largest magnitude (as bits) of both halves
__device__ __forceinline__ uint32_t mag2(uint32_t m, uint32_t x) { return __vmaxu2(m, x & 0x7fff7fffu); }
constexpr uint32_t CK_BIG_IN = (127 + 40) << 7;       // bf16 bits of 2^40
constexpr float CK_BIG_STATE = 1.2089258e24f;         // 2^80: times 2^40 and 128 terms still finite

template <int D>
__global__ void __launch_bounds__(CK_THREADS, 2)
linear_chunk_kernel(const ScanArgs a) {
  constexpr int RB = D * 2, VB = CK_P * 2, MB = CK_L * 2, NT = D / 8;
  extern __shared__ __align__(128) unsigned char ck_smem[];
  ChunkTiles<D>& sm = *reinterpret_cast<ChunkTiles<D>*>(ck_smem);
  const int b = blockIdx.z, h = blockIdx.y, p0 = blockIdx.x * CK_P;
  const int len = a.seq_len[b];
  if (len <= 1) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g4 = lane >> 2, c2 = 2 * (lane & 3);
  const int H = a.H, dv = a.dv, g = h / (H / a.G);
  const size_t start = a.seq_start[b];
  using B = __nv_bfloat16;
  const B* qg = static_cast<const B*>(a.q) + start * a.ldq + static_cast<size_t>(g) * D;
  const B* kg = static_cast<const B*>(a.k) + start * a.ldk + static_cast<size_t>(g) * D;
  const B* vg = static_cast<const B*>(a.v) + start * a.ldv + static_cast<size_t>(h) * dv + p0;
  const float* cp = a.coef + (start * H + h) * 3;
  float* Sg = a.state + (static_cast<size_t>(a.seq_slot[b]) * H + h) * D * dv + p0;
  float* og = a.out + start * H * dv + static_cast<size_t>(h) * dv + p0;
  const float skip = a.skip != nullptr ? a.skip[h] : 0.f;
  auto load_chunk = [&](int t0, int s) {
    for (int idx = tid; idx < CK_L * (D / 8); idx += CK_THREADS) {
      const int j = idx / (D / 8), ch = idx % (D / 8);
      const bool ok = t0 + j < len;
      const size_t row = ok ? t0 + j : 0;
      cp_async_16(reinterpret_cast<unsigned char*>(sm.q[s]) + tile_off(j, ch, RB), qg + row * a.ldq + ch * 8, ok);
      cp_async_16(reinterpret_cast<unsigned char*>(sm.k[s]) + tile_off(j, ch, RB), kg + row * a.ldk + ch * 8, ok);
    }
    for (int idx = tid; idx < CK_L * (CK_P / 8); idx += CK_THREADS) {
      const int j = idx / (CK_P / 8), ch = idx % (CK_P / 8);
      const bool ok = t0 + j < len;
      cp_async_16(reinterpret_cast<unsigned char*>(sm.v[s]) + tile_off(j, ch, VB), vg + (ok ? t0 + j : 0) * a.ldv + ch * 8, ok);
    }
  };
  load_chunk(0, 0);
  cp_async_commit();
  if (warp == 3) chunk_scalars<D>(sm, 0, cp, H, 0, len, lane);
  // S^T fragments: value columns pr (+ 8), key channels nt * 8 + c2 (+ 1)
  const int pr = warp * 16 + g4;
  float S[NT][4];
  const bool carried = a.seq_pos0[b] > 0;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) S[nt][e] = carried ? Sg[static_cast<size_t>(nt * 8 + c2 + (e & 1)) * dv + pr + 8 * (e >> 1)] : 0.f;
  const uint32_t m_u = smem_u32(sm.m);
  const int ra = lane & 15, ca = lane >> 4;                                         // A rows / B rows by [n][k] and [k][n] tiles
  const int rb = (lane >> 4) * 8 + (lane & 7), cb = (lane >> 3) & 1;
  const int rt = ((lane >> 3) & 1) * 8 + (lane & 7), ct = lane >> 4;
  for (int t0 = 0, s = 0; t0 < len; t0 += CK_L, s ^= 1) {
    const int L = min(CK_L, len - t0);
    cp_async_wait<0>();
    // ---- this thread's share of the tiles and of the state within the range of the split?
    bool wild = false;
    {
      __syncthreads();                                                              // the chunk has landed; the previous one is consumed
      uint32_t m = 0;
      const uint4* t4 = reinterpret_cast<const uint4*>(sm.q[s]);
      for (int i = tid; i < CK_L * D / 8; i += CK_THREADS) { const uint4 x = t4[i]; m = mag2(mag2(mag2(mag2(m, x.x), x.y), x.z), x.w); }
      t4 = reinterpret_cast<const uint4*>(sm.k[s]);
      for (int i = tid; i < CK_L * D / 8; i += CK_THREADS) { const uint4 x = t4[i]; m = mag2(mag2(mag2(mag2(m, x.x), x.y), x.z), x.w); }
      t4 = reinterpret_cast<const uint4*>(sm.v[s]);
      for (int i = tid; i < CK_L * CK_P / 8; i += CK_THREADS) { const uint4 x = t4[i]; m = mag2(mag2(mag2(mag2(m, x.x), x.y), x.z), x.w); }
      wild = (m & 0xffffu) >= CK_BIG_IN || (m >> 16) >= CK_BIG_IN || sm.wild[s];
      bool small = true;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) small = small && fabsf(S[nt][e]) < CK_BIG_STATE;
      wild = wild || !small;
    }
    if (t0 + CK_L < len) load_chunk(t0 + CK_L, s ^ 1);
    cp_async_commit();
    if (__syncthreads_or(wild)) {
      // ---- token by token: the same sums, every product in float
      for (int i = 0; i < L; ++i) {
        const float* c = cp + static_cast<size_t>(t0 + i) * H * 3;
        const float c0 = c[0], c1 = c[1];
        const float v0 = to_f(sm.v[s][tile_off(i, pr >> 3, VB) / 2 + (pr & 7)]), v1 = to_f(sm.v[s][tile_off(i, (pr + 8) >> 3, VB) / 2 + (pr & 7)]);
        float o0 = 0.f, o1 = 0.f;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const uint32_t off = tile_off(i, nt, RB) / 2 + c2 + e;
            const float kk = to_f(sm.k[s][off]), qq = to_f(sm.q[s][off]);
            S[nt][e] = c0 * S[nt][e] + kk * (c1 * v0);         o0 += S[nt][e] * qq;
            S[nt][e + 2] = c0 * S[nt][e + 2] + kk * (c1 * v1); o1 += S[nt][e + 2] * qq;
          }
#pragma unroll
        for (int x = 1; x < 4; x <<= 1) { o0 += __shfl_xor_sync(0xffffffffu, o0, x); o1 += __shfl_xor_sync(0xffffffffu, o1, x); }
        if ((lane & 3) == 0) {
          og[static_cast<size_t>(t0 + i) * H * dv + pr] = o0 * a.qscale + skip * v0;
          og[static_cast<size_t>(t0 + i) * H * dv + pr + 8] = o1 * a.qscale + skip * v1;
        }
      }
      if (warp == 3 && t0 + CK_L < len) chunk_scalars<D>(sm, s ^ 1, cp, H, t0 + CK_L, len, lane);
      continue;
    }
    const uint32_t q_u = smem_u32(sm.q[s]), k_u = smem_u32(sm.k[s]), v_u = smem_u32(sm.v[s]);
    // ---- weights of rows 16 warp .. + 15: scores against the keys up to the diagonal, decay and write scale, in three parts
    if (warp * 16 < L) {
      float sc[8][4];
#pragma unroll
      for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[nt][e] = 0.f;
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        uint32_t af[4];
        ldsm4(af, q_u + tile_off(warp * 16 + ra, ks * 2 + ca, RB));
#pragma unroll
        for (int np = 0; np < 4; ++np) {
          if (np <= warp) {
            uint32_t bf[4];
            ldsm4(bf, k_u + tile_off(np * 16 + rb, ks * 2 + cb, RB));
            mma_add(sc[2 * np], af, bf[0], bf[1]);
            mma_add(sc[2 * np + 1], af, bf[2], bf[3]);
          }
        }
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int i = warp * 16 + g4 + 8 * half;
        const double ci = sm.cum[s][i];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
          if (nt <= 2 * warp + 1) {
            const int j = nt * 8 + c2;
            const float x = j <= i ? sc[nt][2 * half] * (exp_sum(ci - sm.cum[s][j]) * sm.w[s][j]) : 0.f;
            const float y = j + 1 <= i ? sc[nt][2 * half + 1] * (exp_sum(ci - sm.cum[s][j + 1]) * sm.w[s][j + 1]) : 0.f;
            uint32_t hi, mid, lo;
            split3(x, y, hi, mid, lo);
            const uint32_t off = (tile_off(i, nt, MB) + c2 * 2) / 4;
            reinterpret_cast<uint32_t*>(sm.m[0])[off] = hi;
            reinterpret_cast<uint32_t*>(sm.m[1])[off] = mid;
            reinterpret_cast<uint32_t*>(sm.m[2])[off] = lo;
          }
        }
      }
    }
    // ---- S^T q: this warp's 16 value columns x the chunk's tokens; the small parts first, so that they are added to small sums
    float o[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[nt][e] = 0.f;
    const bool front = carried || t0 > 0;
    if (front) {
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        uint32_t hi[4], mid[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split3(S[2 * ks + (e >> 1)][2 * (e & 1)], S[2 * ks + (e >> 1)][2 * (e & 1) + 1], hi[e], mid[e], lo[e]);
#pragma unroll
        for (int np = 0; np < 4; ++np) {
          if (np * 16 < L) {
            uint32_t bf[4];
            ldsm4(bf, q_u + tile_off(np * 16 + rb, ks * 2 + cb, RB));
            mma_bf16_16816(o[2 * np], lo, bf[0], bf[1]);
            mma_bf16_16816(o[2 * np + 1], lo, bf[2], bf[3]);
            mma_bf16_16816(o[2 * np], mid, bf[0], bf[1]);
            mma_bf16_16816(o[2 * np + 1], mid, bf[2], bf[3]);
          }
        }
      }
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        uint32_t hi[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) hi[e] = pack_bf16(S[2 * ks + (e >> 1)][2 * (e & 1)], S[2 * ks + (e >> 1)][2 * (e & 1) + 1]);
#pragma unroll
        for (int np = 0; np < 4; ++np) {
          if (np * 16 < L) {
            uint32_t bf[4];
            ldsm4(bf, q_u + tile_off(np * 16 + rb, ks * 2 + cb, RB));
            mma_add(o[2 * np], hi, bf[0], bf[1]);
            mma_add(o[2 * np + 1], hi, bf[2], bf[3]);
          }
        }
      }
    }
    __syncthreads();                                                                // the weights are in shared memory
    if (warp == 3 && t0 + CK_L < len) chunk_scalars<D>(sm, s ^ 1, cp, H, t0 + CK_L, len, lane);
    // ---- the chunk's own tokens, again the small parts first
    uint32_t vf[4][4];                                                              // v transposed: value columns x 16 tokens
    {
      float oi[8][4];
#pragma unroll
      for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) oi[nt][e] = 0.f;
#pragma unroll
      for (int js = 0; js < 4; ++js) ldsm4t(vf[js], v_u + tile_off(js * 16 + rb, warp * 2 + cb, VB));
#pragma unroll
      for (int part = 2; part >= 0; --part)
#pragma unroll
        for (int js = 0; js < 4; ++js)
#pragma unroll
          for (int np = 0; np < 4; ++np) {
            if (np >= js && np * 16 < L) {
              uint32_t bf[4];
              ldsm4(bf, m_u + part * (CK_L * MB) + tile_off(np * 16 + rb, js * 2 + cb, MB));
              if (part > 0) {
                mma_bf16_16816(oi[2 * np], vf[js], bf[0], bf[1]);
                mma_bf16_16816(oi[2 * np + 1], vf[js], bf[2], bf[3]);
              } else {
                mma_add(oi[2 * np], vf[js], bf[0], bf[1]);
                mma_add(oi[2 * np + 1], vf[js], bf[2], bf[3]);
              }
            }
          }
#pragma unroll
      for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = nt * 8 + c2 + (e & 1), p = pr + 8 * (e >> 1);
          if (i < L) {
            float x = (front ? fmaf(sm.ecum[s][i], o[nt][e], oi[nt][e]) : oi[nt][e]) * a.qscale;
            if (a.skip != nullptr) x += skip * to_f(sm.v[s][tile_off(i, p >> 3, VB) / 2 + (p & 7)]);
            og[static_cast<size_t>(t0 + i) * H * dv + p] = x;
          }
        }
    }
    // ---- the state behind the chunk: what the chunk adds is summed by itself, then S <- e^(c_L) S + sum with one rounding
    uint32_t af[4][3][4];
#pragma unroll
    for (int js = 0; js < 4; ++js)
#pragma unroll
      for (int e = 0; e < 4; ++e) {                                                 // registers 0, 1: tokens c2, c2 + 1; 2, 3: eight further on
        const int j = js * 16 + (e >> 1) * 8 + c2;
        split3(bf16lo(vf[js][e]) * sm.wl[s][j], bf16hi(vf[js][e]) * sm.wl[s][j + 1], af[js][0][e], af[js][1][e], af[js][2][e]);
      }
    const float gl = sm.ecum[s][CK_L - 1];                                          // log decays behind the portion's end are zero
#pragma unroll
    for (int np = 0; np < D / 16; ++np) {
      float t[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      uint32_t bf[4][4];
#pragma unroll
      for (int js = 0; js < 4; ++js)
        if (js * 16 < L) ldsm4t(bf[js], k_u + tile_off(js * 16 + rt, np * 2 + ct, RB));
#pragma unroll
      for (int part = 2; part >= 0; --part)
#pragma unroll
        for (int js = 0; js < 4; ++js)
          if (js * 16 < L) {
            if (part > 0) {
              mma_bf16_16816(t[0], af[js][part], bf[js][0], bf[js][1]);
              mma_bf16_16816(t[1], af[js][part], bf[js][2], bf[js][3]);
            } else {
              mma_add(t[0], af[js][part], bf[js][0], bf[js][1]);
              mma_add(t[1], af[js][part], bf[js][2], bf[js][3]);
            }
          }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        S[2 * np][e] = fmaf(gl, S[2 * np][e], t[0][e]);
        S[2 * np + 1][e] = fmaf(gl, S[2 * np + 1][e], t[1][e]);
      }
    }
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) Sg[static_cast<size_t>(nt * 8 + c2 + (e & 1)) * dv + pr + 8 * (e >> 1)] = S[nt][e];
}

bool scan_chunk_applies(const ScanArgs& a) {
  return (a.d == 64 || a.d == 128) && a.dv % CK_P == 0 && a.ldq % 8 == 0 && a.ldk % 8 == 0 && a.ldv % 8 == 0 && aligned16(a.q) &&
         aligned16(a.k) && aligned16(a.v) && a.head_decay == nullptr && !a.divide;
}

template <int D>
static int go_linear(const char* what, const ScanArgs& a, int n_seqs, cudaStream_t st) {
  constexpr int smem = static_cast<int>(sizeof(ChunkTiles<D>));
  const cudaError_t e = cudaFuncSetAttribute(linear_chunk_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return cuda_fail(e, what);
  linear_chunk_kernel<D><<<dim3(a.dv / CK_P, a.H, n_seqs), CK_THREADS, smem, st>>>(a);
  B2_CHECK_LAUNCH(what);
  return B2TTS_OK;
}

int launch_linear_chunk(const char* what, const ScanArgs& a, int n_seqs, cudaStream_t st) {
  return a.d == 64 ? go_linear<64>(what, a, n_seqs, st) : go_linear<128>(what, a, n_seqs, st);
}

}  // namespace row
}  // namespace b2
