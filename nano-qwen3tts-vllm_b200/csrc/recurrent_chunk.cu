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
// No precision is given up against the token-by-token kernel (outputs 7.9e-8 of their norm from 64 bits and the state 7.0e-8, that
// one's 8.5e-8 and 8.1e-8: means over 512 tokens of eight inputs of three sizes; plain chains of MMAs 2.0e-7).  q, k and v are bf16
// and enter their products exactly; the state, the weights and the weighted values are floats and enter as THREE bf16 parts (24
// bits), one MMA each, the small parts first (the tensor core truncates its sums: what is added while they are small costs
// nothing), the large ones summed outside; c is summed in double.
// Numbers that the split could not represent (not finite, or so large that a product might overflow) send their chunk through a
// token-by-token walk over the same registers, so that an infinity reaches the outputs it reaches there and no others.
//
// Bound: the chain of chunks, 22500 cycles each with two CTAs a multiprocessor: 9500 S^T q and the weights, 5200 the update (its 256 m16n8k16 a warp are 4100 of
// them), 4100 the chunk's own tokens and the outputs, 2100 until the chunk has landed and is known to be in range.  Scores of queries and keys do not
// depend on the state and are the same for all heads of a group, so a kernel in front forms them once (chunk_scores_kernel) where at least four
// heads share them; rows up to the diagonal are uneven, so that the weights are shared out by tiles of 8 x 8 (the last warp had four times the
// exponentials of the first and the others waited: 28000 cycles), each small and large part of the state is multiplied beside one reading of the queries, decays are
// differences of pairs of floats (conversions from double were half of them), and skipped values come from the registers that hold them.
// 4 sequences x 2048 tokens, 64 heads of 64 values x 128 channels: 504 -> 452 us, 64 channels and 32 heads 316 -> 237; one sequence of 300 tokens 70 -> 61,
// 64 of 64 tokens 255 -> 239.  Scores that are asked for only during S^T q made it 465, two readings of the queries 527.
// Errors against 64 bits over 512 tokens, 24 inputs of three sizes, outputs / state: 128 channels 8.46e-8 / 7.64e-8 -> 8.43e-8 / 7.64e-8, 64 channels 8.10e-8 /
// 7.83e-8 -> 8.02e-8 / 7.83e-8.  Short portions stay with the token-by-token kernel, see linear_walk_len().
#include <type_traits>

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

// two bf16 in two pairs: the upper four of their significant bits, and the rest (exact)
__device__ __forceinline__ void halves(uint32_t x, uint32_t& head, uint32_t& tail) {
  head = x & 0xfff0fff0u;
  const __nv_bfloat162 r = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&x), *reinterpret_cast<const __nv_bfloat162*>(&head));
  tail = *reinterpret_cast<const uint32_t*>(&r);
}

template <int D> struct ChunkTiles {
  __nv_bfloat16 q[2][CK_L * D], k[2][CK_L * D], v[2][CK_L * CK_P];
  __nv_bfloat16 m[3][CK_L * CK_L];          // the chunk's weights [i][j] in three parts
  float2 cum[2][CK_L];                      // sums of the log decays: a float and what it leaves
  float ecum[2][CK_L], w[2][CK_L], wl[2][CK_L];   // e^(c_i); write scales; e^(c_L - c_j) w_j
  int wild[2];                              // a scalar of the chunk is out of the split's range
};

// e^x for a sum of log decays: x leaves double as a float and a remainder
__device__ __forceinline__ float exp_sum(double x) {
  const float hi = static_cast<float>(x), e = expf(hi);
  return fmaf(e, static_cast<float>(x - hi), e);
}

// e^(a - b) of two such sums in pairs of floats: the difference of the first floats with its rounding error, which joins the differences of the second ones (48
// bits; conversions between float and double cost eight times an addition), then the exponential of the nearest float and what that leaves
__device__ __forceinline__ float exp_between(float2 a, float2 b) {
  const float d = a.x - b.x, t = d - a.x, rest = ((a.x - (d - t)) - (b.x + t)) + (a.y - b.y), x = d + rest, e = expf(x);
  return fmaf(e, rest - (x - d), e);
}

// A log decay as it enters the sums.  e^l is 0 in float below -104; taken as it comes, a very large l would leave the running sum of
// doubles no bits for the decays behind it (from |l| = 1e12 on), so it is cut at a value that gives the same products.
__device__ __forceinline__ float cut_log(float l) { return fmaxf(l, -200.f); }

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
  l[0] = cut_log(l[0]); l[1] = cut_log(l[1]);
  double c1 = static_cast<double>(l[0]) + l[1], x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    x = __shfl_up_sync(0xffffffffu, c1, o);
    if (lane >= o) c1 += x;
  }
  double c0 = __shfl_up_sync(0xffffffffu, c1, 1);
  c0 = (lane == 0 ? 0.0 : c0) + l[0];
  const double cl = __shfl_sync(0xffffffffu, c1, 31);
  const float h0 = static_cast<float>(c0), h1 = static_cast<float>(c1);
  sm.cum[s][2 * lane] = make_float2(h0, static_cast<float>(c0 - h0)); sm.cum[s][2 * lane + 1] = make_float2(h1, static_cast<float>(c1 - h1));
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

// Scores of a chunk's queries 16 warp .. + 15 against its keys up to the diagonal, sc[nt]: keys 8 nt + c2 (+ 1), queries g4 (+ 8).
template <int D>
__device__ __forceinline__ void chunk_row_scores(uint32_t q_u, uint32_t k_u, int warp, int lane, float sc[8][4]) {
  constexpr int RB = D * 2;
  const int ra = lane & 15, ca = lane >> 4, rb = (lane >> 4) * 8 + (lane & 7), cb = (lane >> 3) & 1;
  // the upper halves of q's significant bits give sums of 16 products that a float nearly always holds, the lower ones small sums:
  // what the tensor core cuts off is a sixteenth (outputs 8.8e-8 -> 7.9e-8 from 64 bits, 12 of 574 us)
  float st[8][4];
#pragma unroll
  for (int nt = 0; nt < 8; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) sc[nt][e] = st[nt][e] = 0.f;
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks) {
    uint32_t af[4], hf[4], tf[4];
    ldsm4(af, q_u + tile_off(warp * 16 + ra, ks * 2 + ca, RB));
#pragma unroll
    for (int e = 0; e < 4; ++e) halves(af[e], hf[e], tf[e]);
#pragma unroll
    for (int np = 0; np < 4; ++np) {
      if (np <= warp) {
        uint32_t bf[4];
        ldsm4(bf, k_u + tile_off(np * 16 + rb, ks * 2 + cb, RB));
        mma_bf16_16816(st[2 * np], tf, bf[0], bf[1]);
        mma_bf16_16816(st[2 * np + 1], tf, bf[2], bf[3]);
        mma_add(sc[2 * np], hf, bf[0], bf[1]);
        mma_add(sc[2 * np + 1], hf, bf[2], bf[3]);
      }
    }
  }
#pragma unroll
  for (int nt = 0; nt < 8; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) sc[nt][e] += st[nt][e];
}

// The chunks of the sequences in front of sequence b, which its own are numbered behind: wherever the sequences' rows lie, no two
// chunks of a step share a number.  All 32 lanes of a warp call it.
__device__ __forceinline__ int chunks_before(const int32_t* seq_len, int b, int lane) {
  int n = 0;
  for (int i = lane; i < b; i += 32) n += (max(seq_len[i], 0) + CK_L - 1) / CK_L;
  return __reduce_add_sync(0xffffffffu, n);
}
constexpr int CK_SCORES = CK_L * CK_L;     // floats of a chunk's scores, as the threads hold them: [warp][nt][lane] float4

// The scores of every chunk and group of heads, formed once where many heads share their queries and keys: in the chain of chunks they
// were a fifth of the products and were formed again for every head.  Behind them one word per chunk: something is out of the split's range.
template <int D>
__global__ void __launch_bounds__(CK_THREADS)
chunk_scores_kernel(const ScanArgs a, int64_t chunks) {
  constexpr int RB = D * 2;
  __shared__ __align__(128) __nv_bfloat16 q_s[CK_L * D], k_s[CK_L * D];
  const int b = blockIdx.z, g = blockIdx.y, t0 = blockIdx.x * CK_L, len = a.seq_len[b];
  if (len < a.min_len || t0 >= len) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t start = a.seq_start[b], number = static_cast<int64_t>(chunks_before(a.seq_len, b, lane) + t0 / CK_L) * a.G + g;
  const __nv_bfloat16* qg = static_cast<const __nv_bfloat16*>(a.q) + start * a.ldq + static_cast<size_t>(g) * D;
  const __nv_bfloat16* kg = static_cast<const __nv_bfloat16*>(a.k) + start * a.ldk + static_cast<size_t>(g) * D;
  for (int idx = tid; idx < CK_L * (D / 8); idx += CK_THREADS) {
    const int j = idx / (D / 8), ch = idx % (D / 8);
    const bool ok = t0 + j < len;
    const size_t row = ok ? t0 + j : 0;
    cp_async_16(reinterpret_cast<unsigned char*>(q_s) + tile_off(j, ch, RB), qg + row * a.ldq + ch * 8, ok);
    cp_async_16(reinterpret_cast<unsigned char*>(k_s) + tile_off(j, ch, RB), kg + row * a.ldk + ch * 8, ok);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  uint32_t m = 0;
  for (int i = tid; i < CK_L * D / 8; i += CK_THREADS) {
    const uint4 x = reinterpret_cast<const uint4*>(q_s)[i], y = reinterpret_cast<const uint4*>(k_s)[i];
    m = mag2(mag2(mag2(mag2(m, x.x), x.y), x.z), x.w);
    m = mag2(mag2(mag2(mag2(m, y.x), y.y), y.z), y.w);
  }
  const int wild = __syncthreads_or((m & 0xffffu) >= CK_BIG_IN || (m >> 16) >= CK_BIG_IN);
  if (tid == 0) reinterpret_cast<int*>(a.scores + chunks * a.G * CK_SCORES)[number] = wild;
  float sc[8][4];
  chunk_row_scores<D>(smem_u32(q_s), smem_u32(k_s), warp, lane, sc);
  float4* out = reinterpret_cast<float4*>(a.scores + number * CK_SCORES) + warp * 8 * 32 + lane;
#pragma unroll
  for (int nt = 0; nt < 8; ++nt)
    if (nt <= 2 * warp + 1) out[nt * 32] = make_float4(sc[nt][0], sc[nt][1], sc[nt][2], sc[nt][3]);
}

// The 36 tiles of 8 x 8 up to the diagonal of a chunk, counted row by row: row of tiles * 8 + column
__device__ __forceinline__ int ck_tile(int n) {
  const int row = (n >= 1) + (n >= 3) + (n >= 6) + (n >= 10) + (n >= 15) + (n >= 21) + (n >= 28);
  return row * 8 + n - row * (row + 1) / 2;
}

// AHEAD: chunk_scores_kernel has run
template <int D, bool AHEAD>
__global__ void __launch_bounds__(CK_THREADS, 2)
linear_chunk_kernel(const ScanArgs a, int64_t chunks) {
  constexpr int RB = D * 2, VB = CK_P * 2, MB = CK_L * 2, NT = D / 8;
  extern __shared__ __align__(128) unsigned char ck_smem[];
  ChunkTiles<D>& sm = *reinterpret_cast<ChunkTiles<D>*>(ck_smem);
  const int b = blockIdx.z, h = blockIdx.y, p0 = blockIdx.x * CK_P;
  const int len = a.seq_len[b];
  if (len < a.min_len) return;
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
  for (int i = tid; i < 3 * CK_L * CK_L / 8; i += CK_THREADS) reinterpret_cast<uint4*>(sm.m[0])[i] = make_uint4(0, 0, 0, 0);      // above the diagonal it stays so
  load_chunk(0, 0);
  cp_async_commit();
  int chunk0 = 0, out_of_range = 0;                        // number of the sequence's first chunk; the next chunk's word behind the scores
  if constexpr (AHEAD) {
    chunk0 = chunks_before(a.seq_len, b, lane);
    out_of_range = reinterpret_cast<const int*>(a.scores + chunks * a.G * CK_SCORES)[static_cast<int64_t>(chunk0) * a.G + g];
  }
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
  const int rb = (lane >> 4) * 8 + (lane & 7), cb = (lane >> 3) & 1;
  const int rt = ((lane >> 3) & 1) * 8 + (lane & 7), ct = lane >> 4;
  for (int t0 = 0, s = 0; t0 < len; t0 += CK_L, s ^= 1) {
    const int L = min(CK_L, len - t0);
    cp_async_wait<0>();
    // ---- this thread's share of the tiles and of the state within the range of the split?
    bool wild = false;
    float2 ahead[AHEAD ? 9 : 1];
    {
      __syncthreads();                                                              // the chunk has landed; the previous one is consumed
      uint32_t m = 0;
      const uint4* t4;
      if constexpr (AHEAD) {
        // asked for here, used behind S^T q; whether something is out of range was asked for a chunk ago
        const int64_t number = static_cast<int64_t>(chunk0 + t0 / CK_L) * a.G + g;
        const float2* sc = reinterpret_cast<const float2*>(a.scores + number * CK_SCORES);
#pragma unroll
        for (int x = 0; x < 9; ++x) {
          const int tile = ck_tile(warp + 4 * x), oct = tile >> 3;
          ahead[x] = sc[((((oct >> 1) * 8 + (tile & 7)) * 32) + lane) * 2 + (oct & 1)];
        }
        wild = out_of_range != 0;
        if (t0 + CK_L < len) out_of_range = reinterpret_cast<const int*>(a.scores + chunks * a.G * CK_SCORES)[number + a.G];
      } else {
        t4 = reinterpret_cast<const uint4*>(sm.q[s]);
        for (int i = tid; i < CK_L * D / 8; i += CK_THREADS) { const uint4 x = t4[i]; m = mag2(mag2(mag2(mag2(m, x.x), x.y), x.z), x.w); }
        t4 = reinterpret_cast<const uint4*>(sm.k[s]);
        for (int i = tid; i < CK_L * D / 8; i += CK_THREADS) { const uint4 x = t4[i]; m = mag2(mag2(mag2(mag2(m, x.x), x.y), x.z), x.w); }
      }
      t4 = reinterpret_cast<const uint4*>(sm.v[s]);
      for (int i = tid; i < CK_L * CK_P / 8; i += CK_THREADS) { const uint4 x = t4[i]; m = mag2(mag2(mag2(mag2(m, x.x), x.y), x.z), x.w); }
      wild = wild || (m & 0xffffu) >= CK_BIG_IN || (m >> 16) >= CK_BIG_IN || sm.wild[s];
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
    // ---- S^T q: this warp's 16 value columns x the chunk's tokens; the small parts by themselves, then the large ones with their sum
    float o[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[nt][e] = 0.f;
    const bool front = carried || t0 > 0;
    if (front) {
      float large[8][4];
#pragma unroll
      for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) large[nt][e] = 0.f;
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
            mma_add(large[2 * np], hi, bf[0], bf[1]);
            mma_add(large[2 * np + 1], hi, bf[2], bf[3]);
            mma_bf16_16816(o[2 * np], mid, bf[0], bf[1]);
            mma_bf16_16816(o[2 * np + 1], mid, bf[2], bf[3]);
          }
        }
      }
#pragma unroll
      for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[nt][e] += large[nt][e];
    }
    // ---- the chunk's weights: scores up to the diagonal, decay and write scale, in three parts
    auto weigh = [&](int i, int nt, float s0, float s1) {                           // row i, columns 8 nt + c2 (+ 1)
      const int j = nt * 8 + c2;
      const float2 ci = sm.cum[s][i], wj = *reinterpret_cast<const float2*>(sm.w[s] + j);
      const float4 cj = *reinterpret_cast<const float4*>(sm.cum[s] + j);
      const float x = j <= i ? s0 * (exp_between(ci, make_float2(cj.x, cj.y)) * wj.x) : 0.f;
      const float y = j + 1 <= i ? s1 * (exp_between(ci, make_float2(cj.z, cj.w)) * wj.y) : 0.f;
      uint32_t hi, mid, lo;
      split3(x, y, hi, mid, lo);
      const uint32_t off = (tile_off(i, nt, MB) + c2 * 2) / 4;
      reinterpret_cast<uint32_t*>(sm.m[0])[off] = hi;
      reinterpret_cast<uint32_t*>(sm.m[1])[off] = mid;
      reinterpret_cast<uint32_t*>(sm.m[2])[off] = lo;
    };
    if constexpr (AHEAD) {
#pragma unroll
      for (int x = 0; x < 9; ++x) {                                                 // nine of the 36 tiles of 8 x 8 each: rows up to the diagonal are uneven
        const int tile = ck_tile(warp + 4 * x), oct = tile >> 3;
        if (oct * 8 < L) weigh(oct * 8 + g4, tile & 7, ahead[x].x, ahead[x].y);
      }
    } else if (warp * 16 < L) {
      float sc[8][4];
      chunk_row_scores<D>(q_u, k_u, warp, lane, sc);
#pragma unroll
      for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
          if (nt <= 2 * warp + half) weigh(warp * 16 + g4 + 8 * half, nt, sc[nt][2 * half], sc[nt][2 * half + 1]);
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
      for (int nt = 0; nt < 8; ++nt) {
        const float2 ec = *reinterpret_cast<const float2*>(sm.ecum[s] + nt * 8 + c2);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = nt * 8 + c2 + (e & 1);
          const uint32_t vw = vf[nt >> 1][2 * (nt & 1) + (e >> 1)];                 // v lies in the lanes as the sums do
          float x = (front ? fmaf(e & 1 ? ec.y : ec.x, o[nt][e], oi[nt][e]) : oi[nt][e]) * a.qscale;
          if (a.skip != nullptr) x += skip * (e & 1 ? bf16hi(vw) : bf16lo(vw));
          if (i < L) og[static_cast<size_t>(t0 + i) * H * dv + pr + 8 * (e >> 1)] = x;
        }
      }
    }
    // ---- the state behind the chunk: what the chunk adds is summed by itself, then S <- e^(c_L) S + sum with one rounding
    uint32_t af[4][4][4];
#pragma unroll
    for (int js = 0; js < 4; ++js)
#pragma unroll
      for (int e = 0; e < 4; ++e) {                                                 // registers 0, 1: tokens c2, c2 + 1; 2, 3: eight further on
        const int j = js * 16 + (e >> 1) * 8 + c2;
        uint32_t hi;
        split3(bf16lo(vf[js][e]) * sm.wl[s][j], bf16hi(vf[js][e]) * sm.wl[s][j + 1], hi, af[js][2][e], af[js][3][e]);
        halves(hi, af[js][0][e], af[js][1][e]);                                     // as above: state 7.4e-8 -> 7.0e-8, 28 us
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
      for (int part = 3; part >= 0; --part)
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

// ------------------------------------------------------------------ delta rule
// S <- e^l S; u = beta (v - S^T k^); S <- S + k^ u^T; o = S^T q^ * scale with unit vectors k^ = kn k, q^ = qn q.  Inside a chunk
//
//   u_i + sum_(j < i) A_ij u_j = r_i = beta_i (v_i - e^(c_i) S^T k^_i),   A_ij = beta_i e^(c_i - c_j) (k^_i . k^_j)
//   o_i = e^(c_i) S^T q^_i + sum_(j <= i) M_ij u_j,  M_ij = e^(c_i - c_j) (q^_i . k^_j)          S <- e^(c_L) S + sum_j e^(c_L - c_j) k^_j u_j^T
//
// Everything but r, u, o and S says nothing about the state: decays, norms, M and the solved system u = r - N r with N = 1 - (1 + A)^-1 are
// formed per chunk and head by delta_prepare() - by delta_prepare_kernel for all chunks at once where there is room for them, by the chain itself
// else, to the same bits.  What is left of the chain: S^T k, N r, the state's update (and, beside them, the outputs).
//
// One CTA of eight warps per (sequence, head, 64 value columns).  Warp (wp, wh) owns value columns 16 wp .. + 15 and the wh-th half of
// the key channels of the state, transposed in its accumulators as above.  A pair of warps meets twice a chunk over a barrier of its own: what the
// halves sum of S^T k, then the token blocks of u (wh 0 forms and finishes blocks 0 and 3, wh 1 blocks 1 and 2: five blocks of N and M each).
// Accumulators turn into operands in registers; N and M arrive as the fragments that the lanes need.  Floats enter products as three bf16 parts,
// two floats as the six part products down to 2^-16.
//
// Bound: the chain of chunks, of which a chunk takes about 14000 cycles: S^T k 2700, S^T q 1900, r, N and their exchange 4200, outputs 1800, the update 2500.  Two warps
// a scheduler (a CTA has the shared memory to itself) leave most of that to what products and sums wait for; code is fetched once a chunk, so that shorter
// code is faster than fewer products.  With the tables and a triangular solve per value column in the chain it was 28000.
// All launches in us, that form with dot products alone ahead / now: 4 ragged sequences (4856 tokens, 16 heads of 128 x 128) 455 / 302, 4 x 2048 467 / 326, 32 heads of 64 409 / 273
// and 411 / 314, one sequence of 300 tokens 74 / 51, 8 x 100 62 / 49.  Where there is no room for what is formed ahead, the chain forms it at 13000 cycles a
// chunk; without room then and now: ragged 490 / 492, 4 x 2048 494 / 497, heads of 64 409 / 401 and 411 / 404, 300 tokens 77 / 75, 130 and 20 tokens 47.1 / 46.8, 16 x 40 63 / 61,
// 8 x 100 63 / 66.
//
// Errors against 64 bits over 512 tokens (means of 48 inputs of three sizes, outputs / state; a substitution of floats in the chain, the rows of u rounded to floats, now):
// 128 channels 1.051e-7 / 9.21e-8, 1.049e-7 / 9.23e-8, 1.023e-7 / 8.89e-8; 64 channels 0.998e-7 / 9.21e-8, 0.996e-7 / 9.22e-8, 0.967e-7 / 8.85e-8; keys that point half the
// same way 1.164e-7 / 9.22e-8, 1.171e-7 / 9.37e-8, 1.136e-7 / 8.90e-8; most of it 1.284e-7 / 9.62e-8, 1.303e-7 / 1.003e-7, 1.257e-7 / 9.34e-8; token by token 1.14e-7 /
// 1.05e-7.  What is cut off u costs 14 of 369 us (4 ragged sequences, all launches); what the write scales' products cut off would take 3 % of the states' errors for 3 us more.
constexpr int CK_FS = CK_L + 4;             // padded float rows: a warp's quads fall into distinct banks
constexpr int CK_DELTA_THREADS = 256;

// What a chunk says without the state.  m, n: 16 x 16 blocks (row block i, column block j <= i at i (i + 1) / 2 + j) in three bf16 parts, as the B
// fragments of a lane: rows 8 h + lane / 4, columns 8 w + 2 (lane % 4) at word 2 h + w.
struct DeltaPrep {
  uint4 m[10][3][32], n[10][3][32];
  float ecum[CK_L], beta[CK_L];             // e^(c_i); beta
  float ek[CK_L], eq[CK_L], wk[CK_L];       // e^(c_i) kn; e^(c_i) qn; e^(c_L - c_j) kn
  float kn[CK_L], qn[CK_L];                 // 1 / |k|; scale / |q|
  float wild, pad[3];                       // a key, a query or a scalar of the chunk is out of the split's range
};
static_assert(sizeof(DeltaPrep) % 16 == 0, "copied in 16-byte pieces");
constexpr int CK_DELTA_PREP = sizeof(DeltaPrep) / 4;

struct DeltaWork {                          // scratch of delta_prepare()
  float A[CK_L * CK_FS], E[CK_L * CK_FS];   // A, then N in its blocks on the diagonal; E: e^(c_i - c_j), j <= i, then N below them
  __align__(16) float2 cum[CK_L];           // sums of the log decays: a float and what it leaves
  float beta[CK_L], kn[CK_L], qn[CK_L];
  int wild;
};

__device__ __forceinline__ void pair_sync(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

// Decays and write factors of a chunk, two tokens a lane (zeros behind the portion's end)
struct DeltaCoef { float l[2], b[2]; };
__device__ __forceinline__ DeltaCoef delta_coef(const float* cp, int H, int t0, int len, int lane) {
  DeltaCoef c = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int t = t0 + 2 * lane + e;
    if (t < len) { c.b[e] = cp[static_cast<size_t>(t) * H * 3 + 1]; c.l[e] = cp[static_cast<size_t>(t) * H * 3 + 2]; }
  }
  return c;
}

// The 16 x 16 blocks of the dot products, rows rblk and columns cblk, that warp (wp, wh) has: three for even wp, two for odd ones
__device__ __forceinline__ void delta_block(int wp, int n, int& rblk, int& cblk) {
  const bool extra = wp == 0 && n == 2;                    // warp 0's third block is the first one on the diagonal
  rblk = extra ? 0 : wp == 0 ? 3 : wp == 1 ? 3 : wp == 2 ? 2 : 1;
  cblk = extra ? 0 : (wp == 1 ? 2 : 0) + n;
}
// All of them at once: products of one step of 16 channels for every block, so that none waits for another.  Warps that have two form the second one twice: a branch
// for every step costs more.
template <int D>
__device__ __forceinline__ void delta_block_dots(uint32_t x_u, uint32_t k_u, int wp, int lane, float sc[3][2][4]) {
  constexpr int RB = D * 2;
  const int ra = lane & 15, ca = lane >> 4, rb = (lane >> 4) * 8 + (lane & 7), cb = (lane >> 3) & 1;
  int rblk[3], cblk[3];
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    delta_block(wp, (wp & 1) && n == 2 ? 1 : n, rblk[n], cblk[n]);
#pragma unroll
    for (int w = 0; w < 2; ++w)
#pragma unroll
      for (int e = 0; e < 4; ++e) sc[n][w][e] = 0.f;
  }
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks) {
    uint32_t af[2][4], bf[3][4];
    ldsm4(af[0], x_u + tile_off(rblk[0] * 16 + ra, ks * 2 + ca, RB));       // the first two have the same rows
    ldsm4(af[1], x_u + tile_off(rblk[2] * 16 + ra, ks * 2 + ca, RB));
#pragma unroll
    for (int n = 0; n < 3; ++n) ldsm4(bf[n], k_u + tile_off(cblk[n] * 16 + rb, ks * 2 + cb, RB));
#pragma unroll
    for (int n = 0; n < 3; ++n) {
      mma_add(sc[n][0], af[n >> 1], bf[n][0], bf[n][1]);
      mma_add(sc[n][1], af[n >> 1], bf[n][2], bf[n][3]);
    }
  }
}
// The double of a bf16, by its bits (a conversion takes eight times as long as the addition behind it): right for all normal numbers; zero and what is below 2^-126 come out as
// less than 2^-126.
__device__ __forceinline__ double bf16_double(uint32_t x) { return __hiloint2double(((x & 0x7fffu) << 13) + (896 << 20), 0); }
// 1 / |row| (times the scale for queries) of row tid / 2 of the keys, then of the queries, on the even one of two threads; the largest
// magnitude of what the thread has seen
template <int D>
__device__ __forceinline__ float delta_row_norm(const __nv_bfloat16* k, const __nv_bfloat16* q, int tid, float qscale, uint32_t& m) {
  constexpr int RB = D * 2;
  const int r = tid >> 1;
  const unsigned char* row = reinterpret_cast<const unsigned char*>(r < CK_L ? k : q);
  auto piece = [&](int c) { return *reinterpret_cast<const uint4*>(row + tile_off(r & (CK_L - 1), c * 2 + (tid & 1), RB)); };
  double part[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int c = 0; c < D / 16; ++c) {
    const uint4 x = piece(c);
    m = mag2(mag2(mag2(mag2(m, x.x), x.y), x.z), x.w);
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const double f0 = bf16_double(w[e]), f1 = bf16_double(w[e] >> 16);
      part[e] = fma(f0, f0, part[e]);                      // exact squares: 16 significant bits
      part[e] = fma(f1, f1, part[e]);
    }
  }
  double ss = (part[0] + part[1]) + (part[2] + part[3]);
  ss += __shfl_xor_sync(0xffffffffu, ss, 1);
  const uint32_t both = __vmaxu2(m, __shfl_xor_sync(0xffffffffu, m, 1));
  if (max(both & 0xffffu, both >> 16) >= CK_BIG_IN) {      // infinities and what overflows a float's square reach the token-by-token sums as they always did
    ss = 0.0;
    for (int c = 0; c < D / 16; ++c) {
      const uint4 x = piece(c);
      const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        ss += static_cast<double>(bf16lo(w[e]) * bf16lo(w[e]));
        ss += static_cast<double>(bf16hi(w[e]) * bf16hi(w[e]));
      }
    }
    ss += __shfl_xor_sync(3u << (tid & 30), ss, 1);
    return static_cast<float>((r < CK_L ? 1.0 : static_cast<double>(qscale)) / sqrt(ss + 1e-6));
  }
  // the root's reciprocal to 2^-43: a float's and one Newton step
  ss += 1e-6;
  const double y = rsqrtf(static_cast<float>(ss)), z = fma(0.5 * y, fma(-ss * y, y, 1.0), y);
  return static_cast<float>(r < CK_L ? z : qscale * z);
}

// All 256 threads; keys and queries of the chunk that starts at token t0 in shared memory.  Ends without a barrier.
//
// N in blocks of 16: those on the diagonal by substitution (column c of (1 + A)^-1 solves the system for the unit vector c), those below from them by
// products, 64 threads a block with four neighbouring sums each.  Sums are formed beside the rows: a row is rounded once at its own size and not up to 64 times.
template <int D>
__device__ __forceinline__ void delta_prepare(const ScanArgs& a, const __nv_bfloat16* q_s, const __nv_bfloat16* k_s, DeltaCoef coef, int L, DeltaWork& w, DeltaPrep& p) {
  const int blocks = (L + 15) >> 4;                        // rows of blocks that the portion reaches: nobody asks for those behind them
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wp = warp & 3, wh = warp >> 2, g4 = lane >> 2, c2 = 2 * (lane & 3);
  if (tid == 0) w.wild = 0;
  float ecum[2], wl[2];
  if (warp == 0) {                                         // lane l: tokens 2 l, 2 l + 1
    float *l = coef.l, *b = coef.b;
    const bool fine = fabsf(l[0]) < 1e30f && fabsf(l[1]) < 1e30f && fabsf(b[0]) < 1e6f && fabsf(b[1]) < 1e6f;
    l[0] = cut_log(l[0]); l[1] = cut_log(l[1]);
    double c1 = static_cast<double>(l[0]) + l[1], x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      x = __shfl_up_sync(0xffffffffu, c1, o);
      if (lane >= o) c1 += x;
    }
    double c0 = __shfl_up_sync(0xffffffffu, c1, 1);
    c0 = (lane == 0 ? 0.0 : c0) + l[0];
    const double ce = __shfl_sync(0xffffffffu, c1, 31);
    const float h0 = static_cast<float>(c0), h1 = static_cast<float>(c1);
    *reinterpret_cast<float4*>(w.cum + 2 * lane) = make_float4(h0, static_cast<float>(c0 - h0), h1, static_cast<float>(c1 - h1));
    w.beta[2 * lane] = b[0]; w.beta[2 * lane + 1] = b[1];
    ecum[0] = exp_sum(c0); ecum[1] = exp_sum(c1);
    wl[0] = exp_sum(ce - c0); wl[1] = exp_sum(ce - c1);
    if (!fine) w.wild = 1;                                 // behind lane 0's zero: the shuffles lie between
  }
  uint32_t m = 0;
  const float nrm = delta_row_norm<D>(k_s, q_s, tid, a.qscale, m);
  if ((tid & 1) == 0) (tid < 2 * CK_L ? w.kn[tid >> 1] : w.qn[(tid >> 1) - CK_L]) = nrm;
  const int wild = __syncthreads_or((m & 0xffffu) >= CK_BIG_IN || (m >> 16) >= CK_BIG_IN);
  // ---- decays between the chunk's tokens: the 36 tiles of 8 x 8 up to the diagonal, nine for each 64 threads, none waiting for another
#pragma unroll
  for (int x = 0; x < 9; ++x) {
    const int tile = ck_tile((tid >> 6) + 4 * x), i = (tile >> 3) * 8 + ((tid >> 3) & 7), j = (tile & 7) * 8 + (tid & 7);
    if ((tile >> 4) < blocks) w.E[i * CK_FS + j] = exp_between(w.cum[i], w.cum[j]);
  }
  if (warp == 0) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int i = 2 * lane + e;
      p.ecum[i] = ecum[e]; p.beta[i] = w.beta[i];
      p.ek[i] = ecum[e] * w.kn[i]; p.eq[i] = ecum[e] * w.qn[i]; p.wk[i] = wl[e] * w.kn[i];
      p.kn[i] = w.kn[i]; p.qn[i] = w.qn[i];
    }
  }
  if (tid == 0) { p.wild = wild || w.wild ? 1.f : 0.f; p.pad[0] = p.pad[1] = p.pad[2] = 0.f; }
  __syncthreads();
  // ---- dot products of the keys (wh 0) or the queries (wh 1) with the keys up to the diagonal, in 16 x 16 blocks
  const uint32_t k_u = smem_u32(k_s), x_u = wh ? smem_u32(q_s) : k_u;
  float dots[3][2][4];
  if ((wp == 0 ? 0 : wp == 1 ? 3 : wp == 2 ? 2 : 1) < blocks) delta_block_dots<D>(x_u, k_u, wp, lane, dots);
#pragma unroll
  for (int nb = 0; nb < 3; ++nb) {
    if (nb == 2 && (wp & 1)) break;
    int rblk, cblk;
    delta_block(wp, nb, rblk, cblk);
    if (rblk >= blocks) continue;
    const float (&sc)[2][4] = dots[nb];
    uint32_t part[3][4];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int i = rblk * 16 + g4 + 8 * half;
      const float fi = wh ? w.qn[i] : w.beta[i] * w.kn[i];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int j = cblk * 16 + c * 8 + c2;
        const float2 e2 = *reinterpret_cast<const float2*>(w.E + i * CK_FS + j), k2 = *reinterpret_cast<const float2*>(w.kn + j);
        const bool in0 = wh ? j <= i : j < i, in1 = wh ? j + 1 <= i : j + 1 < i;
        const float x = in0 ? sc[c][2 * half] * (e2.x * (fi * k2.x)) : 0.f, y = in1 ? sc[c][2 * half + 1] * (e2.y * (fi * k2.y)) : 0.f;
        if (wh) split3(x, y, part[0][2 * half + c], part[1][2 * half + c], part[2][2 * half + c]);
        else *reinterpret_cast<float2*>(w.A + i * CK_FS + j) = make_float2(x, y);
      }
    }
    if (wh) {
#pragma unroll
      for (int e = 0; e < 3; ++e) p.m[rblk * (rblk + 1) / 2 + cblk][e][lane] = make_uint4(part[e][0], part[e][1], part[e][2], part[e][3]);
    }
  }
  // ---- N of the 16 x 16 blocks on the diagonal, a warp each, in place of A's; a lane has a column (the upper half of the lanes the same ones)
  if (wh == 0) {
    asm volatile("bar.sync 1, 128;" ::: "memory");         // A is there; the other four warps are still at M
    if (warp < blocks) {
      float* A = w.A + warp * 16 * (CK_FS + 1);
      float n[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) n[i] = 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) {                       // row j is complete: n[j], and u = (the unit vector's entry) - n[j] for the rows behind
        const float u = (j == (lane & 15) ? 1.f : 0.f) - n[j];
#pragma unroll
        for (int i = j + 1; i < 16; ++i) n[i] = fmaf(A[i * CK_FS + j], u, n[i]);
      }
      __syncwarp();
      if (lane < 16)
#pragma unroll
        for (int i = 0; i < 16; ++i) A[i * CK_FS + lane] = n[i];
    }
  }
  __syncthreads();
  // ---- the blocks below, a diagonal of them at a time: X_ij = A_ij (1 - N_jj) - sum_(j < k < i) A_ik N_kj (kept in the mirrored block), N_ij = X_ij - N_ii X_ij
  {
    const int grp = tid >> 6, row = (tid >> 2) & 15, col = 4 * (tid & 3);
    auto product = [&](const float* x, const float* y) -> float4 {     // row of x times four columns of y
      float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
      auto add = [](float4& s, float f, const float4& v) { s.x = fmaf(f, v.x, s.x); s.y = fmaf(f, v.y, s.y); s.z = fmaf(f, v.z, s.z); s.w = fmaf(f, v.w, s.w); };
      auto line = [&](int t) { return *reinterpret_cast<const float4*>(y + t * CK_FS + col); };
#pragma unroll
      for (int t = 0; t < 16; t += 4) {
        const float4 a4 = *reinterpret_cast<const float4*>(x + row * CK_FS + t);
        add(s0, a4.x, line(t));
        add(s1, a4.y, line(t + 1));
        add(s0, a4.z, line(t + 2));
        add(s1, a4.w, line(t + 3));
      }
      return make_float4(s0.x + s1.x, s0.y + s1.y, s0.z + s1.z, s0.w + s1.w);
    };
    auto block = [](float* x, int i, int j) { return x + 16 * i * CK_FS + 16 * j; };
    auto at = [&](float* x) -> float4& { return *reinterpret_cast<float4*>(x + row * CK_FS + col); };
    auto less = [](const float4& x, const float4& y) { return make_float4(x.x - y.x, x.y - y.y, x.z - y.z, x.w - y.w); };
#pragma unroll 1
    for (int d = 1; d < 4; ++d) {
      if (d >= blocks) break;
      const int j = grp, i = grp + d;                      // the group's block of the diagonal
      if (i < blocks) {
        float4 s = product(block(w.A, i, j), block(w.A, j, j));
#pragma unroll 1
        for (int x = 1; x < d; ++x) {
          const float4 y = product(block(w.A, i, j + x), block(w.E, j + x, j));
          s.x += y.x; s.y += y.y; s.z += y.z; s.w += y.w;
        }
        const float4 x = less(at(block(w.A, i, j)), s);
        at(block(w.E, j, i)) = x;
        if (grp == 0) asm volatile("bar.sync 2, 64;" ::: "memory");      // two warps have a block; numbers as constants, of which a CTA then takes few
        else if (grp == 1) asm volatile("bar.sync 3, 64;" ::: "memory");
        else asm volatile("bar.sync 4, 64;" ::: "memory");
        at(block(w.E, i, j)) = less(x, product(block(w.A, i, i), block(w.E, j, i)));
      }
      __syncthreads();
    }
  }
  for (int blk = warp; blk < 10; blk += 8) {
    const int ib = blk >= 6 ? 3 : blk >= 3 ? 2 : blk >= 1 ? 1 : 0, jb = blk - ib * (ib + 1) / 2;
    if (ib >= blocks) break;
    const float* N = ib == jb ? w.A : w.E;
    uint32_t part[3][4];
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int i = ib * 16 + half * 8 + g4, j = jb * 16 + c * 8 + c2;
        const float x = j < i ? N[i * CK_FS + j] : 0.f, y = j + 1 < i ? N[i * CK_FS + j + 1] : 0.f;
        split3(x, y, part[0][2 * half + c], part[1][2 * half + c], part[2][2 * half + c]);
      }
#pragma unroll
    for (int e = 0; e < 3; ++e) p.n[blk][e][lane] = make_uint4(part[e][0], part[e][1], part[e][2], part[e][3]);
  }
}

template <int D> struct DeltaAheadTiles {
  __nv_bfloat16 q[CK_L * D], k[CK_L * D];
  DeltaWork work;
};
template <int D>
__global__ void __launch_bounds__(CK_DELTA_THREADS, 3)
delta_prepare_kernel(const ScanArgs a) {
  constexpr int RB = D * 2;
  extern __shared__ __align__(128) unsigned char ck_smem[];
  DeltaAheadTiles<D>& sm = *reinterpret_cast<DeltaAheadTiles<D>*>(ck_smem);
  const int b = blockIdx.z, h = blockIdx.y, t0 = blockIdx.x * CK_L, len = a.seq_len[b];
  if (len < a.min_len || t0 >= len) return;
  const int tid = threadIdx.x, g = h / (a.H / a.G);
  const int64_t start = a.seq_start[b];
  const __nv_bfloat16* qg = static_cast<const __nv_bfloat16*>(a.q) + start * a.ldq + static_cast<size_t>(g) * D;
  const __nv_bfloat16* kg = static_cast<const __nv_bfloat16*>(a.k) + start * a.ldk + static_cast<size_t>(g) * D;
  for (int idx = tid; idx < CK_L * (D / 8); idx += CK_DELTA_THREADS) {
    const int j = idx / (D / 8), ch = idx % (D / 8);
    const bool ok = t0 + j < len;
    const size_t row = ok ? t0 + j : 0;
    cp_async_16(reinterpret_cast<unsigned char*>(sm.q) + tile_off(j, ch, RB), qg + row * a.ldq + ch * 8, ok);
    cp_async_16(reinterpret_cast<unsigned char*>(sm.k) + tile_off(j, ch, RB), kg + row * a.ldk + ch * 8, ok);
  }
  cp_async_commit();
  DeltaCoef coef = {};
  if (tid < 32) coef = delta_coef(a.coef + (start * a.H + h) * 3, a.H, t0, len, tid);
  const int64_t number = static_cast<int64_t>(chunks_before(a.seq_len, b, tid & 31) + t0 / CK_L) * a.H + h;
  cp_async_wait<0>();
  __syncthreads();
  delta_prepare<D>(a, sm.q, sm.k, coef, min(CK_L, len - t0), sm.work, reinterpret_cast<DeltaPrep*>(a.scores)[number]);
}

template <int D, bool AHEAD> struct DeltaTiles {
  __nv_bfloat16 q[2][CK_L * D], k[2][CK_L * D], v[2][CK_L * CK_P];
  DeltaPrep prep[AHEAD ? 2 : 1];
  float4 part[8][8][32];                    // [warp][8 tokens]: S^T k over the warp's channels; u of its blocks and what was cut off it lie over it
  float4 other[8][4][32];                   // [warp]: S^T q of the partner's blocks
  union {
    float red[2][2][2][CK_P];               // token by token: [parity][k or q][half][value column]
    typename std::conditional<AHEAD, char, DeltaWork>::type work;
  };
};

// t = x n over the blocks jb <= ib of row block ib: x in three parts per column block, n the fragments of a row of blocks; t = small + big
__device__ __forceinline__ void delta_row_product(float small[2][4], float big[2][4], const uint32_t x[4][3][4], const uint4 (*n)[3][32], int ib, int lane) {
  float mid[2][4];
#pragma unroll
  for (int w = 0; w < 2; ++w)
#pragma unroll
    for (int e = 0; e < 4; ++e) small[w][e] = mid[w][e] = big[w][e] = 0.f;
#pragma unroll
  for (int jb = 0; jb < 4; ++jb) {
    if (jb <= ib) {
      const uint4 (*f)[32] = n[ib * (ib + 1) / 2 + jb];
      const uint4 b0 = f[0][lane], b1 = f[1][lane], b2 = f[2][lane];
      // products that add to the same sums lie as far from one another as their order allows.  The large ones by themselves, with what the tensor
      // core cut off their sum (it keeps two bits behind a float's): the same products on top of minus the sum
      const auto pair = [&](float c[2][4], int part, const uint4& b) {
        mma_bf16_16816(c[0], x[jb][part], b.x, b.y);
        mma_bf16_16816(c[1], x[jb][part], b.z, b.w);
      };
      float t[2][4] = {}, r[2][4];
      pair(t, 0, b0);
      pair(small, 2, b0);
      pair(mid, 1, b0);
#pragma unroll
      for (int w = 0; w < 2; ++w)
#pragma unroll
        for (int e = 0; e < 4; ++e) r[w][e] = -t[w][e];
      pair(small, 0, b2);
      pair(r, 0, b0);
      pair(mid, 0, b1);
      pair(small, 1, b1);
#pragma unroll
      for (int w = 0; w < 2; ++w)
#pragma unroll
        for (int e = 0; e < 4; ++e) big[w][e] = (big[w][e] + r[w][e]) + t[w][e];
    }
  }
#pragma unroll
  for (int w = 0; w < 2; ++w)
#pragma unroll
    for (int e = 0; e < 4; ++e) small[w][e] += mid[w][e];
}
// c += x n
__device__ __forceinline__ void delta_add_row(float c[2][4], const uint32_t x[4][3][4], const uint4 (*n)[3][32], int ib, int lane) {
  float small[2][4], big[2][4];
  delta_row_product(small, big, x, n, ib, lane);
#pragma unroll
  for (int w = 0; w < 2; ++w)
#pragma unroll
    for (int e = 0; e < 4; ++e) c[w][e] += small[w][e] + big[w][e];
}
// c -= x n; rest: what the two roundings of that cut off, which joins the last parts of c where it enters products (bf16 as they are, with bits to spare).  Rounded to
// floats, each with an error of its own, the rows of u left states up to 4 % further from 64 bits than a substitution, whose rows take up the errors of those in front.
__device__ __forceinline__ void delta_take_row(float c[2][4], uint32_t rest[2][2], const uint32_t x[4][3][4], const uint4 (*n)[3][32], int ib, int lane) {
  float small[2][4], big[2][4];
  delta_row_product(small, big, x, n, ib, lane);
#pragma unroll
  for (int w = 0; w < 2; ++w)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float cut[2];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        float& y = c[w][2 * h + x];
        const float sm = small[w][2 * h + x], bg = big[w][2 * h + x], t = sm + bg, u = y - t, v = u - y;
        cut[x] = ((y - (u - v)) - (t + v)) - (sm - (t - bg));
        y = u;
      }
      rest[w][h] = pack_bf16(cut[0], cut[1]);
    }
}

// AHEAD: delta_prepare_kernel has run
template <int D, bool AHEAD>
__global__ void __launch_bounds__(CK_DELTA_THREADS, 1)
delta_chunk_kernel(const ScanArgs a) {
  using Sm = DeltaTiles<D, AHEAD>;
  constexpr int RB = D * 2, VB = CK_P * 2, THREADS = CK_DELTA_THREADS, CH = D / 2, NT = CH / 8;
  extern __shared__ __align__(128) unsigned char ck_smem[];
  Sm& sm = *reinterpret_cast<Sm*>(ck_smem);
  const int b = blockIdx.z, h = blockIdx.y, p0 = blockIdx.x * CK_P;
  const int len = a.seq_len[b];
  if (len < a.min_len) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wp = warp & 3, wh = warp >> 2, g4 = lane >> 2, c2 = 2 * (lane & 3);
  const int H = a.H, dv = a.dv, g = h / (H / a.G);
  const size_t start = a.seq_start[b];
  using B = __nv_bfloat16;
  const B* qg = static_cast<const B*>(a.q) + start * a.ldq + static_cast<size_t>(g) * D;
  const B* kg = static_cast<const B*>(a.k) + start * a.ldk + static_cast<size_t>(g) * D;
  const B* vg = static_cast<const B*>(a.v) + start * a.ldv + static_cast<size_t>(h) * dv + p0;
  const float* cp = a.coef + (start * H + h) * 3;
  float* Sg = a.state + (static_cast<size_t>(a.seq_slot[b]) * H + h) * D * dv + p0;
  float* og = a.out + start * H * dv + static_cast<size_t>(h) * dv + p0;
  const DeltaPrep* pg = nullptr;                           // the sequence's first chunk; one chunk is H of them
  if constexpr (AHEAD) pg = reinterpret_cast<const DeltaPrep*>(a.scores) + static_cast<int64_t>(chunks_before(a.seq_len, b, lane)) * H + h;
  auto load_chunk = [&](int t0, int s) {
    for (int idx = tid; idx < CK_L * (D / 8); idx += THREADS) {
      const int j = idx / (D / 8), ch = idx % (D / 8);
      const bool ok = t0 + j < len;
      const size_t row = ok ? t0 + j : 0;
      cp_async_16(reinterpret_cast<unsigned char*>(sm.q[s]) + tile_off(j, ch, RB), qg + row * a.ldq + ch * 8, ok);
      cp_async_16(reinterpret_cast<unsigned char*>(sm.k[s]) + tile_off(j, ch, RB), kg + row * a.ldk + ch * 8, ok);
    }
    for (int idx = tid; idx < CK_L * (CK_P / 8); idx += THREADS) {
      const int j = idx / (CK_P / 8), ch = idx % (CK_P / 8);
      const bool ok = t0 + j < len;
      cp_async_16(reinterpret_cast<unsigned char*>(sm.v[s]) + tile_off(j, ch, VB), vg + (ok ? t0 + j : 0) * a.ldv + ch * 8, ok);
    }
    if constexpr (AHEAD) {
      const uint4* src = reinterpret_cast<const uint4*>(pg + static_cast<int64_t>(t0 / CK_L) * H);
      for (int i = tid; i < CK_DELTA_PREP / 4; i += THREADS) cp_async_16(reinterpret_cast<uint4*>(&sm.prep[s]) + i, src + i, true);
    }
  };
  load_chunk(0, 0);
  cp_async_commit();
  DeltaCoef coef = {};                                     // of the next chunk, where the chain prepares it
  if (!AHEAD && warp == 0) coef = delta_coef(cp, H, 0, len, lane);
  const int pr = wp * 16 + g4, n0 = wh * CH;               // S^T fragments: value columns pr (+ 8), key channels n0 + nt * 8 + c2 (+ 1)
  float S[NT][4];
  const bool carried = a.seq_pos0[b] > 0;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) S[nt][e] = carried ? Sg[static_cast<size_t>(n0 + nt * 8 + c2 + (e & 1)) * dv + pr + 8 * (e >> 1)] : 0.f;
  const int rb = (lane >> 4) * 8 + (lane & 7), cb = (lane >> 3) & 1;
  const int rt = ((lane >> 3) & 1) * 8 + (lane & 7), ct = lane >> 4;
  for (int t0 = 0, s = 0; t0 < len; t0 += CK_L, s ^= 1) {
    const int L = min(CK_L, len - t0);
    cp_async_wait<0>();
    // ---- the range of what this thread has copied and of its part of the state
    bool wild = false;
    {
      uint32_t m = 0;
      for (int idx = tid; idx < CK_L * (CK_P / 8); idx += THREADS) {
        const uint4 x = *reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned char*>(sm.v[s]) + tile_off(idx / (CK_P / 8), idx % (CK_P / 8), VB));
        m = mag2(mag2(mag2(mag2(m, x.x), x.y), x.z), x.w);
      }
      wild = (m & 0xffffu) >= CK_BIG_IN || (m >> 16) >= CK_BIG_IN;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) wild = wild || !(fabsf(S[nt][e]) < CK_BIG_STATE);
    }
    wild = __syncthreads_or(wild);                         // the chunk has landed; the previous one is consumed
    if constexpr (!AHEAD) {
      delta_prepare<D>(a, sm.q[s], sm.k[s], coef, L, sm.work, sm.prep[0]);
      if (warp == 0) coef = delta_coef(cp, H, t0 + CK_L, len, lane);
      __syncthreads();
    }
    const DeltaPrep& pre = sm.prep[AHEAD ? s : 0];
    wild = wild || pre.wild != 0.f;
    if (t0 + CK_L < len) load_chunk(t0 + CK_L, s ^ 1);
    cp_async_commit();
    if (wild) {
      // ---- token by token: the same sums, every product in float
      for (int i = 0; i < L; ++i) {
        const float* c = cp + static_cast<size_t>(t0 + i) * H * 3;
        const float c0 = c[0], c1 = c[1], kn = pre.kn[i];
        float (*red)[2][CK_P] = sm.red[i & 1];
        float x0 = 0.f, x1 = 0.f;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float kk = to_f(sm.k[s][tile_off(i, n0 / 8 + nt, RB) / 2 + c2 + e]);
            S[nt][e] *= c0;     x0 += S[nt][e] * kk;
            S[nt][e + 2] *= c0; x1 += S[nt][e + 2] * kk;
          }
#pragma unroll
        for (int x = 1; x < 4; x <<= 1) { x0 += __shfl_xor_sync(0xffffffffu, x0, x); x1 += __shfl_xor_sync(0xffffffffu, x1, x); }
        if ((lane & 3) == 0) { red[0][wh][pr] = x0; red[0][wh][pr + 8] = x1; }
        __syncthreads();
        const float v0 = to_f(sm.v[s][tile_off(i, pr >> 3, VB) / 2 + (pr & 7)]), v1 = to_f(sm.v[s][tile_off(i, (pr + 8) >> 3, VB) / 2 + (pr & 7)]);
        const float w0 = c1 * (v0 - (red[0][0][pr] + red[0][1][pr]) * kn) * kn, w1 = c1 * (v1 - (red[0][0][pr + 8] + red[0][1][pr + 8]) * kn) * kn;
        x0 = x1 = 0.f;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const uint32_t off = tile_off(i, n0 / 8 + nt, RB) / 2 + c2 + e;
            const float kk = to_f(sm.k[s][off]), qq = to_f(sm.q[s][off]);
            S[nt][e] += kk * w0;     x0 += S[nt][e] * qq;
            S[nt][e + 2] += kk * w1; x1 += S[nt][e + 2] * qq;
          }
#pragma unroll
        for (int x = 1; x < 4; x <<= 1) { x0 += __shfl_xor_sync(0xffffffffu, x0, x); x1 += __shfl_xor_sync(0xffffffffu, x1, x); }
        if ((lane & 3) == 0) { red[1][wh][pr] = x0; red[1][wh][pr + 8] = x1; }
        __syncthreads();
        if (tid < CK_P) og[static_cast<size_t>(t0 + i) * H * dv + tid] = (red[1][0][tid] + red[1][1][tid]) * pre.qn[i];
      }
      continue;
    }
    const uint32_t q_u = smem_u32(sm.q[s]), k_u = smem_u32(sm.k[s]), v_u = smem_u32(sm.v[s]);
    const bool front = carried || t0 > 0;
    // ---- S^T k, then S^T q over this half of the channels, the small parts first
    float oq[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) oq[nt][e] = 0.f;
    if (front) {
      uint32_t part[3][CH / 16][4];
#pragma unroll
      for (int ks = 0; ks < CH / 16; ++ks)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          split3(S[2 * ks + (e >> 1)][2 * (e & 1)], S[2 * ks + (e >> 1)][2 * (e & 1) + 1], part[0][ks][e], part[1][ks][e], part[2][ks][e]);
      // sums are added to every eight products, so that none waits for the one in front of it; all 64 tokens, however many there are (zeros behind the last one): code for
      // fewer of them costs every chunk more, by what has to be fetched, than it saves the last one
      auto against = [&](uint32_t x_u, float c[8][4]) {
        constexpr int NP = CK_L / 16;
#pragma unroll
        for (int pass = 0; pass < 2; ++pass)
#pragma unroll
          for (int ks = 0; ks < CH / 16; ++ks) {
            uint32_t bf[NP][4];
#pragma unroll
            for (int np = 0; np < NP; ++np) ldsm4(bf[np], x_u + tile_off(np * 16 + rb, n0 / 8 + ks * 2 + cb, RB));
            if (pass == 0) {
#pragma unroll
              for (int y = 2; y > 0; --y)
#pragma unroll
                for (int np = 0; np < NP; ++np) {
                  mma_bf16_16816(c[2 * np], part[y][ks], bf[np][0], bf[np][1]);
                  mma_bf16_16816(c[2 * np + 1], part[y][ks], bf[np][2], bf[np][3]);
                }
            } else {
              float t[2 * NP][4] = {};
#pragma unroll
              for (int np = 0; np < NP; ++np) {
                mma_bf16_16816(t[2 * np], part[0][ks], bf[np][0], bf[np][1]);
                mma_bf16_16816(t[2 * np + 1], part[0][ks], bf[np][2], bf[np][3]);
              }
#pragma unroll
              for (int x = 0; x < 2 * NP; ++x)
#pragma unroll
                for (int e = 0; e < 4; ++e) c[x][e] += t[x][e];
            }
          }
      };
      float ok[8][4];
#pragma unroll
      for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) ok[nt][e] = 0.f;
      against(k_u, ok);
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) sm.part[warp][nt][lane] = make_float4(ok[nt][0], ok[nt][1], ok[nt][2], ok[nt][3]);
      against(q_u, oq);
    } else {
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) sm.part[warp][nt][lane] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int x = 0; x < 4; ++x) {                          // the partner's token blocks
      const float* y = wh ? oq[x < 2 ? x : 4 + x] : oq[2 + x];
      sm.other[warp][x][lane] = make_float4(y[0], y[1], y[2], y[3]);
    }
    pair_sync(1 + wp);
    // ---- what the chunk has to write before its tokens see one another
    float r[8][4];                                         // r, then u
    {
      uint32_t vf[4][4];
#pragma unroll
      for (int js = 0; js < 4; ++js) ldsm4t(vf[js], v_u + tile_off(js * 16 + rb, wp * 2 + cb, VB));
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        const float4 x = sm.part[wp][nt][lane], y = sm.part[wp + 4][nt][lane];
        const float2 be = *reinterpret_cast<const float2*>(pre.beta + nt * 8 + c2), ek = *reinterpret_cast<const float2*>(pre.ek + nt * 8 + c2);
        const uint32_t v0 = vf[nt >> 1][2 * (nt & 1)], v1 = vf[nt >> 1][2 * (nt & 1) + 1];
        r[nt][0] = be.x * (bf16lo(v0) - ek.x * (x.x + y.x)); r[nt][1] = be.y * (bf16hi(v0) - ek.y * (x.y + y.y));
        r[nt][2] = be.x * (bf16lo(v1) - ek.x * (x.z + y.z)); r[nt][3] = be.y * (bf16hi(v1) - ek.y * (x.w + y.w));
      }
    }
    // ---- u = r - N r, this warp's two token blocks
    uint32_t xf[4][3][4];
    auto split_all = [&](auto rest) {
#pragma unroll
      for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = 2 * (nt & 1) + h;
          split3(r[nt][2 * h], r[nt][2 * h + 1], xf[nt >> 1][0][e], xf[nt >> 1][1][e], xf[nt >> 1][2][e]);
          rest(nt, h, xf[nt >> 1][2][e]);
        }
    };
    split_all([](int, int, uint32_t&) {});
    uint32_t rest[4][2] = {};                              // what was cut off u
    if (wh == 0) {
      delta_take_row(r + 0, rest + 0, xf, pre.n, 0, lane);
      if (48 < L) delta_take_row(r + 6, rest + 2, xf, pre.n, 3, lane);
    } else {
      if (16 < L) delta_take_row(r + 2, rest + 0, xf, pre.n, 1, lane);
      if (32 < L) delta_take_row(r + 4, rest + 2, xf, pre.n, 2, lane);
    }
    pair_sync(1 + wp);                                     // both have read the sums that u takes the place of
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float* y = wh ? r[2 + x] : r[x < 2 ? x : 4 + x];
      sm.part[warp][x][lane] = make_float4(y[0], y[1], y[2], y[3]);
    }
    uint4* cut_s = reinterpret_cast<uint4*>(sm.part[warp][4]);
    cut_s[lane] = make_uint4(rest[0][0], rest[0][1], rest[1][0], rest[1][1]);
    cut_s[32 + lane] = make_uint4(rest[2][0], rest[2][1], rest[3][0], rest[3][1]);
    pair_sync(1 + wp);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float4 y = sm.part[warp ^ 4][x][lane];
      float* z = wh ? r[x < 2 ? x : 4 + x] : r[2 + x];
      z[0] = y.x; z[1] = y.y; z[2] = y.z; z[3] = y.w;
    }
    // what was cut off u for eight tokens (row h of the lane's two), by the warp of the pair that formed it
    auto cut_off = [&](int nt, int h) {
      const bool second = nt >= 2 && nt < 6;
      const int x = second ? nt - 2 : nt < 2 ? nt : nt - 4;
      return reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint4*>(sm.part[second ? wp + 4 : wp][4]) + (x >> 1) * 32 + lane)[2 * (x & 1) + h];
    };
    split_all([&](int nt, int h, uint32_t& lo) { lo = add_bf16x2(lo, cut_off(nt, h)); });
    // ---- the outputs of this warp's blocks
    {
      auto finish = [&](int ib, float* const c0, float* const c1) {
        float c[2][4];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          const float* y = w ? c1 : c0;
          const float4 x = sm.other[warp ^ 4][(wh ? (ib - 1) : (ib ? 1 : 0)) * 2 + w][lane];
          const float2 eq = *reinterpret_cast<const float2*>(pre.eq + ib * 16 + w * 8 + c2);
          c[w][0] = (y[0] + x.x) * eq.x; c[w][1] = (y[1] + x.y) * eq.y; c[w][2] = (y[2] + x.z) * eq.x; c[w][3] = (y[3] + x.w) * eq.y;
        }
        delta_add_row(c, xf, pre.m, ib, lane);
#pragma unroll
        for (int w = 0; w < 2; ++w)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = ib * 16 + w * 8 + c2 + (e & 1), p = pr + 8 * (e >> 1);
            if (i < L) og[static_cast<size_t>(t0 + i) * H * dv + p] = c[w][e];
          }
      };
      if (wh == 0) {
        finish(0, oq[0], oq[1]);
        if (48 < L) finish(3, oq[6], oq[7]);
      } else {
        if (16 < L) finish(1, oq[2], oq[3]);
        if (32 < L) finish(2, oq[4], oq[5]);
      }
    }
    // ---- the state behind the chunk, this half of the channels: what the chunk adds is summed by itself, then S <- e^(c_L) S + sum
    {
      uint32_t off[8][2];
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        const float2 wk = *reinterpret_cast<const float2*>(pre.wk + nt * 8 + c2);
        const uint32_t w2 = pack_bf16(wk.x, wk.y);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          r[nt][2 * h] *= wk.x; r[nt][2 * h + 1] *= wk.y;
          off[nt][h] = mul_bf16x2(cut_off(nt, h), w2);
        }
      }
      split_all([&](int nt, int h, uint32_t& lo) { lo = add_bf16x2(lo, off[nt][h]); });
      const float gl = pre.ecum[CK_L - 1];
      constexpr int JS = CK_L / 16;
#pragma unroll
      for (int np = 0; np < CH / 16; np += 2) {
        float t[4][4] = {};
        uint32_t bf[JS][2][4];
#pragma unroll
        for (int js = 0; js < JS; ++js)
#pragma unroll
          for (int h = 0; h < 2; ++h) ldsm4t(bf[js][h], k_u + tile_off(js * 16 + rt, n0 / 8 + (np + h) * 2 + ct, RB));
#pragma unroll
        for (int part = 2; part > 0; --part)
#pragma unroll
          for (int js = 0; js < JS; ++js)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              mma_bf16_16816(t[2 * h], xf[js][part], bf[js][h][0], bf[js][h][1]);
              mma_bf16_16816(t[2 * h + 1], xf[js][part], bf[js][h][2], bf[js][h][3]);
            }
#pragma unroll
        for (int js = 0; js < JS; ++js) {
          float y[4][4] = {};
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            mma_bf16_16816(y[2 * h], xf[js][0], bf[js][h][0], bf[js][h][1]);
            mma_bf16_16816(y[2 * h + 1], xf[js][0], bf[js][h][2], bf[js][h][3]);
          }
#pragma unroll
          for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int e = 0; e < 4; ++e) t[x][e] += y[x][e];
        }
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int e = 0; e < 4; ++e) S[2 * np + x][e] = fmaf(gl, S[2 * np + x][e], t[x][e]);
      }
    }
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) Sg[static_cast<size_t>(n0 + nt * 8 + c2 + (e & 1)) * dv + pr + 8 * (e >> 1)] = S[nt][e];
}

bool scan_chunk_applies(const ScanArgs& a) {
  return (a.d == 64 || a.d == 128) && a.dv % CK_P == 0 && a.ldq % 8 == 0 && a.ldk % 8 == 0 && a.ldv % 8 == 0 && aligned16(a.q) &&
         aligned16(a.k) && aligned16(a.v) && a.head_decay == nullptr && !a.divide;
}

// The longest portion that is left to the token-by-token kernel.  A chunk costs the same whatever the portion's length, a token of the
// other kernel the same whatever its place, so each size has one crossing; it lies elsewhere while the CTAs are fewer than the
// multiprocessors (both kernels wait for their own chain) than above (both wait for their turn), and a little earlier for a portion
// that is alone in its step, where no second kernel looks for short ones.  Token by token / in chunks, us, behind and in front of the
// lines (portions x tokens); over 588 such steps the choice is within 5 % of the better kernel:
//   state space   128 channels, 64 heads    1 x 24 20 / 17    4 x 14 28 / 22    16 x 14 67 / 68    64 x 14 269 / 235    64 x 10 208 / 233
//                 64 channels, 32 heads     64 x 24 90 / 80   64 x 18 73 / 80
//   delta rule    128 channels, 16 heads    8 x 24 50 / 38    16 x 24 76 / 69    64 x 24 258 / 244    64 x 20 217 / 241
//                 64 channels, 32 heads     16 x 48 67 / 61   64 x 48 228 / 208  64 x 32 156 / 192
static int64_t chunk_ctas(const ScanArgs& a, int n_seqs) { return static_cast<int64_t>(n_seqs) * a.H * (a.dv / CK_P); }
int linear_walk_len(const ScanArgs& a, int n_seqs) {
  const int64_t ctas = chunk_ctas(a, n_seqs), sms = sm_count();
  if (a.d == 128) return ctas <= sms ? (n_seqs == 1 ? 20 : 24) : ctas <= 2 * sms ? 10 : 12;
  return ctas <= sms ? (n_seqs == 1 ? 22 : 26) : 20;
}
int delta_walk_len(const ScanArgs& a, int n_seqs) {
  const int64_t ctas = chunk_ctas(a, n_seqs), sms = sm_count();
  if (a.d == 128) return ctas <= sms ? 19 : ctas <= 2 * sms ? 16 : 21;
  return ctas <= sms ? (n_seqs == 1 ? 24 : 28) : 40;
}

int64_t chunk_scores_floats(int n_tokens, int n_seqs, int G) {
  return (static_cast<int64_t>(n_tokens) / CK_L + n_seqs + 1) * G * (CK_SCORES + 1);
}

template <int D, bool AHEAD>
static int go_linear(const char* what, const ScanArgs& a, int n_seqs, int longest, int64_t chunks, cudaStream_t st) {
  constexpr int smem = static_cast<int>(sizeof(ChunkTiles<D>));
  const cudaError_t e = cudaFuncSetAttribute(linear_chunk_kernel<D, AHEAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return cuda_fail(e, what);
  if constexpr (AHEAD) {
    chunk_scores_kernel<D><<<dim3((longest + CK_L - 1) / CK_L, a.G, n_seqs), CK_THREADS, 0, st>>>(a, chunks);
    B2_CHECK_LAUNCH(what);
  }
  linear_chunk_kernel<D, AHEAD><<<dim3(a.dv / CK_P, a.H, n_seqs), CK_THREADS, smem, st>>>(a, chunks);
  B2_CHECK_LAUNCH(what);
  return B2TTS_OK;
}

int launch_linear_chunk(const char* what, const ScanArgs& a, int n_seqs, int longest, int64_t chunks, cudaStream_t st) {
  if (a.scores == nullptr) return a.d == 64 ? go_linear<64, false>(what, a, n_seqs, longest, 0, st) : go_linear<128, false>(what, a, n_seqs, longest, 0, st);
  return a.d == 64 ? go_linear<64, true>(what, a, n_seqs, longest, chunks, st) : go_linear<128, true>(what, a, n_seqs, longest, chunks, st);
}

int64_t delta_prep_floats(int n_tokens, int n_seqs, int H) { return (static_cast<int64_t>(n_tokens) / CK_L + n_seqs + 1) * H * CK_DELTA_PREP; }

template <int D, bool AHEAD>
static int go_delta(const char* what, const ScanArgs& a, int n_seqs, int longest, cudaStream_t st) {
  constexpr int smem = static_cast<int>(sizeof(DeltaTiles<D, AHEAD>));
  cudaError_t e = cudaFuncSetAttribute(delta_chunk_kernel<D, AHEAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return cuda_fail(e, what);
  if constexpr (AHEAD) {
    constexpr int ahead = static_cast<int>(sizeof(DeltaAheadTiles<D>));
    e = cudaFuncSetAttribute(delta_prepare_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, ahead);
    if (e != cudaSuccess) return cuda_fail(e, what);
    delta_prepare_kernel<D><<<dim3((longest + CK_L - 1) / CK_L, a.H, n_seqs), CK_DELTA_THREADS, ahead, st>>>(a);
    B2_CHECK_LAUNCH(what);
  }
  delta_chunk_kernel<D, AHEAD><<<dim3(a.dv / CK_P, a.H, n_seqs), CK_DELTA_THREADS, smem, st>>>(a);
  B2_CHECK_LAUNCH(what);
  return B2TTS_OK;
}

int launch_delta_chunk(const char* what, const ScanArgs& a, int n_seqs, int longest, cudaStream_t st) {
  if (a.scores == nullptr) return a.d == 64 ? go_delta<64, false>(what, a, n_seqs, longest, st) : go_delta<128, false>(what, a, n_seqs, longest, st);
  return a.d == 64 ? go_delta<64, true>(what, a, n_seqs, longest, st) : go_delta<128, true>(what, a, n_seqs, longest, st);
}

}  // namespace row
}  // namespace b2
