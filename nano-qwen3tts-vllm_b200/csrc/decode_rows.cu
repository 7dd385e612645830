// decode_rows.cu - one decode step of a whole decoder stack (models/qwen3_tts_share.py:96-176 of the reference, every layer and the final norm) for up to
// 8 rows as ONE persistent launch.
//
// A step of a few rows is a stream of weights (100 MB a layer of the 1.7B talker, 15.4 us at the copy rate) through a chain of dependent phases.  As
// separate launches the chain costs 44 us a layer: each starts its stream anew and pays drain, boundary and first fetch.  Here one CTA per SM lives for the
// whole step:
//   * a warp of its own copies the CTA's weights - tiles of 8 features, slices of K, layer after layer - into a ring of 144 or 160 KB and waits for nobody but its
//     readers, so that what a phase needs is in shared memory when its input arrives and HBM stays busy while the phases hand over.  A stage is 64
//     or 128 columns of every slice; its copies take up to four tiles at once: copies of 1 KB come in at 33 KB/us a multiprocessor, those of 2 KB and more at the
//     rate of HBM (49);
//   * 8 warps share the tiles and the slices;
//   * the rows are the 16-row operand of mma.sync: the work of a tile is the same for 1 and for 8 rows and a third of what the stream takes, so that
//     the tensor cores' rate does not matter;
//   * hand-overs carry their own flags: every 8-byte word of an activation is two bf16 and the number of the phase that wrote it.  A reader polls the data
//     itself: one L2 trip from store to use, no fence, no counter, no grid barrier (2 to 2.5 us a hand-over in decoder_stack.cu).
// Attention is a phase of its own: a unit (row, key head) per CTA, a warp per query head and split of the context; contexts of more than 4 splits take several
// CTAs, whose partial sums meet in the first one.
//
// Every sum is formed in the order of the separate launches, so that a row has the same bits on either path: products by chains of 16-wide MMAs over
// the K slices of gemm.cu (mma.sync rounds as tcgen05.mma does: equal bits over K of 64 .. 2048), slices added in order; row norms over the threads' vectors of
// rmsnorm_kernel; attention in the tiles and splits of attention_fused.cu.
//
// Why no word is overwritten before its readers are done: a phase's outputs are complete only when all its readers have read (each sum needs
// all slices), and a phase that reads whole rows waits for all outputs of the phase before.  So who writes a buffer again, a layer later,
// has waited for something that followed the last read of it.  A CTA that has no tile in a phase does not read that phase's input; so every CTA has to have tiles of
// gate_up (dr_form() asks for it): with rows that are all padding nobody waits for qkv, and without gate_up a CTA would wait for nothing between two layers.
// All waits are bounded; a wait that runs out is counted (waits.cuh), and the launch goes on to its end with what it has: who has given up waits for no more words, but
// reads, writes and meets the others of its CTA as ever, so that other CTAs find their words, every copy its readers and the next launch everything as it should be.
//
// Bound: a layer of the talker takes 28 us for one row, 13.9 of them the stream at HBM's rate; hand-overs of 1.2 to 2.5 us, five a layer, are the rest (a word
// takes about 0.8 us from store to load while L2 feeds the stream), with 2 us of a tile's softmax after another in attention.  28 layers of the talker and its head, one row
// behind 97 tokens: 1251 us as launches, 812 so (slices of 16 warps in copies of 1 KB: 931).  Tables with room for more tokens cut a context into more splits and CTAs, whatever
// its length: the stack alone, one row behind 100 tokens in tables of 4096 1240 / 1020, behind 2700 1535 / 1250; 4 rows see b2tts_decode_rows_taken().
// What did not do: cp.async of the warps themselves (25 to 40 cycles a 512-byte instruction, 1610 us), 16 warps with one tile each (four times the
// instructions a byte), projections of 5 and more rows (every CTA reads every row, with flags).
#include <type_traits>

#include "fused_attn.cuh"
#include "umma.cuh"
#include "waits.cuh"

namespace b2 {

constexpr int DR_WARPS = 8, DR_READERS = DR_WARPS * 32, DR_THREADS = DR_READERS + 32;
constexpr int DR_HD = 128, DR_GROUP = 2, DR_Q = 2048, DR_KV = DR_Q / DR_GROUP, DR_KVH = DR_KV / DR_HD, DR_MAX_LAYERS = 40, DR_MAX_ROWS = 8;
constexpr int DR_PART_SPLITS = DR_WARPS / DR_GROUP;        // splits of a context that one CTA takes: a warp a query head
constexpr int DR_POLLS = 1 << 20, DR_PAGES = 64;         // tries for a word; pages of a row that are kept
constexpr int DR_UNIT = 1024;                      // 8 features x 64 columns, as the packed weights have them
constexpr int DR_STAGES = 16;                      // stages in flight at most
constexpr int DR_SUMS = 32;                        // (tile, slice) sums of a CTA's phase
constexpr int DR_MAX_TILES = 4;                    // tiles of a warp in a phase
constexpr unsigned DR_LAST_BASE = 0xffffffffu - 2 * DR_MAX_LAYERS * 8;      // behind a later one the numbers of a step might pass 2^32
enum { DR_E_QKV = 1, DR_E_ATT = 2, DR_E_RES1 = 3, DR_E_ACT = 4, DR_E_RES2 = 5, DR_E_PART = 6, DR_E_LAYER = 8 };

__device__ int g_rows_timeouts = 0;                // see waits.cuh
__device__ __forceinline__ void dr_report(int* word) {
  const int n = atomicAdd(&g_rows_timeouts, 1) + 1;
  if (word != nullptr) *reinterpret_cast<volatile int*>(word) = n;
  __threadfence_system();
}

struct DrLayer {
  const uint8_t *w_qkv, *w_o, *w_gu, *w_down;            // packed weights
  const __nv_bfloat16 *ln_in, *ln_post, *qn_w, *kn_w;    // norm weights
  __nv_bfloat16 *k_cache, *v_cache;                      // [pages, page, kvh, 128]
};
struct DrParams {
  int num_layers, m;
  const __nv_bfloat16* x_in;
  int64_t x_stride;
  __nv_bfloat16* out;
  int64_t out_stride;
  const __nv_bfloat16* final_w;
  float eps;
  const int64_t* positions;
  int64_t pos_row_stride;
  const float* inv_freq;
  const int32_t* modality;
  float attention_scaling, scale_log2;
  const int32_t* slot_mapping;
  const int32_t* block_table;
  int bt_stride, page_shift;
  const int32_t* context_lens;
  int polls;                                             // tries after which a wait for a word gives up
  int nsplit, max_parts;                                 // splits of a context; CTAs a unit may take
  unsigned* sync;                                        // [0] the number of the last phase, [1] CTAs that are done
  uint64_t *qkv, *att, *res1, *act, *res2, *part, *words_end;
  int* waits;                                            // host word of waits that ran out (or null)
  DrLayer layer[DR_MAX_LAYERS];
};

// ---------------------------------------------------------------- words with flags
__device__ __forceinline__ void dr_put(uint64_t* at, uint32_t data, uint32_t flag) {
  const uint64_t w = static_cast<uint64_t>(flag) << 32 | data;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(at), "l"(w) : "memory");
}
__device__ __forceinline__ uint64_t dr_get(const uint64_t* at) {
  uint64_t w;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(at) : "memory");
  return w;
}
__device__ __forceinline__ void dr_get2(const uint64_t* at, uint64_t& a, uint64_t& b) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(at) : "memory");
}
// one word, polled
__device__ __forceinline__ uint32_t dr_wait(const uint64_t* at, uint32_t flag, int polls, bool& alive) {
  uint64_t w = dr_get(at);
  for (int n = 0; static_cast<uint32_t>(w >> 32) != flag && alive; ++n) {
    if (n >= polls) alive = false;
    w = dr_get(at);
  }
  return static_cast<uint32_t>(w);
}
// the first n of N vectors of four words (32-byte aligned), `apart` words from one another: all asked for at once, those that are not there yet again
template <int N>
__device__ __forceinline__ void dr_wait_all(const uint64_t* at, int apart, int n, uint32_t flag, uint4 (&x)[N], int polls, bool& alive) {
  uint32_t todo = (1u << n) - 1;
  for (int tries = 0; todo != 0; ++tries) {
    uint64_t w[N][4];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      w[i][0] = w[i][1] = w[i][2] = w[i][3] = 0;
      if (todo >> i & 1) { dr_get2(at + i * apart, w[i][0], w[i][1]); dr_get2(at + i * apart + 2, w[i][2], w[i][3]); }
    }
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (todo >> i & 1) {
        bool ok = true;
#pragma unroll
        for (int e = 0; e < 4; ++e) ok = ok && static_cast<uint32_t>(w[i][e] >> 32) == flag;
        if (ok || !alive) {
          x[i] = make_uint4(static_cast<uint32_t>(w[i][0]), static_cast<uint32_t>(w[i][1]), static_cast<uint32_t>(w[i][2]), static_cast<uint32_t>(w[i][3]));
          todo &= ~(1u << i);
        }
      }
    if (tries >= polls) alive = false;
  }
}

__device__ __forceinline__ void dr_ldsm4(uint32_t* f, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3]) : "r"(addr));
}
// This CTA's tiles of a phase, in groups that lie in one piece of the packed weights: four where that makes no CTA's share longer by more than a tile, two where
// it makes none longer
__host__ __device__ __forceinline__ int dr_group(int tiles, int ctas) {
  const int most = (tiles + ctas - 1) / ctas;
  return ((tiles + 3) / 4 + ctas - 1) / ctas * 4 <= most + 1 ? 4 : ((tiles + 1) / 2 + ctas - 1) / ctas * 2 <= most ? 2 : 1;
}
__device__ __forceinline__ void dr_span(int tiles, int& t0, int& t1) {
  const int g = dr_group(tiles, gridDim.x), n = (tiles + g - 1) / g;
  t0 = min(tiles, static_cast<int>(blockIdx.x * n / gridDim.x) * g);
  t1 = min(tiles, static_cast<int>((blockIdx.x + 1) * n / gridDim.x) * g);
}
// The sums of a phase, [tile][slice][row][8 features]: columns col, col + 1 of a row, slices in order
template <int S>
__device__ __forceinline__ float2 dr_sum(const float* red, int tile, int row, int col) {
  const float* at = red + tile * S * 64 + row * 8 + col;
  float2 s = make_float2(0.f, 0.f);
#pragma unroll
  for (int w = 0; w < S; ++w) {
    const float2 y = *reinterpret_cast<const float2*>(at + w * 64);
    s.x += y.x; s.y += y.y;
  }
  return s;
}
__device__ __forceinline__ void dr_sync() { asm volatile("bar.sync 1, %0;" ::"n"(DR_READERS) : "memory"); }

// A unit of attention: a row's key head, which of the CTAs that have it this is, the context, and the CTA's splits of it
struct DrUnit { int row, head, part, L, s0, s1; };

// The arithmetic of fused_decode_attn_kernel, a warp a query head of a split; returns whether no wait ran out.
template <bool EAGER>
__device__ __forceinline__ bool dr_attend(const DrParams& p, const DrLayer& y, uint32_t e0, const DrUnit& a, __nv_bfloat16* q_s, const uint4* trig_s, const int* pages, uint8_t* x_s,
                                       bool alive) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, ag = lane >> 3, aj = lane & 7;
  const int row = a.row, head = a.head, part = a.part, L = a.L, s0 = a.s0, s1 = a.s1, tiles = (L + FA_TILE - 1) / FA_TILE;
  // element offset of a cached token's head in the layer's pool
  auto cached_at = [&](int t) -> int64_t {
    const int i = t >> p.page_shift;
    const int page = i < DR_PAGES ? pages[i] : max(0, __ldg(p.block_table + static_cast<int64_t>(row) * p.bt_stride + i));        // never faults on a stale (-1) entry
    return (((static_cast<int64_t>(page) << p.page_shift) + (t & ((1 << p.page_shift) - 1))) * DR_KVH + head) * DR_HD + 8 * aj;
  };
  float2* fold_ml = reinterpret_cast<float2*>(x_s);                               // [head][split] (largest score, sum)
  float* fold_av = reinterpret_cast<float*>(fold_ml + DR_GROUP * 32);             // [head][split][128]
  uint64_t* part_w = p.part + static_cast<int64_t>(row * DR_KVH + head) * 32 * DR_GROUP * (2 + DR_HD);

  // keys and values of a tile of 8 tokens: slot ag of each four, dims 8 aj .. and 64 + 8 aj ..
  struct Tile { uint4 k[2][2], v[2][2]; };
  Tile t0 = {}, t1 = {};
  auto fetch = [&](Tile& f, int tile) {
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      const int t = tile * FA_TILE + it * 4 + ag;
      f.k[it][0] = f.k[it][1] = f.v[it][0] = f.v[it][1] = make_uint4(0, 0, 0, 0);
      if (t < L - 1) {
        const int64_t at = cached_at(t);
        f.k[it][0] = __ldg(reinterpret_cast<const uint4*>(y.k_cache + at));      // the other head's warp finds them in L1
        f.k[it][1] = __ldg(reinterpret_cast<const uint4*>(y.k_cache + at + 64));
        f.v[it][0] = __ldg(reinterpret_cast<const uint4*>(y.v_cache + at));
        f.v[it][1] = __ldg(reinterpret_cast<const uint4*>(y.v_cache + at + 64));
      }
    }
  };
  const int ah = warp & 1;                                                    // this warp's query head
  int sp = s0 + (warp >> 1), tb = 0, te = 0;
  auto start = [&]() {
    tb = sp * tiles / p.nsplit;
    te = (sp + 1) * tiles / p.nsplit;
    if (tb < te) fetch(t0, tb);
    if (tb + 1 < te) fetch(t1, tb + 1);
  };
  if (sp < s1) {
    start();
    // the other tiles of the split on their way to L2 (the weights of a step have driven them out): half of them by each of the two warps
    for (int t = (tb + 2) * FA_TILE + lane; t < min(te * FA_TILE, L - 1); t += 32) {
      const __nv_bfloat16* at = (ah ? y.v_cache : y.k_cache) + cached_at(t) - 8 * aj;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(at + 64));
    }
  }
  // the new token: warps 0, 1 a query head each, 2 the key, 3 the value
  if (L > 0 && warp < DR_GROUP + 2) {
    const int col = warp < DR_GROUP ? (head * DR_GROUP + warp) * DR_HD : DR_Q + (warp - DR_GROUP) * DR_KV + head * DR_HD;
    const uint64_t* at = p.qkv + row * ((DR_Q + 2 * DR_KV) / 2) + col / 2 + lane;
    const __nv_bfloat16* nw = warp < DR_GROUP ? y.qn_w : y.kn_w;
    const uint32_t w1 = nw != nullptr ? __ldg(reinterpret_cast<const unsigned*>(nw + 2 * lane)) : 0u;
    const uint32_t w2 = nw != nullptr ? __ldg(reinterpret_cast<const unsigned*>(nw + 64 + 2 * lane)) : 0u;
    uint32_t y1 = dr_wait(at, e0 + DR_E_QKV, p.polls, alive), y2 = dr_wait(at + 32, e0 + DR_E_QKV, p.polls, alive);
    __syncwarp();
    if (warp < DR_GROUP + 1) {
      if (nw != nullptr) {
        float ss = bf16lo(y1) * bf16lo(y1);
        ss = fmaf(bf16hi(y1), bf16hi(y1), ss); ss = fmaf(bf16lo(y2), bf16lo(y2), ss); ss = fmaf(bf16hi(y2), bf16hi(y2), ss);
        const float var = warp_sum(ss) / static_cast<float>(DR_HD) + p.eps;
        const float rstd = EAGER ? 1.0f / sqrtf(var) : rsqrtf(var);
        y1 = norm_pair<EAGER>(y1, rstd, w1);
        y2 = norm_pair<EAGER>(y2, rstd, w2);
      }
      const uint4 z = trig_s[lane];
      const uint32_t x1 = y1, x2 = y2;
      y1 = turn_first(x1, x2, z.x, z.y);
      y2 = turn_second(x1, x2, z.z, z.w);
    }
    uint32_t* to = reinterpret_cast<uint32_t*>(q_s + warp * DR_HD);
    to[lane] = y1; to[32 + lane] = y2;
    const int slot_new = part == 0 && warp >= DR_GROUP ? __ldg(p.slot_mapping + row) : -1;
    if (slot_new >= 0) {
      uint32_t* cd = reinterpret_cast<uint32_t*>((warp == DR_GROUP ? y.k_cache : y.v_cache) + (static_cast<int64_t>(slot_new) * DR_KVH + head) * DR_HD);
      cd[lane] = y1; cd[32 + lane] = y2;
    }
  }
  dr_sync();
  for (bool first = true; sp < s1; sp += DR_WARPS / DR_GROUP, first = false) {
    if (!first) start();
    float qv[16], mx = -INFINITY, ls = 0.f, acc[16];
    fa_unpack8(*reinterpret_cast<const uint4*>(q_s + ah * DR_HD + 8 * aj), qv);
    fa_unpack8(*reinterpret_cast<const uint4*>(q_s + ah * DR_HD + 64 + 8 * aj), qv + 8);
#pragma unroll
    for (int d = 0; d < 16; ++d) { qv[d] *= p.scale_log2; acc[d] = 0.f; }
    auto step = [&](Tile& f, int tile) {
      float sc[2];
#pragma unroll
      for (int it = 0; it < 2; ++it) {
        const int t = tile * FA_TILE + it * 4 + ag;
        if (t == L - 1) {                                                         // the new token
          f.k[it][0] = *reinterpret_cast<const uint4*>(q_s + DR_GROUP * DR_HD + 8 * aj);
          f.k[it][1] = *reinterpret_cast<const uint4*>(q_s + DR_GROUP * DR_HD + 64 + 8 * aj);
          f.v[it][0] = *reinterpret_cast<const uint4*>(q_s + (DR_GROUP + 1) * DR_HD + 8 * aj);
          f.v[it][1] = *reinterpret_cast<const uint4*>(q_s + (DR_GROUP + 1) * DR_HD + 64 + 8 * aj);
        }
        float z[16], d0 = 0.f, d1 = 0.f;
        fa_unpack8(f.k[it][0], z);
        fa_unpack8(f.k[it][1], z + 8);
#pragma unroll
        for (int d = 0; d < 16; d += 2) { d0 = fmaf(qv[d], z[d], d0); d1 = fmaf(qv[d + 1], z[d + 1], d1); }
        float dot = d0 + d1;
        dot += __shfl_xor_sync(0xffffffffu, dot, 1);
        dot += __shfl_xor_sync(0xffffffffu, dot, 2);
        dot += __shfl_xor_sync(0xffffffffu, dot, 4);
        sc[it] = t < L ? dot : -INFINITY;
      }
      float mt = fmaxf(sc[0], sc[1]);
      mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 8));
      mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 16));
      const float mn = fmaxf(mx, mt), alpha = fa_exp2(mx - mn);
      mx = mn;
      float ps = 0.f;
#pragma unroll
      for (int it = 0; it < 2; ++it) { sc[it] = fa_exp2(sc[it] - mn); ps += sc[it]; }
      ls = fmaf(ls, alpha, ps);
#pragma unroll
      for (int d = 0; d < 16; ++d) acc[d] *= alpha;
#pragma unroll
      for (int it = 0; it < 2; ++it) {
        float z[16];
        fa_unpack8(f.v[it][0], z);
        fa_unpack8(f.v[it][1], z + 8);
#pragma unroll
        for (int d = 0; d < 16; ++d) acc[d] = fmaf(sc[it], z[d], acc[d]);
      }
      if (tile + 2 < te) fetch(f, tile + 2);
    };
#pragma unroll 1
    for (int tile = tb; tile < te; tile += 2) {
      step(t0, tile);
      if (tile + 1 < te) step(t1, tile + 1);
    }
    ls += __shfl_xor_sync(0xffffffffu, ls, 8);
    ls += __shfl_xor_sync(0xffffffffu, ls, 16);
#pragma unroll
    for (int d = 0; d < 16; ++d) {
      acc[d] += __shfl_xor_sync(0xffffffffu, acc[d], 8);
      acc[d] += __shfl_xor_sync(0xffffffffu, acc[d], 16);
    }
    if (ag == 0) {
      if (part == 0) {
        if (aj == 0) fold_ml[ah * 32 + sp] = make_float2(mx, ls);
        float* to = fold_av + (ah * 32 + sp) * DR_HD + 8 * aj;
#pragma unroll
        for (int d = 0; d < 16; d += 4) *reinterpret_cast<float4*>(to + (d < 8 ? d : 56 + d)) = make_float4(acc[d], acc[d + 1], acc[d + 2], acc[d + 3]);
      } else {
        uint64_t* to = part_w + (ah * 32 + sp) * (2 + DR_HD);
        if (aj == 0) { dr_put(to, __float_as_uint(mx), e0 + DR_E_PART); dr_put(to + 1, __float_as_uint(ls), e0 + DR_E_PART); }
#pragma unroll
        for (int d = 0; d < 16; ++d) dr_put(to + 2 + 8 * aj + (d < 8 ? d : 56 + d), __float_as_uint(acc[d]), e0 + DR_E_PART);
      }
    }
    __syncwarp();
  }
  // ---- the splits in order; those of other CTAs come in first, all words at once
  if (part == 0) {
    const int words = (p.nsplit - s1) * (2 + DR_HD);                              // of a head; [head][split][score, sum, values]
#pragma unroll 1
    for (int k = tid; k < DR_GROUP * words; k += DR_READERS) {
      const int h = k >= words ? 1 : 0, at = k - h * words, s = s1 + at / (2 + DR_HD), e = at % (2 + DR_HD);
      const float z = __uint_as_float(dr_wait(part_w + (h * 32 + s) * (2 + DR_HD) + e, e0 + DR_E_PART, p.polls, alive));
      if (e < 2) reinterpret_cast<float*>(fold_ml + h * 32 + s)[e] = z;
      else fold_av[(h * 32 + s) * DR_HD + e - 2] = z;
    }
    __syncwarp();
    dr_sync();
    if (tid < DR_GROUP * DR_HD / 2) {
      const int h = tid >> 6, d = 2 * (tid & 63);
      float top = -INFINITY, den = 0.f, n0 = 0.f, n1 = 0.f;
      if (L > 0) {
#pragma unroll 4
        for (int s = 0; s < p.nsplit; ++s) top = fmaxf(top, fold_ml[h * 32 + s].x);
#pragma unroll 4
        for (int s = 0; s < p.nsplit; ++s) {
          const float2 z = fold_ml[h * 32 + s], v = *reinterpret_cast<const float2*>(fold_av + (h * 32 + s) * DR_HD + d);
          if (z.y > 0.f) {
            const float w = fa_exp2(z.x - top);
            n0 = fmaf(w, v.x, n0); n1 = fmaf(w, v.y, n1);
            den = fmaf(w, z.y, den);
          }
        }
      }
      const float inv = den > 0.f ? 1.f / den : 0.f;                              // a padding row has no tokens: zeros
      dr_put(p.att + (row * DR_Q + (head * DR_GROUP + h) * DR_HD + d) / 2, pack_bf16(n0 * inv, n1 * inv), e0 + DR_E_ATT);
    }
    __syncwarp();
  }
  return alive;
}

// What a CTA does in every layer
struct DrPlan { int t0[4], t1[4]; DrUnit unit; };        // tiles of qkv, o, gate_up, down
// Shared memory.  Rows that the residual stream, attention or gate_up leave are held whole, the ring has what is left of 222 KB
template <int H, int I, int ROWS> struct DrShared {
  static constexpr int WIDE = I > DR_Q ? I : DR_Q, FOLD = DR_GROUP * 32 * (2 + DR_HD) * 4, XS = ROWS * WIDE * 2 > FOLD ? ROWS * WIDE * 2 : FOLD;
  static constexpr int UNITS = (222 * 1024 - XS - 2 * DR_SUMS * 64 * 4 - 4096) / DR_UNIT / 16 * 16;
  uint8_t ring[UNITS][DR_UNIT];
  uint8_t x[XS];                                         // a phase's rows; or attention's splits
  float red[2][DR_SUMS * 64];                            // of even and odd phases: [tile][slice][row][8 features]
  float ssq[DR_MAX_ROWS][8];
  __nv_bfloat16 q[(DR_GROUP + 2) * DR_HD];               // two query heads, key, value of the new token
  __align__(16) __nv_bfloat16 trig[DR_HD / 4][4][2];     // for dims 2l, 2l + 1: cosines, sines, and those of dims 64 + 2l, 65 + 2l
  int pages[DR_PAGES];                                   // of the unit's row
  uint64_t full[DR_STAGES], empty[DR_STAGES];
  DrPlan plan;
  unsigned base;
  int lost;                                              // somebody gave up
};

// H, I: hidden and inner width; SG, SQ: slices of K of gate_up and of the other projections; ROWS: most rows
template <int H, int I, int SQ, int SG, int ROWS, bool EAGER>
__global__ void __launch_bounds__(DR_THREADS, 1)
decode_rows_kernel(const __grid_constant__ DrParams p) {
  using Sm = DrShared<H, I, ROWS>;
  static_assert((SG & (SG - 1)) == 0 && SQ == DR_WARPS && ROWS <= DR_MAX_ROWS, "warps are slices x tiles");
  constexpr int VECS = H / 8;
  extern __shared__ __align__(1024) uint8_t dr_smem[];
  Sm& sm = *reinterpret_cast<Sm*>(dr_smem);
  int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int m = p.m;
  if (tid == 0) {
    for (int s = 0; s < DR_STAGES; ++s) { mbar_init(sm.full + s, 1); mbar_init(sm.empty + s, DR_WARPS); }
    mbar_fence_init();
    sm.base = *reinterpret_cast<volatile unsigned*>(p.sync);
    sm.lost = 0;
    DrPlan& a = sm.plan;
    dr_span((DR_Q + 2 * DR_KV) / 8, a.t0[0], a.t1[0]);
    dr_span(H / 8, a.t0[1], a.t1[1]);
    dr_span(2 * I / 8, a.t0[2], a.t1[2]);
    a.t0[3] = a.t0[1]; a.t1[3] = a.t1[1];
    // this CTA's unit of attention, the same in every layer: a row's key head, and which of the CTAs that have it this one is
    DrUnit& u = a.unit;
    u.part = blockIdx.x / (m * DR_KVH); u.row = blockIdx.x % (m * DR_KVH) / DR_KVH; u.head = blockIdx.x % DR_KVH;
    u.L = u.part < p.max_parts ? max(0, p.context_lens[u.row]) : 0;
    const int parts = u.L > 0 ? p.max_parts : 1;
    u.s0 = u.part * p.nsplit / parts; u.s1 = u.part < parts ? (u.part + 1) * p.nsplit / parts : 0;      // no splits: no part in it
  }
  __syncthreads();
  auto slices_of = [](int phase) { return phase == 2 ? SG : SQ; };
  // a stage: two steps of 64 columns of every slice, of qkv (whose steps are the widest) one
  auto per_stage_of = [](int phase) { return phase == 0 ? 1 : 2; };
  auto steps_of = [](int phase) { return phase == 0 ? H / 64 / SQ : phase == 1 ? DR_Q / 64 / SQ : phase == 2 ? H / 64 / SG : I / 64 / SQ; };

  if (warp == DR_WARPS) {
    // =========================== the stream of weights.  A lane has a slice and four tiles in a row (from a multiple of four: in one piece as they are packed)
    bool alive = true;
    int count = 0, oldest = 0, head = 0, my_start = 0;     // stages asked for, the oldest that may still be read, where the next one begins; lane k: stage k's begin
#pragma unroll 1
    for (int i = 0; i < 4 * p.num_layers && alive; ++i) {
      const int phase = i & 3, t0 = sm.plan.t0[phase], t1 = sm.plan.t1[phase], nt = t1 - t0, S = slices_of(phase), per = 32 / S;
      if (nt == 0) continue;
      const DrLayer& y = p.layer[i >> 2];
      const uint8_t* w = phase == 0 ? y.w_qkv : phase == 1 ? y.w_o : phase == 2 ? y.w_gu : y.w_down;
      const int steps = steps_of(phase), slice = lane / per, first = (t0 & ~3) + 4 * (lane % per);
      const int ta = max(t0, first), bytes = (min(t1, first + 4) - ta) * DR_UNIT;
      const uint8_t* src = w + (static_cast<int64_t>(ta >> 4) * (steps * S) + slice * steps) * G_WTILE_BYTES + (ta & 15) * DR_UNIT;
      const int unit = slice * nt + ta - t0, row = nt * S, subs = per_stage_of(phase), size = row * subs;
#pragma unroll 1
      for (int j = 0; j < steps && alive; j += subs) {
        const int at = head + size > Sm::UNITS ? 0 : head;
        while (alive && oldest < count) {                  // room: stages lie one behind the other from the oldest one's begin to head
          const int begin = __shfl_sync(0xffffffffu, my_start, oldest % DR_STAGES);
          const bool free = head > begin ? (at == head || size <= begin) : (at == head && head + size <= begin);
          if (free && count - oldest < DR_STAGES) break;
          alive = mbar_wait_limit(sm.empty + oldest % DR_STAGES, (oldest / DR_STAGES) & 1);
          ++oldest;
        }
        if (!alive) break;
        uint64_t* bar = sm.full + count % DR_STAGES;
        if (lane == 0) mbar_expect_tx(bar, size * DR_UNIT);
        __syncwarp();
#pragma unroll 1
        for (int k = 0; k < subs; ++k) {
          if (bytes > 0) bulk_g2s(sm.ring[at + k * row + unit], src, bytes, bar);
          src += G_WTILE_BYTES;
        }
        if (lane == count % DR_STAGES) my_start = at;
        head = at + size;
        ++count;
      }
    }
    if (!alive && lane == 0) sm.lost = 1;
    // nothing of this CTA's is in flight when it leaves
#pragma unroll 1
    for (int k = max(0, count - DR_STAGES); k < count; ++k) mbar_wait_limit(sm.full + k % DR_STAGES, (k / DR_STAGES) & 1);
    __syncthreads();
    return;
  }

  // =========================== the phases
  const uint32_t base = sm.base;
  bool alive = true, stream = true;                        // no wait of this lane for words, of this warp for weights ran out
  int stage = 0, head = 0;                                 // the next one of the stream, and where the one before it ends
  // Rows lie in shared memory as they are, vector v (8 columns) of row r at v ^ r in its group of eight: a warp's ldmatrix reads eight rows without conflicts
  auto put_vec = [&](int width, int r, int v, const uint4& x) {
    *reinterpret_cast<uint4*>(sm.x + r * (width * 2) + (((v & ~7) | ((v ^ r) & 7)) << 4)) = x;
  };
  auto squares = [](const uint4& x) -> float {
    const uint32_t e[4] = {x.x, x.y, x.z, x.w};
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) { s = fmaf(bf16lo(e[k]), bf16lo(e[k]), s); s = fmaf(bf16hi(e[k]), bf16hi(e[k]), s); }
    return s;
  };
  auto rstd_of = [&](float s) -> float { const float var = s / static_cast<float>(H) + p.eps; return EAGER ? 1.0f / sqrtf(var) : rsqrtf(var); };
  // Normed rows: thread tid has vector tid % VECS of rows tid / VECS, + 256 / VECS, ...  Sums: a thread's eight squares in order, the lanes of a warp, the
  // warps of a row.
  auto norm_rows = [&](bool first, const uint64_t* res, uint32_t flag, const __nv_bfloat16* w) {
    constexpr int RP = DR_READERS / VECS, PASSES = (ROWS + RP - 1) / RP, RW = VECS / 32;        // rows a pass; warps a row
    const int v = tid % VECS, r0 = tid / VECS;
    const uint32_t* w4 = reinterpret_cast<const uint32_t*>(w) + 4 * v;
    const uint4 wv = make_uint4(__ldg(w4), __ldg(w4 + 1), __ldg(w4 + 2), __ldg(w4 + 3));
    uint4 x[PASSES] = {};
    if (first) {
#pragma unroll
      for (int i = 0; i < PASSES; ++i) {
        const int r = r0 + i * RP;
        const uint32_t* at = reinterpret_cast<const uint32_t*>(p.x_in + r * p.x_stride) + 4 * v;
        if (r < m) x[i] = make_uint4(at[0], at[1], at[2], at[3]);
      }
    } else {
      dr_wait_all<PASSES>(res + r0 * (H / 2) + 4 * v, RP * (H / 2), r0 < m ? (m - r0 + RP - 1) / RP : 0, flag, x, p.polls, alive);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < PASSES; ++i) {
      const int r = r0 + i * RP;
      if (r < m) {                                                                // a warp has vectors of one row
        const float s = warp_sum(squares(x[i]));
        if (lane == 0) sm.ssq[r][warp % RW] = s;
      }
    }
    dr_sync();
#pragma unroll
    for (int i = 0; i < PASSES; ++i) {
      const int r = r0 + i * RP;
      if (r < m) put_vec(H, r, v, norm8(x[i], wv, rstd_of(warp_sum(lane < RW ? sm.ssq[r][lane & 7] : 0.f)), EAGER));
    }
    dr_sync();
  };
  // rows of `width` columns that another phase leaves
  auto take_rows = [&](int width, const uint64_t* in, uint32_t flag) {
    constexpr int AT_ONCE = ROWS == 2 ? 4 : 8;
    const int per = width / 8, all = m * per;
#pragma unroll 1
    for (int i0 = tid; i0 < all; i0 += AT_ONCE * DR_READERS) {
      uint4 x[AT_ONCE] = {};
      const int n = min(AT_ONCE, (all - i0 + DR_READERS - 1) / DR_READERS);
      dr_wait_all<AT_ONCE>(in + 4 * i0, 4 * DR_READERS, n, flag, x, p.polls, alive);
      __syncwarp();                                        // lanes leave the polling one by one, the barrier behind it wants whole warps
#pragma unroll
      for (int u = 0; u < AT_ONCE; ++u) {
        const int i = i0 + u * DR_READERS;
        if (u < n) put_vec(width, i / per, i % per, x[u]);
      }
    }
    dr_sync();
  };
  // The rows x this warp's tiles (of a slice's, every 8 / slices-th), whose chains of products take turns.  A step's fragments are read while the products of the
  // one before it run.
  auto products = [&](int phase, int width, float* red) {
    const int S = slices_of(phase), tiles = sm.plan.t1[phase] - sm.plan.t0[phase], steps = steps_of(phase), subs = per_stage_of(phase);
    const int slice = warp & (S - 1), tl = DR_WARPS / S, t0 = warp / S, row_bytes = tiles * S * DR_UNIT, size = tiles * S * subs;
    const int nt = t0 < tiles ? (tiles - t0 + tl - 1) / tl : 0, r = lane & (ROWS - 1), mi = lane >> 3;     // rows that there is no room for read others: nobody reads their sums
    float acc[DR_MAX_TILES][4] = {};
    const uint32_t w_at = smem_u32(sm.ring[0]) + (slice * tiles + t0) * DR_UNIT + (lane & 7) * 128, tile_step = tl * DR_UNIT;
    const uint32_t w0 = w_at + ((mi ^ (lane & 7)) << 4), w1 = w_at + (((4 + mi) ^ (lane & 7)) << 4);
    const uint32_t x_at = smem_u32(sm.x) + r * (width * 2) + slice * steps * 128, x0 = x_at + ((mi ^ r) << 4), x1 = x_at + (((4 + mi) ^ r) << 4);
    struct Stage { uint32_t x[2][4], w[DR_MAX_TILES][2][4]; };
    uint32_t in = 0;
    auto enter = [&]() {                                                          // the next stage
      const int at = head + size > Sm::UNITS ? 0 : head;
      head = at + size;
      in = at * DR_UNIT;
      // (alive or not: readers that ran ahead of the copies would free stages that are still to land)
      if (stream && !mbar_wait_limit(sm.full + stage % DR_STAGES, (stage / DR_STAGES) & 1)) stream = alive = false;
      ++stage;
    };
    auto read = [&](int j, Stage& f) {
#pragma unroll
      for (int i = 0; i < DR_MAX_TILES; ++i)
        if (i < nt) { dr_ldsm4(f.w[i][0], w0 + in + i * tile_step); dr_ldsm4(f.w[i][1], w1 + in + i * tile_step); }
      dr_ldsm4(f.x[0], x0 + j * 128);
      dr_ldsm4(f.x[1], x1 + j * 128);
    };
    auto multiply = [&](const Stage& f) {
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const uint32_t a0[4] = {f.x[b][0], 0u, f.x[b][1], 0u}, a1[4] = {f.x[b][2], 0u, f.x[b][3], 0u};
#pragma unroll
        for (int i = 0; i < DR_MAX_TILES; ++i)
          if (i < nt) mma_bf16_16816(acc[i], a0, f.w[i][b][0], f.w[i][b][1]);
#pragma unroll
        for (int i = 0; i < DR_MAX_TILES; ++i)
          if (i < nt) mma_bf16_16816(acc[i], a1, f.w[i][b][2], f.w[i][b][3]);
      }
    };
    auto leave = [&](int number) {
      __syncwarp();
      if (lane == 0) mbar_arrive(sm.empty + number % DR_STAGES);
    };
    Stage f0 = {}, f1 = {};                                                       // (what is set under a condition alone counts as live everywhere)
    enter();
    read(0, f0);
#pragma unroll 1
    for (int j = 0; j < steps; j += 2) {                                          // an even number
      if (subs == 1) enter();
      else in += row_bytes;
      read(j + 1, f1);
      multiply(f0);
      if (subs == 1) leave(stage - 2);
      const int mine = stage - 1;
      if (j + 2 < steps) { enter(); read(j + 2, f0); }
      multiply(f1);
      leave(mine);
    }
#pragma unroll
    for (int i = 0; i < DR_MAX_TILES; ++i)
      if (i < nt) *reinterpret_cast<float2*>(red + (warp + i * DR_WARPS) * 64 + (lane >> 2) * 8 + 2 * (lane & 3)) = make_float2(acc[i][0], acc[i][1]);
    dr_sync();
  };

  if (sm.plan.unit.s1 > 0 && tid < min(p.bt_stride, DR_PAGES)) sm.pages[tid] = max(0, __ldg(p.block_table + static_cast<int64_t>(sm.plan.unit.row) * p.bt_stride + tid));
  if (sm.plan.unit.s1 > 0 && sm.plan.unit.L > 0 && tid < DR_HD / 2) {
    const int row = sm.plan.unit.row;
    int64_t pos[3];
    pos[0] = pos[1] = pos[2] = __ldg(p.positions + row);
    if (p.modality != nullptr && p.pos_row_stride != 0) {
      pos[1] = __ldg(p.positions + p.pos_row_stride + row);
      pos[2] = __ldg(p.positions + 2 * p.pos_row_stride + row);
    }
    const float f = __ldg(p.inv_freq + tid);
    const int m1 = p.modality != nullptr ? __ldg(p.modality + tid) : 0, m2 = p.modality != nullptr ? __ldg(p.modality + 64 + tid) : 0;
    const float a1 = static_cast<float>(m1 == 0 ? pos[0] : m1 == 1 ? pos[1] : pos[2]) * f;
    const float a2 = static_cast<float>(m2 == 0 ? pos[0] : m2 == 1 ? pos[1] : pos[2]) * f;
    __nv_bfloat16(*to)[2] = sm.trig[tid >> 1];
    to[0][tid & 1] = __float2bfloat16_rn(cosf(a1) * p.attention_scaling);
    to[1][tid & 1] = __float2bfloat16_rn(sinf(a1) * p.attention_scaling);
    to[2][tid & 1] = __float2bfloat16_rn(cosf(a2) * p.attention_scaling);
    to[3][tid & 1] = __float2bfloat16_rn(sinf(a2) * p.attention_scaling);
  }
  dr_sync();

  // Four phases a layer: qkv; attention and o; gate_up; down.  One copy of the code that copies, multiplies and norms: it is read once a phase, and an
  // instruction cache that does not hold it costs more than the products
#pragma unroll 1
  for (int i = 0; i < 4 * p.num_layers; ++i) {
    // addresses are formed where they are used: kept from phase to phase they would take the registers that attention needs
    asm volatile("" : "+r"(tid), "+r"(warp), "+r"(lane));
    const int l = i >> 2;
    int phase = i & 3;
    asm volatile("" : "+r"(phase));
    const DrLayer& y = p.layer[l];
    const uint32_t e0 = base + l * DR_E_LAYER;
    const int tile0 = sm.plan.t0[phase], tile1 = sm.plan.t1[phase];
    const int row = (tid >> 2) & 7, n = (tile0 + (tid >> 5)) * 8 + 2 * (tid & 3);                // of o and down: whose sum this thread finishes
    const bool mine = (phase & 1) && tile0 + (tid >> 5) < tile1 && row < m;
    uint32_t r = 0;
    if (phase & 1) {
      if (phase == 1) {
        if (sm.plan.unit.s1 > 0) alive = dr_attend<EAGER>(p, y, e0, sm.plan.unit, sm.q, reinterpret_cast<const uint4*>(sm.trig), sm.pages, sm.x, alive);
        dr_sync();                                                                // its splits have been read
        asm volatile("" : "+r"(tid), "+r"(warp), "+r"(lane));
      }
      if (tile0 == tile1) continue;
      take_rows(phase == 3 ? I : DR_Q, phase == 3 ? p.act : p.att, e0 + (phase == 3 ? DR_E_ACT : DR_E_ATT));
      if (mine)
        r = i == 1 ? *reinterpret_cast<const uint32_t*>(p.x_in + row * p.x_stride + n)
                   : dr_wait((phase == 3 ? p.res1 : p.res2) + (row * H + n) / 2, phase == 3 ? e0 + DR_E_RES1 : e0 - DR_E_LAYER + DR_E_RES2, p.polls, alive);
      __syncwarp();
    } else {
      if (tile0 == tile1) continue;
      norm_rows(i == 0, phase == 2 ? p.res1 : p.res2, phase == 2 ? e0 + DR_E_RES1 : e0 - DR_E_LAYER + DR_E_RES2, phase == 2 ? y.ln_post : y.ln_in);
    }
    // the next norm's weights on their way to L2
    if ((phase & 1) && tid < H / 64 && blockIdx.x < 4) {
      const __nv_bfloat16* w = phase == 1 ? y.ln_post : l + 1 < p.num_layers ? p.layer[l + 1].ln_in : p.final_w;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(w + tid * 64));
    }
    products(phase, phase == 1 ? DR_Q : phase == 3 ? I : H, sm.red[phase & 1]);
    if (phase & 1) {
      if (mine) {
        const float2 s = dr_sum<SQ>(sm.red[1], tid >> 5, row, 2 * (tid & 3));
        dr_put((phase == 3 ? p.res2 : p.res1) + (row * H + n) / 2, pack_bf16(rbf(s.x) + bf16lo(r), rbf(s.y) + bf16hi(r)), e0 + (phase == 3 ? DR_E_RES2 : DR_E_RES1));
      }
    } else if (phase == 0) {
#pragma unroll 1
      for (int k = tid; k < (tile1 - tile0) * 32; k += DR_READERS) {
        const int tile = k >> 5, q = (k >> 2) & 7;
        if (q < m) {
          const float2 s = dr_sum<SQ>(sm.red[0], tile, q, 2 * (k & 3));
          dr_put(p.qkv + q * ((DR_Q + 2 * DR_KV) / 2) + (tile0 + tile) * 4 + (k & 3), pack_bf16(s.x, s.y), e0 + DR_E_QKV);
        }
      }
    } else {
#pragma unroll 1
      for (int k = tid; k < (tile1 - tile0) * 16; k += DR_READERS) {
        const int tile = k >> 4, q = (k >> 1) & 7, col = 2 * (k & 1);
        if (q < m) {
          const float2 gs = dr_sum<SG>(sm.red[0], tile, q, col), us = dr_sum<SG>(sm.red[0], tile, q, 4 + col);
          const float ga = rbf(gs.x), gb = rbf(gs.y), ua = rbf(us.x), ub = rbf(us.y);
          const float va = EAGER ? rbf(gsilu_f(ga)) * ua : gsilu_f(ga) * ua, vb = EAGER ? rbf(gsilu_f(gb)) * ub : gsilu_f(gb) * ub;
          dr_put(p.act + (q * I + (tile0 + tile) * 4 + col) / 2, pack_bf16(va, vb), e0 + DR_E_ACT);
        }
      }
    }
  }
  // ---- the final norm, a row a CTA
  const uint32_t last = base + (p.num_layers - 1) * DR_E_LAYER + DR_E_RES2;
  if (blockIdx.x < m) {
    const int r = blockIdx.x;
    uint4 x = make_uint4(0, 0, 0, 0);
    if (tid < VECS) {
      uint4 y[1] = {};
      dr_wait_all<1>(p.res2 + r * (H / 2) + 4 * tid, 0, 1, last, y, p.polls, alive);
      x = y[0];
      __syncwarp();
      const float s = warp_sum(squares(x));
      if (lane == 0) sm.ssq[0][warp] = s;
    }
    dr_sync();
    if (tid < VECS) {
      const uint32_t* w4 = reinterpret_cast<const uint32_t*>(p.final_w) + 4 * tid;
      x = norm8(x, make_uint4(__ldg(w4), __ldg(w4 + 1), __ldg(w4 + 2), __ldg(w4 + 3)), rstd_of(warp_sum(lane < VECS / 32 ? sm.ssq[0][lane & 7] : 0.f)), EAGER);
      uint32_t* to = reinterpret_cast<uint32_t*>(p.out + r * p.out_stride) + 4 * tid;
      to[0] = x.x; to[1] = x.y; to[2] = x.z; to[3] = x.w;
    }
  }
  // ---- the last CTA to leave moves the phase number on: all have read it
  if (!alive) sm.lost = 1;
  __syncthreads();                                         // the copying warp too
  if (tid == 0) {
    if (sm.lost) {
      dr_report(p.waits);
    }
    __threadfence();
    const bool last_out = atomicAdd(p.sync + 1, 1u) == gridDim.x - 1;
    if (last_out) {
      p.sync[1] = 0;
      p.sync[0] = base > DR_LAST_BASE ? 0 : base + p.num_layers * DR_E_LAYER;
    }
    sm.plan.unit.L = last_out;
    __threadfence();
  }
  // Numbers would come again after 2^32 / 8 layers (four hours of steps), and words of rows that were not used meanwhile would be taken for theirs.  Before that the last
  // CTA writes zeros over all words, 5 MB, and numbers start anew.
  if (base > DR_LAST_BASE) {
    dr_sync();
    if (sm.plan.unit.L)
      for (uint64_t* at = p.qkv + tid; at < p.words_end; at += DR_READERS) *at = 0;
  }
}

// CTAs that a unit of attention may take
static int dr_parts(int m, int nsplit) {
  const int want = (nsplit + DR_PART_SPLITS - 1) / DR_PART_SPLITS, most = sm_count() / (m * DR_KVH);
  return want < most ? want : most;
}

struct DrSizes { size_t qkv, att, res, act, part, total; };
static DrSizes dr_sizes(int hidden, int inter) {
  DrSizes s{};
  auto words = [](size_t n) { return (n * 8 + 255) / 256 * 256; };
  s.qkv = words(static_cast<size_t>(DR_MAX_ROWS) * (DR_Q + 2 * DR_KV) / 2);
  s.att = words(static_cast<size_t>(DR_MAX_ROWS) * DR_Q / 2);
  s.res = words(static_cast<size_t>(DR_MAX_ROWS) * hidden / 2);
  s.act = words(static_cast<size_t>(DR_MAX_ROWS) * inter / 2);
  s.part = words(static_cast<size_t>(DR_MAX_ROWS) * DR_KVH * 32 * DR_GROUP * (2 + DR_HD));
  s.total = 256 + s.qkv + s.att + 2 * s.res + s.act + s.part;
  return s;
}

// The widths for which there is a kernel: the shipped ones, where gemm.cu cuts K as the instances do, no warp has more than DR_MAX_TILES of a phase
static int dr_form(int hidden, int q, int kv, int inter) {
  const int n = sm_count();
  if (q != DR_Q || kv != DR_KV || DR_MAX_ROWS * DR_KVH > n) return 0;
  auto fits = [&](int features, int k, int s) {
    const int all = features / 8, group = dr_group(all, n), tiles = (((all + group - 1) / group + n - 1) / n) * group;        // most of a CTA
    return gemm_splits(features, k, DR_MAX_ROWS) == s && (tiles + DR_WARPS / s - 1) / (DR_WARPS / s) <= DR_MAX_TILES && tiles * s <= DR_SUMS &&
           (tiles + 3) / 4 + 1 <= 32 / s;
  };
  const int width = q + 2 * kv;
  if ((2 * inter / 8 + dr_group(2 * inter / 8, n) - 1) / dr_group(2 * inter / 8, n) < n) return 0;        // tiles of gate_up for every CTA, see the head of this file
  if (!fits(width, hidden, 8) || !fits(hidden, q, 8) || !fits(hidden, inter, 8)) return 0;
  if (hidden == 2048 && inter == 6144 && fits(2 * inter, hidden, 2)) return 1;
  if (hidden == 1024 && inter == 3072 && fits(2 * inter, hidden, 4)) return 2;
  return 0;
}

template <int H, int I, int SQ, int SG, int ROWS, bool EAGER>
static int go_rows(const DrParams& p, cudaStream_t st) {
  auto kern = decode_rows_kernel<H, I, SQ, SG, ROWS, EAGER>;
  constexpr int smem = static_cast<int>(sizeof(DrShared<H, I, ROWS>));
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return cuda_fail(e, "decode_rows(smem attr)");
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(sm_count(), 1, 1);
  cfg.blockDim = dim3(DR_THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;                                    // every CTA polls its peers' words: all of them must be resident
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, kern, p);
  count_launch();
  return e != cudaSuccess ? cuda_fail(e, "decode_rows") : B2TTS_OK;
}

// The multiprocessors that a launch on this stream (null: of the current context) gets: a green context has fewer than the device
static int dr_multiprocessors(cudaStream_t st) {
  auto entry = [](const char* name) -> void* {
    void* at = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint(name, &at, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess) at = nullptr;
    cudaGetLastError();
    return at;
  };
  static const auto green_of = reinterpret_cast<decltype(&cuStreamGetGreenCtx)>(entry("cuStreamGetGreenCtx"));
  static const auto green_has = reinterpret_cast<decltype(&cuGreenCtxGetDevResource)>(entry("cuGreenCtxGetDevResource"));
  static const auto current = reinterpret_cast<decltype(&cuCtxGetCurrent)>(entry("cuCtxGetCurrent"));
  static const auto context_has = reinterpret_cast<decltype(&cuCtxGetDevResource)>(entry("cuCtxGetDevResource"));
  CUdevResource r{};
  CUgreenCtx green = nullptr;
  if (st != nullptr && green_of != nullptr && green_has != nullptr && green_of(st, &green) == CUDA_SUCCESS && green != nullptr)
    return green_has(green, &r, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS ? static_cast<int>(r.sm.smCount) : 0;
  CUcontext c = nullptr;
  if (current == nullptr || context_has == nullptr || current(&c) != CUDA_SUCCESS || c == nullptr || context_has(c, &r, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS) return sm_count();
  return static_cast<int>(r.sm.smCount);
}

// Whether a CTA fits a multiprocessor: asked once for each number of rows (a device that this library runs on is an sm_100a like another), and only for those that
// steps have, since asking loads the kernel
template <int H, int I, int SQ, int SG, int ROWS>
static bool dr_one_fits() {
  static const bool fits = [] {
    constexpr int smem = static_cast<int>(sizeof(DrShared<H, I, ROWS>));
    auto kern = decode_rows_kernel<H, I, SQ, SG, ROWS, true>;             // the other rounding has the same registers and shared memory
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, DR_THREADS, smem) == cudaSuccess)
      return n >= 1;
    cudaGetLastError();
    return false;
  }();
  return fits;
}
// Whether a CTA can be resident on every multiprocessor at once, as the launch wants (without a device: as if so)
static bool dr_resident(int form, int m, cudaStream_t st) {
  int dev = 0, cooperative = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  if (cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || cooperative == 0) return false;
  const bool fits = form == 1 ? (m <= 2 ? dr_one_fits<2048, 6144, 8, 2, 2>() : dr_one_fits<2048, 6144, 8, 2, 4>())
                              : m <= 2 ? dr_one_fits<1024, 3072, 8, 4, 2>() : m <= 4 ? dr_one_fits<1024, 3072, 8, 4, 4>() : dr_one_fits<1024, 3072, 8, 4, DR_MAX_ROWS>();
  return fits && dr_multiprocessors(st) >= sm_count();
}

}  // namespace b2

namespace b2 {
// The kernel for these rows and widths (dr_form), or 0
static int dr_form_for(int m, int hidden, int q_size, int kv_size, int intermediate) {
  // Every CTA reads all rows of an activation, twice their size with the flags: what hand-overs take grows with the rows, what separate launches take hardly
  // does.  Separate launches / this, us: talker of 28 layers, contexts of 97 and of 400 tokens, 1 row 1241 1386 / 825 955, 2 rows 1268 1430 / 918 1059,
  // 4 rows 1321 1453 / 1047 1183, 5 rows 1343 1450 / 1280 1422, 6 rows 1322 1460 / 1342 1488, 8 rows 1333 1467 / 1410 1684; predictor of 5 layers with its head
  // 1 row 170 / 117, 4 rows 175 / 136, 6 rows 177 / 151, 8 rows 179 / 160.
  const int form = dr_form(hidden, q_size, kv_size, intermediate);
  return form != 0 && m >= 1 && m <= (form == 1 ? 4 : DR_MAX_ROWS) ? form : 0;
}
}  // namespace b2

extern "C" int b2tts_decode_rows_supported(int m, int hidden, int q_size, int kv_size, int intermediate) {
  const int form = b2::dr_form_for(m, hidden, q_size, kv_size, intermediate);
  return form != 0 && b2::dr_resident(form, m, nullptr);
}
extern "C" int b2tts_decode_rows_taken(int m, int max_context_len, int hidden, int q_size, int kv_size, int intermediate, void* stream) {
  using namespace b2;
  // ... and what attention takes grows with the contexts, by one chain of tiles after another where a CTA has more splits than it can walk at once (DR_PART_SPLITS).  So
  // the tables' room decides: no CTA has a second turn.  28 layers, contexts that fill the tables, separate launches / this in us, the last size that is taken and the first one
  // that is not: 2048 wide, 3 rows 1536 1435 / 1341, 2048 1475 / 1593; 4 rows 1024 1404 / 1292, 1536 1449 / 1527; 1024 wide, 4 rows 1024 1090 / 882, 1536 1142 / 1111; 6 rows
  // 768 1085 / 914, 1024 1105 / 1123; 8 rows 512 1064 / 910, 768 1094 / 1115.  Up to 2 rows have the CTAs for any context: 2048 wide 4000 1741 / 1522, 16000 3339 / 2789.
  // Tables of 16384 with 4 rows behind 16000 tokens 3382 / 4479, 1024 wide with 8 rows 3167 / 7012; the same behind 100 tokens 1278 / 1233 and 1014 / 920.
  const int form = dr_form_for(m, hidden, q_size, kv_size, intermediate);
  if (max_context_len <= 0 || form == 0) return 0;
  const int nsplit = fa_choose_nsplit(m, max_context_len);
  return nsplit <= DR_PART_SPLITS * dr_parts(m, nsplit) && dr_resident(form, m, static_cast<cudaStream_t>(stream));
}
extern "C" size_t b2tts_decode_rows_workspace_bytes(int hidden, int q_size, int kv_size, int intermediate) {
  return b2::dr_form(hidden, q_size, kv_size, intermediate) != 0 ? b2::dr_sizes(hidden, intermediate).total : 0;
}
extern "C" int b2tts_decode_rows_polls(const void* x, int64_t x_row_stride, void* out, int64_t out_row_stride, const b2tts_stack_layer* layers, int num_layers,
                                 const void* final_norm_weight, int m, int hidden, int num_heads, int num_kv_heads, int head_dim, int intermediate,
                                 float eps, int rounding, const int64_t* positions, int64_t pos_row_stride, const float* inv_freq, const int32_t* modality,
                                 float attention_scaling, const int32_t* slot_mapping, const int32_t* block_table, int bt_stride,
                                 const int32_t* context_lens, int page_size, int max_context_len, float scale, void* workspace, size_t workspace_bytes,
                                 int polls, void* stream) {
  using namespace b2;
  const char* what = "decode_rows";
  if (m == 0) return B2TTS_OK;
  B2_REQUIRE(layers && num_layers >= 1 && num_layers <= DR_MAX_LAYERS, B2TTS_EUNSUPPORTED, "%s: 1..%d layers", what, DR_MAX_LAYERS);
  B2_REQUIRE(head_dim == DR_HD && num_kv_heads >= 1 && num_heads == DR_GROUP * num_kv_heads, B2TTS_EUNSUPPORTED,
             "%s: head_dim %d / heads %d / kv heads %d unsupported (128, heads = 2 x kv heads)", what, head_dim, num_heads, num_kv_heads);
  const int Q = num_heads * head_dim, KV = num_kv_heads * head_dim, form = dr_form_for(m, hidden, Q, KV, intermediate);
  B2_REQUIRE(form != 0, B2TTS_EUNSUPPORTED, "%s: %d rows of widths %d / %d / %d", what, m, hidden, Q, intermediate);
  B2_REQUIRE(x && out && final_norm_weight && positions && inv_freq && slot_mapping && block_table && context_lens && workspace, B2TTS_EINVAL,
             "%s: null pointer", what);
  B2_REQUIRE(rounding == B2TTS_ROUND_EAGER || rounding == B2TTS_ROUND_FUSED, B2TTS_EINVAL, "%s: rounding %d", what, rounding);
  B2_REQUIRE(page_size > 0 && bt_stride > 0 && max_context_len > 0, B2TTS_EINVAL, "%s: page_size=%d bt_stride=%d max_context_len=%d", what, page_size, bt_stride,
             max_context_len);
  B2_REQUIRE((page_size & (page_size - 1)) == 0 && page_size % FA_TILE == 0, B2TTS_EUNSUPPORTED, "%s: pages of %d tokens (a power of two, %d or more)", what, page_size,
             FA_TILE);
  auto word = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 3u) == 0; };
  B2_REQUIRE(word(x) && word(out) && word(final_norm_weight) && x_row_stride % 2 == 0 && out_row_stride % 2 == 0 &&
                 (reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, B2TTS_EALIGN, "%s: rows must be 4-byte, the workspace 256-byte aligned", what);
  const DrSizes z = dr_sizes(hidden, intermediate);
  B2_REQUIRE(workspace_bytes >= z.total, B2TTS_EWORKSPACE, "%s: workspace %zu B too small", what, workspace_bytes);
  const int lost = wait_check(WAITS_ROWS, what);
  if (lost != B2TTS_OK) return lost;
  DrParams p{};
  for (int l = 0; l < num_layers; ++l) {
    const b2tts_stack_layer& s = layers[l];
    B2_REQUIRE(s.qkv_w && s.o_w && s.gate_up_w && s.down_w && s.input_norm_w && s.post_norm_w && s.k_cache && s.v_cache, B2TTS_EINVAL,
               "%s: layer %d null pointer", what, l);
    B2_REQUIRE(aligned16(s.qkv_w) && aligned16(s.o_w) && aligned16(s.gate_up_w) && aligned16(s.down_w) && aligned16(s.k_cache) && aligned16(s.v_cache) &&
                   word(s.input_norm_w) && word(s.post_norm_w) && word(s.q_norm_w) && word(s.k_norm_w), B2TTS_EALIGN, "%s: layer %d alignment", what, l);
    DrLayer& d = p.layer[l];
    d.w_qkv = static_cast<const uint8_t*>(s.qkv_w); d.w_o = static_cast<const uint8_t*>(s.o_w);
    d.w_gu = static_cast<const uint8_t*>(s.gate_up_w); d.w_down = static_cast<const uint8_t*>(s.down_w);
    d.ln_in = static_cast<const __nv_bfloat16*>(s.input_norm_w); d.ln_post = static_cast<const __nv_bfloat16*>(s.post_norm_w);
    d.qn_w = static_cast<const __nv_bfloat16*>(s.q_norm_w); d.kn_w = static_cast<const __nv_bfloat16*>(s.k_norm_w);
    d.k_cache = static_cast<__nv_bfloat16*>(s.k_cache); d.v_cache = static_cast<__nv_bfloat16*>(s.v_cache);
  }
  p.num_layers = num_layers; p.m = m;
  p.x_in = static_cast<const __nv_bfloat16*>(x); p.x_stride = x_row_stride;
  p.out = static_cast<__nv_bfloat16*>(out); p.out_stride = out_row_stride;
  p.final_w = static_cast<const __nv_bfloat16*>(final_norm_weight);
  p.eps = eps;
  p.positions = positions; p.pos_row_stride = pos_row_stride; p.inv_freq = inv_freq; p.modality = modality;
  p.attention_scaling = attention_scaling; p.scale_log2 = scale * 1.4426950408889634f;
  p.slot_mapping = slot_mapping; p.block_table = block_table; p.bt_stride = bt_stride; p.context_lens = context_lens;
  while ((1 << p.page_shift) < page_size) ++p.page_shift;
  p.nsplit = fa_choose_nsplit(m, max_context_len);
  p.max_parts = dr_parts(m, p.nsplit);
  uint8_t* w = static_cast<uint8_t*>(workspace);
  auto take = [&w](size_t n) { uint64_t* at = reinterpret_cast<uint64_t*>(w); w += n; return at; };
  p.sync = reinterpret_cast<unsigned*>(take(256));
  p.qkv = take(z.qkv); p.att = take(z.att); p.res1 = take(z.res); p.res2 = take(z.res); p.act = take(z.act); p.part = take(z.part); p.words_end = take(0);
  p.waits = wait_word(WAITS_ROWS);
  p.polls = polls;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool eager = rounding == B2TTS_ROUND_EAGER;
  // few rows leave the ring more room: instances for 2, 4 and 8
  auto go = [&](auto rows) -> int {
    constexpr int R = decltype(rows)::value;
    if constexpr (R <= 4) {
      if (form == 1) return eager ? go_rows<2048, 6144, 8, 2, R, true>(p, st) : go_rows<2048, 6144, 8, 2, R, false>(p, st);
    }
    return eager ? go_rows<1024, 3072, 8, 4, R, true>(p, st) : go_rows<1024, 3072, 8, 4, R, false>(p, st);
  };
  return m <= 2 ? go(std::integral_constant<int, 2>{}) : m <= 4 ? go(std::integral_constant<int, 4>{}) : go(std::integral_constant<int, DR_MAX_ROWS>{});
}
extern "C" int b2tts_decode_rows(const void* x, int64_t x_row_stride, void* out, int64_t out_row_stride, const b2tts_stack_layer* layers, int num_layers,
                                 const void* final_norm_weight, int m, int hidden, int num_heads, int num_kv_heads, int head_dim, int intermediate,
                                 float eps, int rounding, const int64_t* positions, int64_t pos_row_stride, const float* inv_freq, const int32_t* modality,
                                 float attention_scaling, const int32_t* slot_mapping, const int32_t* block_table, int bt_stride,
                                 const int32_t* context_lens, int page_size, int max_context_len, float scale, void* workspace, size_t workspace_bytes,
                                 void* stream) {
  return b2tts_decode_rows_polls(x, x_row_stride, out, out_row_stride, layers, num_layers, final_norm_weight, m, hidden, num_heads, num_kv_heads, head_dim, intermediate, eps,
                                 rounding, positions, pos_row_stride, inv_freq, modality, attention_scaling, slot_mapping, block_table, bt_stride, context_lens, page_size,
                                 max_context_len, scale, workspace, workspace_bytes, b2::DR_POLLS, stream);
}

namespace b2 {
// One wait for a word that nobody writes, with a short limit
__device__ uint64_t g_rows_unwritten = 0;
__global__ void rows_lost_wait_kernel(int* word) {
  bool alive = true;
  dr_wait(&g_rows_unwritten, 1u, 64, alive);
  if (!alive && threadIdx.x == 0) dr_report(word);
}
}  // namespace b2

extern "C" int b2tts_decode_rows_timeouts(void) { return b2::wait_count(b2::WAITS_ROWS); }
extern "C" int b2tts_decode_rows_lose_wait(void* stream) {
  using namespace b2;
  int* word = wait_word(WAITS_ROWS);
  B2_REQUIRE(word != nullptr, B2TTS_ECUDA, "decode_rows_lose_wait: no host memory");
  rows_lost_wait_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(word);
  B2_CHECK_LAUNCH("decode_rows_lose_wait");
  return B2TTS_OK;
}
