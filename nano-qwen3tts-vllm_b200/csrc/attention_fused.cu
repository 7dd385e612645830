// attention_fused.cu - the decode step of Qwen3TTSAttention.forward (models/qwen3_tts_share.py:96-109)
// as ONE kernel: per-head q/k RMSNorm + RoPE (layers/rotary_embedding.py:11-212), the paged KV write of
// the new token (store_kvcache, layers/attention.py:10-54), the block_table paged GQA attention
// (flash_attn_with_kvcache, attention.py:92-95) and the split-KV combine.  The separate
// qknorm_rope_kvwrite / paged_attn / attn_combine launches of the decode path collapse into this one.
//
// Same HBM design as attention.cu: one CTA per (sequence, KV split) covers all kv heads; a producer
// warp streams 8-token K and V tiles (all heads of a token are contiguous in the page) with 1-D bulk
// async copies into a 3-stage mbarrier ring; consumer warp w owns kv head w and its GROUP q heads.
// Fusion:
//   * prologue: the consumer warps run the arithmetic of qknorm_rope_kvwrite_kernel (norm_rope.cu; same
//     lane mapping, rounding points and summation order, so K cache bytes are identical to the unfused
//     path) on the one new token: q heads go to shared memory; the split that owns the sequence's last
//     tile also normalises + rotates k, writes it and the raw v to cache[slot] and keeps a copy in
//     shared memory: when the last tile lands, each warp overwrites its head's slice of the new token's
//     row with that copy, so it never depends on reading its own global write;
//   * combine: split partials go to the workspace; the LAST CTA of a sequence to finish (atomic
//     ticket) folds them in split order - deterministic - and resets the ticket for the next launch.
#include <stdlib.h>

#include "fused_attn.cuh"

namespace b2 {

constexpr int FA_HD = 128;
constexpr int FA_NSTAGE = 3;
// The per-row split-KV tickets live in a FIXED span at the start of the workspace, whatever the batch size of the
// launch: one workspace serves every batch size / graph of a runner, and the partial accumulators of one launch
// must never land on the (always-zero-between-launches) tickets another launch will read.
constexpr int FA_MAX_ROWS = 4096;
constexpr size_t FA_TICKET_BYTES = (size_t)FA_MAX_ROWS * sizeof(int);

struct FusedAttnParams {
  const __nv_bfloat16 *q, *k, *v;          // rows of the QKV projection
  int64_t q_stride, k_stride, v_stride;
  const __nv_bfloat16 *q_w, *k_w;          // head-norm weights [128]
  float eps;
  const int64_t* positions;                // [rows] or [3][rows]
  int64_t pos_row_stride;
  const float* inv_freq;                   // [64]
  const int32_t* modality;                 // [128] or null
  float attention_scaling;
  const int32_t* slot_mapping;             // [rows]
  __nv_bfloat16 *k_cache, *v_cache;        // [pages, page, kvh, 128]
  const int32_t* block_table;
  int bt_stride, page_size;
  const int32_t* context_lens;
  __nv_bfloat16* out;                      // [rows, heads*128]
  float* part_acc;                         // [rows, nsplit, heads, 128]
  float* part_ml;                          // [rows, nsplit, heads, 2]
  int* tickets;                            // [rows], zero between launches
  int nsplit, num_heads, num_kv_heads;
  float scale_log2;
};

__device__ __forceinline__ uint4 fa_pack8(const float* f) {
  uint4 r;
  r.x = pack_bf16(f[0], f[1]); r.y = pack_bf16(f[2], f[3]); r.z = pack_bf16(f[4], f[5]); r.w = pack_bf16(f[6], f[7]);
  return r;
}

// The splits of a sequence in order, by its last CTA to finish.  Not inline: its registers would be taken from the loop over tiles (32 rows of 2000 tokens, two query and two key
// heads 28.6 us inline, 19.2 so; 8 and 2 heads 41, 33).
template <int GROUP>
__device__ __noinline__ void fa_fold(const float* part_ml, const float* part_acc, __nv_bfloat16* out, int nsplit, int num_heads, int row, int head0) {
  const int lane = threadIdx.x & 31;
  // warp w folds heads head0 .. head0+GROUP-1; lane owns 4 consecutive dims.  Lane s asks for split s's maximum and sum (at most 32 splits), and the partials of
  // four splits of all heads are asked for at once: a split after another was up to three dependent round trips for each: 64 rows of 40
  // tokens 10.4 -> 8.5 us, of 200 16.1 -> 14.7, 16 rows of 700 22.3 -> 15.9, 4 of 2000 25.7 -> 18.4 (16 query and 8 key heads).
  float top[GROUP], sum[GROUP];
#pragma unroll
  for (int h = 0; h < GROUP; ++h) {
    const int64_t at = ((int64_t)row * nsplit + lane) * num_heads + head0 + h;
    top[h] = lane < nsplit ? __ldcg(part_ml + at * 2) : -INFINITY;
    sum[h] = lane < nsplit ? __ldcg(part_ml + at * 2 + 1) : 0.f;
  }
  float4 num[GROUP];
  float den[GROUP];
#pragma unroll
  for (int h = 0; h < GROUP; ++h) { num[h] = make_float4(0.f, 0.f, 0.f, 0.f); den[h] = 0.f; }
  for (int s0 = 0; s0 < nsplit; s0 += 4) {
    float4 a[4][GROUP];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int h = 0; h < GROUP; ++h) {
        const int64_t idx = ((int64_t)row * nsplit + s0 + u) * num_heads + head0 + h;
        a[u][h] = s0 + u < nsplit ? __ldcg(reinterpret_cast<const float4*>(part_acc + idx * FA_HD) + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    if (s0 == 0) {
#pragma unroll
      for (int h = 0; h < GROUP; ++h) top[h] = fa_exp2(top[h] - warp_max(top[h]));          // the splits' weights
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int h = 0; h < GROUP; ++h) {
        const float w = __shfl_sync(0xffffffffu, top[h], (s0 + u) & 31), ls = __shfl_sync(0xffffffffu, sum[h], (s0 + u) & 31);
        if (s0 + u < nsplit && ls > 0.f) {
          num[h].x = fmaf(w, a[u][h].x, num[h].x); num[h].y = fmaf(w, a[u][h].y, num[h].y);
          num[h].z = fmaf(w, a[u][h].z, num[h].z); num[h].w = fmaf(w, a[u][h].w, num[h].w);
          den[h] = fmaf(w, ls, den[h]);
        }
      }
  }
#pragma unroll
  for (int h = 0; h < GROUP; ++h) {
    const float inv = den[h] > 0.f ? 1.f / den[h] : 0.f;
    uint2 o;
    o.x = pack_bf16(num[h].x * inv, num[h].y * inv);
    o.y = pack_bf16(num[h].z * inv, num[h].w * inv);
    stg_v2(out + ((int64_t)row * num_heads + head0 + h) * FA_HD + 4 * lane, o);
  }
}

// HEADS: as many key heads at most, see fa_pick()
template <int GROUP, bool EAGER, bool SPLIT, int HEADS>
__global__ void __launch_bounds__(GROUP == 4 ? 32 * (HEADS + 1) : 288, GROUP < 4 || HEADS > 4 ? 2 : HEADS > 2 ? 3 : 4)
fused_decode_attn_kernel(const FusedAttnParams p) {
  constexpr int UNROLL = GROUP == 2 && (!SPLIT || HEADS <= 4) ? FA_NSTAGE : 1;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const int kvh = p.num_kv_heads;
  const int kv_dim = kvh * FA_HD;
  const int stage_elems = FA_TILE * kv_dim;
  __nv_bfloat16* Ks = reinterpret_cast<__nv_bfloat16*>(smem_raw);
  __nv_bfloat16* Vs = Ks + FA_NSTAGE * stage_elems;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(Vs + FA_NSTAGE * stage_elems);
  uint64_t* empty_bar = full_bar + FA_NSTAGE;
  int* last_flag = reinterpret_cast<int*>(empty_bar + FA_NSTAGE);
  __nv_bfloat16* q_s = reinterpret_cast<__nv_bfloat16*>(last_flag + 4);     // [heads][128] normed + rotated q
  __nv_bfloat16* kn_s = q_s + p.num_heads * FA_HD;                          // [kvh][128] the new token's K
  __nv_bfloat16* vn_s = kn_s + kv_dim;                                      // [kvh][128] the new token's V

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x;
  const int split = blockIdx.y;

  pdl_launch();
  if (threadIdx.x == 0) {
    for (int s = 0; s < FA_NSTAGE; ++s) {
      mbar_init(full_bar + s, 1);
      mbar_init(empty_bar + s, kvh);
    }
    mbar_fence_init();
  }
  // Latency discipline: this kernel runs 103 times per codec frame on contexts of 3 .. a few hundred tokens, so
  // its cost is the chain of dependent global-memory round trips, not bytes.  Everything that does not depend on
  // the previous kernel (rotary frequencies, M-RoPE row selectors, head-norm weights) is requested BEFORE
  // griddepcontrol.wait; everything that does (length, slot, positions, the q/k/v rows, the block table) is
  // requested in ONE batch right after it, so the prologue costs one round trip instead of six.
  const int g = lane >> 3;        // token slot within a 4-token step
  const int j = lane & 7;         // which 16 head-dims: [8j,8j+8) and [64+8j,64+8j+8)
  const bool consumer = warp < kvh;
  float frq[2] = {0.f, 0.f};
  int md1[2] = {0, 0}, md2[2] = {0, 0};
  uint32_t qw1 = 0, qw2 = 0, kw1 = 0, kw2 = 0;
  if (consumer) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int fi = 2 * lane + e;
      frq[e] = __ldg(p.inv_freq + fi);
      if (p.modality) { md1[e] = __ldg(p.modality + fi); md2[e] = __ldg(p.modality + FA_HD / 2 + fi); }
    }
    if (p.q_w) { qw1 = *reinterpret_cast<const uint32_t*>(p.q_w + 2 * lane); qw2 = *reinterpret_cast<const uint32_t*>(p.q_w + 64 + 2 * lane); }
    if (p.k_w) { kw1 = *reinterpret_cast<const uint32_t*>(p.k_w + 2 * lane); kw2 = *reinterpret_cast<const uint32_t*>(p.k_w + 64 + 2 * lane); }
  }
  __syncthreads();
  pdl_wait();                                   // q/k/v rows, slots and lengths come from earlier kernels

  const bool writer = (split == p.nsplit - 1);  // owns the last tile, i.e. the token appended this step
  int L = __ldg(p.context_lens + row);
  // ---- one batch of independent requests (consumers: this token's rows; producer: the block-table row)
  int tbl = 0;                                  // producer: lane l holds block_table[row][l]
  int slot = -1;
  int64_t pos[3] = {0, 0, 0};
  uint32_t raw1[GROUP + 1], raw2[GROUP + 1];
  uint4 vraw = make_uint4(0, 0, 0, 0);
  const int nh_q = p.num_heads / kvh;           // q heads this warp normalises: warp, warp + kvh, ...  (== GROUP)
  if (consumer) {
    if (writer) slot = __ldg(p.slot_mapping + row);
    pos[0] = __ldg(p.positions + row);
    if (p.modality && p.pos_row_stride) {
      pos[1] = __ldg(p.positions + p.pos_row_stride + row);
      pos[2] = __ldg(p.positions + 2 * p.pos_row_stride + row);
    } else {
      pos[1] = pos[2] = pos[0];
    }
#pragma unroll
    for (int i = 0; i < GROUP + 1; ++i) {
      const bool is_k = i == GROUP;
      raw1[i] = raw2[i] = 0u;
      if (i < nh_q || (is_k && writer)) {
        const __nv_bfloat16* src = is_k ? p.k + (int64_t)row * p.k_stride + warp * FA_HD
                                        : p.q + (int64_t)row * p.q_stride + (warp + i * kvh) * FA_HD;
        raw1[i] = *reinterpret_cast<const uint32_t*>(src + 2 * lane);
        raw2[i] = *reinterpret_cast<const uint32_t*>(src + 64 + 2 * lane);
      }
    }
    if (writer && (int)threadIdx.x < (kv_dim >> 3)) vraw = ldg_v4(p.v + (int64_t)row * p.v_stride + 8 * threadIdx.x);
  } else if (lane < p.bt_stride) {
    tbl = __ldg(p.block_table + (int64_t)row * p.bt_stride + lane);
  }
  if (L < 0) L = 0;
  const int n_tiles = (L + FA_TILE - 1) / FA_TILE;
  const int t_begin = (int)(((int64_t)split * n_tiles) / p.nsplit);
  const int t_end = (int)(((int64_t)(split + 1) * n_tiles) / p.nsplit);
  const int my_tiles = t_end - t_begin;

  if (warp == kvh) {
    // =========================== producer warp: the whole warp walks the ring (the page of a tile comes from the
    // lanes' copy of the block-table row), lane 0 issues the copies
    for (int i = 0; i < my_tiles; ++i) {
      const int stage = i % FA_NSTAGE;
      const uint32_t ph = (i / FA_NSTAGE) & 1;
      const int tok0 = (t_begin + i) * FA_TILE;
      const int pidx = tok0 / p.page_size;
      int page = __shfl_sync(0xffffffffu, tbl, pidx & 31);
      if (pidx >= 32) page = __ldg(p.block_table + (int64_t)row * p.bt_stride + pidx);
      if (lane == 0) {
        mbar_wait(empty_bar + stage, ph ^ 1);
        const int ntok = min(FA_TILE, L - tok0);
        if (page < 0) page = 0;                  // never faults on a stale (-1) table entry
        const int64_t slot0 = (int64_t)page * p.page_size + tok0 % p.page_size;
        const uint32_t bytes = (uint32_t)(ntok * kv_dim * 2);
        mbar_expect_tx(full_bar + stage, 2u * bytes);
        bulk_g2s(Ks + stage * stage_elems, p.k_cache + slot0 * kv_dim, bytes, full_bar + stage);
        bulk_g2s(Vs + stage * stage_elems, p.v_cache + slot0 * kv_dim, bytes, full_bar + stage);
      }
      __syncwarp();
    }
    return;
  }

  // =========================== consumer warps
  const int head0 = warp * GROUP;

  if (L == 0) {                   // CUDA-graph padding row (talker_mode_runner.py:97-100): zeros, no ticket
    if (split == 0 && g == 0) {
#pragma unroll
      for (int h = 0; h < GROUP; ++h) {
        __nv_bfloat16* o = p.out + ((int64_t)row * p.num_heads + head0 + h) * FA_HD;
        stg_v4(o + 8 * j, make_uint4(0, 0, 0, 0));
        stg_v4(o + 64 + 8 * j, make_uint4(0, 0, 0, 0));
      }
    }
    return;
  }

  // ---- prologue: the body of qknorm_rope_kvwrite_kernel (norm_rope.cu) for this one token, same lane
  // mapping and arithmetic (lane l holds dims {2l, 2l+1, 64+2l, 64+2l+1}; a warp walks heads warp,
  // warp+kvh, ...): q heads -> shared memory, and on the writer split k (normed + rotated) and v (raw)
  // -> cache[slot] and shared memory.
  {
    float cf[2][2], sf[2][2];                             // [column half][dim 2l, 2l + 1]
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float a1 = (float)(md1[e] == 0 ? pos[0] : md1[e] == 1 ? pos[1] : pos[2]) * frq[e];
      cf[0][e] = cosf(a1) * p.attention_scaling;
      sf[0][e] = sinf(a1) * p.attention_scaling;
      cf[1][e] = cf[0][e];
      sf[1][e] = sf[0][e];
      if (md2[e] != md1[e]) {
        const float a2 = (float)(md2[e] == 0 ? pos[0] : md2[e] == 1 ? pos[1] : pos[2]) * frq[e];
        cf[1][e] = cosf(a2) * p.attention_scaling;
        sf[1][e] = sinf(a2) * p.attention_scaling;
      }
    }
    const uint32_t c1 = pack_bf16(cf[0][0], cf[0][1]), s1 = pack_bf16(sf[0][0], sf[0][1]), c2 = pack_bf16(cf[1][0], cf[1][1]), s2 = pack_bf16(sf[1][0], sf[1][1]);
#pragma unroll
    for (int i = 0; i < GROUP + 1; ++i) {
      const bool is_k = i == GROUP;
      if (!(i < nh_q || (is_k && writer))) continue;
      const int h = is_k ? warp : warp + i * kvh;
      const bool has_w = is_k ? (p.k_w != nullptr) : (p.q_w != nullptr);
      uint32_t x1 = raw1[i], x2 = raw2[i];
      if (has_w) {
        float ss = bf16lo(x1) * bf16lo(x1);
        ss = fmaf(bf16hi(x1), bf16hi(x1), ss); ss = fmaf(bf16lo(x2), bf16lo(x2), ss); ss = fmaf(bf16hi(x2), bf16hi(x2), ss);
        const float var = warp_sum(ss) / (float)FA_HD + p.eps;
        const float rstd = EAGER ? 1.0f / sqrtf(var) : rsqrtf(var);
        x1 = norm_pair<EAGER>(x1, rstd, is_k ? kw1 : qw1);
        x2 = norm_pair<EAGER>(x2, rstd, is_k ? kw2 : qw2);
      }
      const uint32_t y1 = turn_first(x1, x2, c1, s1), y2 = turn_second(x1, x2, c2, s2);
      __nv_bfloat16* dst = is_k ? kn_s + h * FA_HD : q_s + h * FA_HD;
      *reinterpret_cast<uint32_t*>(dst + 2 * lane) = y1;
      *reinterpret_cast<uint32_t*>(dst + 64 + 2 * lane) = y2;
      if (is_k && slot >= 0) {
        __nv_bfloat16* cd = p.k_cache + (int64_t)slot * kv_dim + h * FA_HD;
        *reinterpret_cast<uint32_t*>(cd + 2 * lane) = y1;
        *reinterpret_cast<uint32_t*>(cd + 64 + 2 * lane) = y2;
      }
    }
    if (writer && (int)threadIdx.x < (kv_dim >> 3)) {      // V goes to the cache untouched
      *reinterpret_cast<uint4*>(vn_s + 8 * threadIdx.x) = vraw;
      if (slot >= 0) stg_v4(p.v_cache + (int64_t)slot * kv_dim + 8 * threadIdx.x, vraw);
    }
  }
  asm volatile("bar.sync 1, %0;" :: "r"(kvh * 32) : "memory");      // the consumer warps only

  // a tile in its stage, with the new token in its place: tokens, keys and values of this warp's key head
  auto enter = [&](int i, __nv_bfloat16*& kt, __nv_bfloat16*& vt) -> int {
    const int stage = i % FA_NSTAGE;
    const uint32_t ph = (i / FA_NSTAGE) & 1;
    const int tok0 = (t_begin + i) * FA_TILE;
    const int ntok = min(FA_TILE, L - tok0);
    mbar_wait(full_bar + stage, ph);
    kt = Ks + stage * stage_elems + warp * FA_HD;
    vt = Vs + stage * stage_elems + warp * FA_HD;
    if (writer && i == my_tiles - 1) {
      // the bulk copy may have read the new token's row before or after the global store above:
      // replace this head's slice of that row with the register copy
      if (g == 0) {
        __nv_bfloat16* kr = kt + (L - 1 - tok0) * kv_dim;
        __nv_bfloat16* vr = vt + (L - 1 - tok0) * kv_dim;
        const __nv_bfloat16* kn = kn_s + warp * FA_HD;
        const __nv_bfloat16* vn = vn_s + warp * FA_HD;
        *reinterpret_cast<uint4*>(kr + 8 * j) = *reinterpret_cast<const uint4*>(kn + 8 * j);
        *reinterpret_cast<uint4*>(kr + 64 + 8 * j) = *reinterpret_cast<const uint4*>(kn + 64 + 8 * j);
        *reinterpret_cast<uint4*>(vr + 8 * j) = *reinterpret_cast<const uint4*>(vn + 8 * j);
        *reinterpret_cast<uint4*>(vr + 64 + 8 * j) = *reinterpret_cast<const uint4*>(vn + 64 + 8 * j);
      }
      __syncwarp();
    }
    return ntok;
  };
  auto leave = [&](int i) {
    __syncwarp();
    if (lane == 0) mbar_arrive(empty_bar + i % FA_NSTAGE);
  };

  // ---- this warp's q heads from shared memory, pre-scaled for exp2, against its tiles
  float m[GROUP], l[GROUP], acc[GROUP][16];
  if constexpr (GROUP < 4) {
    uint64_t qv[GROUP][8];
#pragma unroll
    for (int h = 0; h < GROUP; ++h) {
      const __nv_bfloat16* qp = q_s + (head0 + h) * FA_HD;
      fa_pairs8(*reinterpret_cast<const uint4*>(qp + 8 * j), qv[h]);
      fa_pairs8(*reinterpret_cast<const uint4*>(qp + 64 + 8 * j), qv[h] + 4);
#pragma unroll
      for (int d = 0; d < 8; ++d) qv[h][d] = f2_mul(qv[h][d], f2_pack(p.scale_log2, p.scale_log2));
    }

    uint64_t acc2[GROUP][8];                                // weighted sums of values, in pairs
#pragma unroll
    for (int h = 0; h < GROUP; ++h) {
      m[h] = -INFINITY; l[h] = 0.f;
#pragma unroll
      for (int d = 0; d < 8; ++d) acc2[h][d] = 0;
    }

#pragma unroll UNROLL
    for (int i = 0; i < my_tiles; ++i) {
      __nv_bfloat16 *kt, *vt;
      const int ntok = enter(i, kt, vt);
      // Keys of all token slots, their products, then the values on their way while the products are summed over lanes and turned into weights
      float s[FA_TILE / 4][GROUP];
      uint4 raw[FA_TILE / 4][2];
      int at[FA_TILE / 4];
#pragma unroll
      for (int it = 0; it < FA_TILE / 4; ++it) {
        const int tok = it * 4 + g;
        at[it] = (tok < ntok ? tok : 0) * kv_dim + 8 * j;
        raw[it][0] = *reinterpret_cast<const uint4*>(kt + at[it]);
        raw[it][1] = *reinterpret_cast<const uint4*>(kt + at[it] + 64);
      }
#pragma unroll
      for (int it = 0; it < FA_TILE / 4; ++it) {
        uint64_t kf[8];
        fa_pairs8(raw[it][0], kf);
        fa_pairs8(raw[it][1], kf + 4);
#pragma unroll
        for (int h = 0; h < GROUP; ++h) s[it][h] = fa_dot16(qv[h], kf);
      }
#pragma unroll
      for (int it = 0; it < FA_TILE / 4; ++it) {
        raw[it][0] = *reinterpret_cast<const uint4*>(vt + at[it]);
        raw[it][1] = *reinterpret_cast<const uint4*>(vt + at[it] + 64);
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1)
#pragma unroll
        for (int it = 0; it < FA_TILE / 4; ++it)
#pragma unroll
          for (int h = 0; h < GROUP; ++h) s[it][h] += __shfl_xor_sync(0xffffffffu, s[it][h], o);
#pragma unroll
      for (int it = 0; it < FA_TILE / 4; ++it)
#pragma unroll
        for (int h = 0; h < GROUP; ++h) s[it][h] = it * 4 + g < ntok ? s[it][h] : -INFINITY;
      float alpha[GROUP];
#pragma unroll
      for (int h = 0; h < GROUP; ++h) {
        float mt = s[0][h];
#pragma unroll
        for (int it = 1; it < FA_TILE / 4; ++it) mt = fmaxf(mt, s[it][h]);
        mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 8));
        mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 16));
        const float mn = fmaxf(m[h], mt);
        alpha[h] = fa_exp2(m[h] - mn);
        m[h] = mn;
        float ps = 0.f;
#pragma unroll
        for (int it = 0; it < FA_TILE / 4; ++it) {
          s[it][h] = fa_exp2(s[it][h] - mn);
          ps += s[it][h];
        }
        l[h] = fmaf(l[h], alpha[h], ps);
#pragma unroll
        for (int d = 0; d < 8; ++d) acc2[h][d] = f2_mul(acc2[h][d], f2_pack(alpha[h], alpha[h]));
      }
#pragma unroll
      for (int it = 0; it < FA_TILE / 4; ++it) {
        uint64_t vf[8];
        fa_pairs8(raw[it][0], vf);
        fa_pairs8(raw[it][1], vf + 4);
#pragma unroll
        for (int h = 0; h < GROUP; ++h)
#pragma unroll
          for (int d = 0; d < 8; ++d) acc2[h][d] = f2_fma(f2_pack(s[it][h], s[it][h]), vf[d], acc2[h][d]);
      }
      leave(i);
    }
#pragma unroll
    for (int h = 0; h < GROUP; ++h)
#pragma unroll
      for (int d = 0; d < 8; ++d) f2_unpack(acc2[h][d], acc[h][2 * d], acc[h][2 * d + 1]);
  } else {
    float qv[GROUP][16];
#pragma unroll
    for (int h = 0; h < GROUP; ++h) {
      const __nv_bfloat16* qp = q_s + (head0 + h) * FA_HD;
      fa_unpack8(*reinterpret_cast<const uint4*>(qp + 8 * j), qv[h]);
      fa_unpack8(*reinterpret_cast<const uint4*>(qp + 64 + 8 * j), qv[h] + 8);
#pragma unroll
      for (int d = 0; d < 16; ++d) qv[h][d] *= p.scale_log2;
    }

#pragma unroll
    for (int h = 0; h < GROUP; ++h) {
      m[h] = -INFINITY; l[h] = 0.f;
#pragma unroll
      for (int d = 0; d < 16; ++d) acc[h][d] = 0.f;
    }

    for (int i = 0; i < my_tiles; ++i) {
      __nv_bfloat16 *kt, *vt;
      const int ntok = enter(i, kt, vt);
      float s[FA_TILE / 4][GROUP];
      int tokc[FA_TILE / 4];
#pragma unroll
      for (int it = 0; it < FA_TILE / 4; ++it) {
        const int tok = it * 4 + g;
        const bool valid = tok < ntok;
        tokc[it] = valid ? tok : 0;
        const __nv_bfloat16* kr = kt + tokc[it] * kv_dim;
        float kf[16];
        fa_unpack8(*reinterpret_cast<const uint4*>(kr + 8 * j), kf);
        fa_unpack8(*reinterpret_cast<const uint4*>(kr + 64 + 8 * j), kf + 8);
#pragma unroll
        for (int h = 0; h < GROUP; ++h) {
          float d0 = 0.f, d1 = 0.f;
#pragma unroll
          for (int d = 0; d < 16; d += 2) {
            d0 = fmaf(qv[h][d], kf[d], d0);
            d1 = fmaf(qv[h][d + 1], kf[d + 1], d1);
          }
          float dot = d0 + d1;
          dot += __shfl_xor_sync(0xffffffffu, dot, 1);
          dot += __shfl_xor_sync(0xffffffffu, dot, 2);
          dot += __shfl_xor_sync(0xffffffffu, dot, 4);
          s[it][h] = valid ? dot : -INFINITY;
        }
      }
      float alpha[GROUP];
#pragma unroll
      for (int h = 0; h < GROUP; ++h) {
        float mt = s[0][h];
#pragma unroll
        for (int it = 1; it < FA_TILE / 4; ++it) mt = fmaxf(mt, s[it][h]);
        mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 8));
        mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 16));
        const float mn = fmaxf(m[h], mt);
        alpha[h] = fa_exp2(m[h] - mn);
        m[h] = mn;
        float ps = 0.f;
#pragma unroll
        for (int it = 0; it < FA_TILE / 4; ++it) {
          s[it][h] = fa_exp2(s[it][h] - mn);
          ps += s[it][h];
        }
        l[h] = fmaf(l[h], alpha[h], ps);
#pragma unroll
        for (int d = 0; d < 16; ++d) acc[h][d] *= alpha[h];
      }
#pragma unroll
      for (int it = 0; it < FA_TILE / 4; ++it) {
        const __nv_bfloat16* vr = vt + tokc[it] * kv_dim;
        float vf[16];
        fa_unpack8(*reinterpret_cast<const uint4*>(vr + 8 * j), vf);
        fa_unpack8(*reinterpret_cast<const uint4*>(vr + 64 + 8 * j), vf + 8);
#pragma unroll
        for (int h = 0; h < GROUP; ++h)
#pragma unroll
          for (int d = 0; d < 16; ++d) acc[h][d] = fmaf(s[it][h], vf[d], acc[h][d]);
      }
      leave(i);
    }
  }

  // ---- fold the 4 token slots of the warp
#pragma unroll
  for (int h = 0; h < GROUP; ++h) {
    l[h] += __shfl_xor_sync(0xffffffffu, l[h], 8);
    l[h] += __shfl_xor_sync(0xffffffffu, l[h], 16);
#pragma unroll
    for (int d = 0; d < 16; ++d) {
      acc[h][d] += __shfl_xor_sync(0xffffffffu, acc[h][d], 8);
      acc[h][d] += __shfl_xor_sync(0xffffffffu, acc[h][d], 16);
    }
  }

  if constexpr (!SPLIT) {
    if (g == 0) {
#pragma unroll
      for (int h = 0; h < GROUP; ++h) {
        const float inv = 1.f / l[h];
        float o[16];
#pragma unroll
        for (int d = 0; d < 16; ++d) o[d] = acc[h][d] * inv;
        __nv_bfloat16* op = p.out + ((int64_t)row * p.num_heads + head0 + h) * FA_HD;
        stg_v4(op + 8 * j, fa_pack8(o));
        stg_v4(op + 64 + 8 * j, fa_pack8(o + 8));
      }
    }
  } else {
  // ---- split-KV: partials out, then the last CTA of this sequence folds all of them
  if (g == 0) {
#pragma unroll
    for (int h = 0; h < GROUP; ++h) {
      const int64_t idx = ((int64_t)row * p.nsplit + split) * p.num_heads + head0 + h;
      float* pa = p.part_acc + idx * FA_HD;
      *reinterpret_cast<float4*>(pa + 8 * j) = make_float4(acc[h][0], acc[h][1], acc[h][2], acc[h][3]);
      *reinterpret_cast<float4*>(pa + 8 * j + 4) = make_float4(acc[h][4], acc[h][5], acc[h][6], acc[h][7]);
      *reinterpret_cast<float4*>(pa + 64 + 8 * j) = make_float4(acc[h][8], acc[h][9], acc[h][10], acc[h][11]);
      *reinterpret_cast<float4*>(pa + 64 + 8 * j + 4) = make_float4(acc[h][12], acc[h][13], acc[h][14], acc[h][15]);
      if (j == 0) {
        p.part_ml[idx * 2] = my_tiles > 0 ? m[h] : -INFINITY;
        p.part_ml[idx * 2 + 1] = my_tiles > 0 ? l[h] : 0.f;
      }
    }
  }
  // One thread releases the CTA's partials after the CTA barrier (cumulative over the other threads' stores, as in a
  // cooperative-groups grid sync) and acquires for the CTA when it turns out to be the last: a __threadfence() per
  // thread is a MEMBAR.SC.GPU + L1 invalidate each (~1-2 us with 256 threads storing).  The readers below use ld.cg.
  asm volatile("bar.sync 1, %0;" :: "r"(kvh * 32) : "memory");      // the consumer warps only
  if (threadIdx.x == 0) {
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    const int t = atomicAdd(p.tickets + row, 1);
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    *last_flag = (t == p.nsplit - 1);
    if (t == p.nsplit - 1) p.tickets[row] = 0;                     // ready for the next launch
  }
  asm volatile("bar.sync 1, %0;" :: "r"(kvh * 32) : "memory");
  if (!*last_flag) return;
  fa_fold<GROUP>(p.part_ml, p.part_acc, p.out, p.nsplit, p.num_heads, row, head0);
  }
}

// ---------------------------------------------------------------------------------------------------------
// Short contexts (the code predictor: 3..17 tokens, 75 launches per codec frame).  The kernel above is built to stream
// long contexts (bulk-copy ring, producer warp, split-KV tickets); for a handful of tokens all of that is latency.
// Here one WARP owns one (sequence, kv head) item: no shared-memory ring, no block barrier, no split - the cached
// rows are read straight from the paged cache, two 8-token tiles per round trip, and the new token never leaves
// the warp.  Arithmetic, lane mapping and summation order are those of fused_decode_attn_kernel with nsplit == 1
// (GROUP 2, 1-D RoPE), so outputs and K / V cache bytes are bit-identical.
// One product after another: pairs gave nothing for a tile or two (201 rows of 17 tokens 10.8 us) and cost a third for more (300 rows of 50 29.6 -> 41.1, 200 of 200 in tables
// said to have room for 60 63 -> 101).
constexpr int FS_WARPS = 4;
constexpr int FS_MAX_CTX = 64;

template <bool EAGER>
__global__ void __launch_bounds__(FS_WARPS * 32)
fused_decode_attn_small_kernel(const FusedAttnParams p, int rows) {
  constexpr int GROUP = 2;
  __shared__ __align__(16) __nv_bfloat16 scr_all[FS_WARPS][(GROUP + 2) * FA_HD];   // q [2][128], k [128], v [128] of the new token
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = p.num_kv_heads, kv_dim = kvh * FA_HD;
  const int item = blockIdx.x * FS_WARPS + warp;
  pdl_launch();
  if (item >= rows * kvh) return;
  const int row = item / kvh, hk = item - row * kvh;
  const int head0 = hk * GROUP;
  const int g = lane >> 3, j = lane & 7;
  __nv_bfloat16* q_s = scr_all[warp];
  __nv_bfloat16* kn_s = q_s + GROUP * FA_HD;
  __nv_bfloat16* vn_s = kn_s + FA_HD;
  // independent of the previous kernel: rotary frequencies, head-norm weights
  float frq[2];
  frq[0] = __ldg(p.inv_freq + 2 * lane);
  frq[1] = __ldg(p.inv_freq + 2 * lane + 1);
  uint32_t qw1 = 0, qw2 = 0, kw1 = 0, kw2 = 0;
  if (p.q_w) { qw1 = *reinterpret_cast<const uint32_t*>(p.q_w + 2 * lane); qw2 = *reinterpret_cast<const uint32_t*>(p.q_w + 64 + 2 * lane); }
  if (p.k_w) { kw1 = *reinterpret_cast<const uint32_t*>(p.k_w + 2 * lane); kw2 = *reinterpret_cast<const uint32_t*>(p.k_w + 64 + 2 * lane); }
  pdl_wait();
  // ---- one batch of independent requests
  int L = __ldg(p.context_lens + row);
  const int slot = __ldg(p.slot_mapping + row);
  const int64_t pos = __ldg(p.positions + row);
  const int32_t* bt = p.block_table + (int64_t)row * p.bt_stride;
  int page0 = __ldg(bt);
  uint32_t raw1[GROUP + 1], raw2[GROUP + 1];
#pragma unroll
  for (int i = 0; i < GROUP + 1; ++i) {
    const __nv_bfloat16* src = i == GROUP ? p.k + (int64_t)row * p.k_stride + hk * FA_HD
                                          : p.q + (int64_t)row * p.q_stride + (head0 + i) * FA_HD;
    raw1[i] = *reinterpret_cast<const uint32_t*>(src + 2 * lane);
    raw2[i] = *reinterpret_cast<const uint32_t*>(src + 64 + 2 * lane);
  }
  uint4 vraw = make_uint4(0, 0, 0, 0);
  if (lane < 16) vraw = ldg_v4(p.v + (int64_t)row * p.v_stride + hk * FA_HD + 8 * lane);
  if (L <= 0) {                   // CUDA-graph padding row: zeros
    if (g == 0) {
#pragma unroll
      for (int h = 0; h < GROUP; ++h) {
        __nv_bfloat16* o = p.out + ((int64_t)row * p.num_heads + head0 + h) * FA_HD;
        stg_v4(o + 8 * j, make_uint4(0, 0, 0, 0));
        stg_v4(o + 64 + 8 * j, make_uint4(0, 0, 0, 0));
      }
    }
    return;
  }
  if (page0 < 0) page0 = 0;
  // a token's K / V row of this head in the paged cache
  auto tok_off = [&](int t) -> int64_t {
    int page = page0;
    if (t >= p.page_size) { page = __ldg(bt + t / p.page_size); if (page < 0) page = 0; }
    return ((int64_t)page * p.page_size + t % p.page_size) * kv_dim + hk * FA_HD;
  };
  // the cached rows of the first two tiles are requested NOW, under the prologue arithmetic
  const int n_tiles = (L + FA_TILE - 1) / FA_TILE;
  uint4 kbuf[2][2][2], vbuf[2][2][2];            // [tile of the pair][token slot][half]
  auto load_pair = [&](int i0) {
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int tok0 = (i0 + u) * FA_TILE;
        const int ntok = min(FA_TILE, L - tok0);
        const int tok = s * 4 + g;
        const int t = tok0 + (tok < ntok ? tok : 0);
        if (i0 + u < n_tiles && t != L - 1) {
          const int64_t off = tok_off(t);
          kbuf[u][s][0] = ldg_v4(p.k_cache + off + 8 * j);
          kbuf[u][s][1] = ldg_v4(p.k_cache + off + 64 + 8 * j);
          vbuf[u][s][0] = ldg_v4(p.v_cache + off + 8 * j);
          vbuf[u][s][1] = ldg_v4(p.v_cache + off + 64 + 8 * j);
        }
      }
  };
  load_pair(0);
  // ---- prologue: q/k head norm + RoPE of the new token (the body of qknorm_rope_kvwrite_kernel), K / V to the cache
  {
    float cf[2], sf[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float a1 = (float)pos * frq[e];
      cf[e] = cosf(a1) * p.attention_scaling;
      sf[e] = sinf(a1) * p.attention_scaling;
    }
    const uint32_t c1 = pack_bf16(cf[0], cf[1]), s1 = pack_bf16(sf[0], sf[1]);
#pragma unroll
    for (int i = 0; i < GROUP + 1; ++i) {
      const bool is_k = i == GROUP;
      const bool has_w = is_k ? (p.k_w != nullptr) : (p.q_w != nullptr);
      uint32_t x1 = raw1[i], x2 = raw2[i];
      if (has_w) {
        float ss = bf16lo(x1) * bf16lo(x1);
        ss = fmaf(bf16hi(x1), bf16hi(x1), ss); ss = fmaf(bf16lo(x2), bf16lo(x2), ss); ss = fmaf(bf16hi(x2), bf16hi(x2), ss);
        const float var = warp_sum(ss) / (float)FA_HD + p.eps;
        const float rstd = EAGER ? 1.0f / sqrtf(var) : rsqrtf(var);
        x1 = norm_pair<EAGER>(x1, rstd, is_k ? kw1 : qw1);
        x2 = norm_pair<EAGER>(x2, rstd, is_k ? kw2 : qw2);
      }
      const uint32_t y1 = turn_first(x1, x2, c1, s1), y2 = turn_second(x1, x2, c1, s1);
      __nv_bfloat16* dst = is_k ? kn_s : q_s + i * FA_HD;
      *reinterpret_cast<uint32_t*>(dst + 2 * lane) = y1;
      *reinterpret_cast<uint32_t*>(dst + 64 + 2 * lane) = y2;
      if (is_k && slot >= 0) {
        __nv_bfloat16* cd = p.k_cache + (int64_t)slot * kv_dim + hk * FA_HD;
        *reinterpret_cast<uint32_t*>(cd + 2 * lane) = y1;
        *reinterpret_cast<uint32_t*>(cd + 64 + 2 * lane) = y2;
      }
    }
    if (lane < 16) {
      *reinterpret_cast<uint4*>(vn_s + 8 * lane) = vraw;
      if (slot >= 0) stg_v4(p.v_cache + (int64_t)slot * kv_dim + hk * FA_HD + 8 * lane, vraw);
    }
  }
  __syncwarp();
  float qv[GROUP][16];
#pragma unroll
  for (int h = 0; h < GROUP; ++h) {
    const __nv_bfloat16* qp = q_s + h * FA_HD;
    fa_unpack8(*reinterpret_cast<const uint4*>(qp + 8 * j), qv[h]);
    fa_unpack8(*reinterpret_cast<const uint4*>(qp + 64 + 8 * j), qv[h] + 8);
#pragma unroll
    for (int d = 0; d < 16; ++d) qv[h][d] *= p.scale_log2;
  }
  float m[GROUP], l[GROUP], acc[GROUP][16];
#pragma unroll
  for (int h = 0; h < GROUP; ++h) {
    m[h] = -INFINITY; l[h] = 0.f;
#pragma unroll
    for (int d = 0; d < 16; ++d) acc[h][d] = 0.f;
  }
  for (int i0 = 0; i0 < n_tiles; i0 += 2) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (i0 + u >= n_tiles) break;
      const int tok0 = (i0 + u) * FA_TILE;
      const int ntok = min(FA_TILE, L - tok0);
      float s[FA_TILE / 4][GROUP];
      bool isnew[FA_TILE / 4];
#pragma unroll
      for (int it = 0; it < FA_TILE / 4; ++it) {
        const int tok = it * 4 + g;
        const bool valid = tok < ntok;
        isnew[it] = tok0 + (valid ? tok : 0) == L - 1;
        float kf[16];
        if (isnew[it]) {
          fa_unpack8(*reinterpret_cast<const uint4*>(kn_s + 8 * j), kf);
          fa_unpack8(*reinterpret_cast<const uint4*>(kn_s + 64 + 8 * j), kf + 8);
        } else {
          fa_unpack8(kbuf[u][it][0], kf);
          fa_unpack8(kbuf[u][it][1], kf + 8);
        }
#pragma unroll
        for (int h = 0; h < GROUP; ++h) {
          float d0 = 0.f, d1 = 0.f;
#pragma unroll
          for (int d = 0; d < 16; d += 2) {
            d0 = fmaf(qv[h][d], kf[d], d0);
            d1 = fmaf(qv[h][d + 1], kf[d + 1], d1);
          }
          float dot = d0 + d1;
          dot += __shfl_xor_sync(0xffffffffu, dot, 1);
          dot += __shfl_xor_sync(0xffffffffu, dot, 2);
          dot += __shfl_xor_sync(0xffffffffu, dot, 4);
          s[it][h] = valid ? dot : -INFINITY;
        }
      }
      float alpha[GROUP];
#pragma unroll
      for (int h = 0; h < GROUP; ++h) {
        float mt = s[0][h];
#pragma unroll
        for (int it = 1; it < FA_TILE / 4; ++it) mt = fmaxf(mt, s[it][h]);
        mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 8));
        mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 16));
        const float mn = fmaxf(m[h], mt);
        alpha[h] = fa_exp2(m[h] - mn);
        m[h] = mn;
        float ps = 0.f;
#pragma unroll
        for (int it = 0; it < FA_TILE / 4; ++it) {
          s[it][h] = fa_exp2(s[it][h] - mn);
          ps += s[it][h];
        }
        l[h] = fmaf(l[h], alpha[h], ps);
#pragma unroll
        for (int d = 0; d < 16; ++d) acc[h][d] *= alpha[h];
      }
#pragma unroll
      for (int it = 0; it < FA_TILE / 4; ++it) {
        float vf[16];
        if (isnew[it]) {
          fa_unpack8(*reinterpret_cast<const uint4*>(vn_s + 8 * j), vf);
          fa_unpack8(*reinterpret_cast<const uint4*>(vn_s + 64 + 8 * j), vf + 8);
        } else {
          fa_unpack8(vbuf[u][it][0], vf);
          fa_unpack8(vbuf[u][it][1], vf + 8);
        }
#pragma unroll
        for (int h = 0; h < GROUP; ++h)
#pragma unroll
          for (int d = 0; d < 16; ++d) acc[h][d] = fmaf(s[it][h], vf[d], acc[h][d]);
      }
    }
    if (i0 + 2 < n_tiles) load_pair(i0 + 2);
  }
#pragma unroll
  for (int h = 0; h < GROUP; ++h) {
    l[h] += __shfl_xor_sync(0xffffffffu, l[h], 8);
    l[h] += __shfl_xor_sync(0xffffffffu, l[h], 16);
#pragma unroll
    for (int d = 0; d < 16; ++d) {
      acc[h][d] += __shfl_xor_sync(0xffffffffu, acc[h][d], 8);
      acc[h][d] += __shfl_xor_sync(0xffffffffu, acc[h][d], 16);
    }
  }
  if (g == 0) {
#pragma unroll
    for (int h = 0; h < GROUP; ++h) {
      const float inv = 1.f / l[h];
      float o[16];
#pragma unroll
      for (int d = 0; d < 16; ++d) o[d] = acc[h][d] * inv;
      __nv_bfloat16* op = p.out + ((int64_t)row * p.num_heads + head0 + h) * FA_HD;
      stg_v4(op + 8 * j, fa_pack8(o));
      stg_v4(op + 64 + 8 * j, fa_pack8(o + 8));
    }
  }
}

// One and two query heads a key head: two products an instruction, keys and values of a tile asked for together.  A turn of the ring without branches (unrolled) where there
// are many tiles a CTA: without splits (200 rows of 200 tokens, 16 and 8 heads, 32.5 -> 30.2 us), and with few key heads, whose CTAs wait for each tile (32 rows of 2000 tokens, 4
// and 2 heads 31 -> 22, 8 and 4 35 -> 30; 28 and 34 before pairs); else the longer code costs more than it gives (64 rows of 40 tokens, 16 and 8 heads 8.8, unrolled 10.1).
// Four query heads a key head: products one by one (pairs spill: 113 us for 200 rows of 200 tokens and 32 heads, 106 so), and as many registers as the CTAs of few key heads
// leave: 300 rows of 1000 tokens, 8 and 2 heads 162 us, with 96 registers 245 (285 with pairs' order of loads, 233 before pairs), 16 and 4 245 (447); 32 and 8 heads have no more: 765 (743).
static void (*fa_pick(int group, bool split, int kv_heads, bool eager))(const FusedAttnParams) {
#define FA_ONE(G, K) (split ? (eager ? fused_decode_attn_kernel<G, true, true, K> : fused_decode_attn_kernel<G, false, true, K>) \
                            : (eager ? fused_decode_attn_kernel<G, true, false, K> : fused_decode_attn_kernel<G, false, false, K>))
  if (group == 1) return FA_ONE(1, 8);
  if (group == 2) return kv_heads <= 4 ? FA_ONE(2, 4) : FA_ONE(2, 8);
  if (group == 4) return kv_heads <= 2 ? FA_ONE(4, 2) : kv_heads <= 4 ? FA_ONE(4, 4) : FA_ONE(4, 8);
#undef FA_ONE
  return nullptr;
}

static size_t fa_smem_bytes(int kv_heads, int num_heads) {
  return (size_t)2 * FA_NSTAGE * FA_TILE * kv_heads * FA_HD * 2 + 2 * FA_NSTAGE * sizeof(uint64_t) + 16 +
         (size_t)(num_heads + 2 * kv_heads) * FA_HD * 2;
}

// split-KV factor: one wave of 2 CTAs per SM, at least 8 tiles (64 tokens) of table capacity per split
int fa_choose_nsplit(int rows, int max_ctx) {
  if (const char* e = getenv("B2TTS_FA_NSPLIT")) {             // experiments only
    const int v = atoi(e);
    if (v >= 1 && v <= 32) return v;
  }
  const int max_tiles = (max_ctx + FA_TILE - 1) / FA_TILE;
  int n = (2 * sm_count()) / (rows > 0 ? rows : 1);
  const int cap = max_tiles / 8;
  if (n > cap) n = cap;
  if (n < 1) n = 1;
  if (n > 32) n = 32;
  return n;
}

}  // namespace b2

extern "C" size_t b2tts_fused_decode_attn_workspace_bytes(int batch, int num_heads, int head_dim, int max_ctx) {
  if (batch <= 0 || num_heads <= 0 || head_dim <= 0 || max_ctx <= 0) return 0;
  const int nsplit = b2::fa_choose_nsplit(batch, max_ctx);
  // fixed ticket span (zero before the first launch, left zero by every launch) + partials + (m, l)
  return b2::FA_TICKET_BYTES + (size_t)batch * nsplit * num_heads * (head_dim + 2) * sizeof(float) + 16;
}

extern "C" int b2tts_fused_decode_attn(const void* q, int64_t q_row_stride, const void* k, int64_t k_row_stride,
                                       const void* v, int64_t v_row_stride,
                                       const void* q_weight, const void* k_weight, float eps,
                                       const int64_t* positions, int64_t pos_row_stride,
                                       const float* inv_freq, const int32_t* modality, float attention_scaling,
                                       const int32_t* slot_mapping, void* k_cache, void* v_cache,
                                       const int32_t* block_table, int bt_stride, const int32_t* context_lens,
                                       void* out, void* workspace, size_t workspace_bytes,
                                       int batch, int num_heads, int num_kv_heads, int head_dim, int page_size,
                                       float scale, int max_ctx, int rounding, int pdl, void* stream) {
  using namespace b2;
  const char* what = "fused_decode_attn";
  B2_REQUIRE(batch >= 0 && max_ctx > 0 && page_size > 0 && bt_stride > 0, B2TTS_EINVAL,
             "%s: batch=%d max_ctx=%d page_size=%d bt_stride=%d", what, batch, max_ctx, page_size, bt_stride);
  if (batch == 0) return B2TTS_OK;
  B2_REQUIRE(batch <= FA_MAX_ROWS, B2TTS_EUNSUPPORTED, "%s: batch %d > %d rows", what, batch, FA_MAX_ROWS);
  B2_REQUIRE(q && k && v && positions && inv_freq && slot_mapping && k_cache && v_cache && block_table && context_lens &&
                 out && workspace, B2TTS_EINVAL, "%s: null pointer", what);
  B2_REQUIRE(head_dim == FA_HD, B2TTS_EUNSUPPORTED, "%s: head_dim %d unsupported (128)", what, head_dim);
  B2_REQUIRE(num_kv_heads >= 1 && num_kv_heads <= 8 && num_heads % num_kv_heads == 0, B2TTS_EUNSUPPORTED,
             "%s: heads %d / kv heads %d unsupported", what, num_heads, num_kv_heads);
  B2_REQUIRE(page_size % FA_TILE == 0, B2TTS_EUNSUPPORTED, "%s: page_size %d must be a multiple of %d", what, page_size,
             FA_TILE);
  B2_REQUIRE(rounding == B2TTS_ROUND_EAGER || rounding == B2TTS_ROUND_FUSED, B2TTS_EINVAL, "%s: rounding %d", what, rounding);
  B2_REQUIRE(aligned16(q) && aligned16(k) && aligned16(v) && aligned16(k_cache) && aligned16(v_cache) && aligned16(out) &&
                 aligned16(workspace) && q_row_stride % 8 == 0 && k_row_stride % 8 == 0 && v_row_stride % 8 == 0 &&
                 (!q_weight || aligned16(q_weight)) && (!k_weight || aligned16(k_weight)),
             B2TTS_EALIGN, "%s: pointers / strides must be 16-byte aligned", what);
  FusedAttnParams p{};
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.k = static_cast<const __nv_bfloat16*>(k);
  p.v = static_cast<const __nv_bfloat16*>(v);
  p.q_stride = q_row_stride; p.k_stride = k_row_stride; p.v_stride = v_row_stride;
  p.q_w = static_cast<const __nv_bfloat16*>(q_weight);
  p.k_w = static_cast<const __nv_bfloat16*>(k_weight);
  p.eps = eps;
  p.positions = positions;
  p.pos_row_stride = pos_row_stride;
  p.inv_freq = inv_freq;
  p.modality = modality;
  p.attention_scaling = attention_scaling;
  p.slot_mapping = slot_mapping;
  p.k_cache = static_cast<__nv_bfloat16*>(k_cache);
  p.v_cache = static_cast<__nv_bfloat16*>(v_cache);
  p.block_table = block_table;
  p.bt_stride = bt_stride;
  p.page_size = page_size;
  p.context_lens = context_lens;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.nsplit = fa_choose_nsplit(batch, max_ctx);
  p.num_heads = num_heads;
  p.num_kv_heads = num_kv_heads;
  p.scale_log2 = scale * 1.4426950408889634f;
  const size_t acc_elems = (size_t)batch * p.nsplit * num_heads * head_dim;
  const size_t need = b2tts_fused_decode_attn_workspace_bytes(batch, num_heads, head_dim, max_ctx);
  B2_REQUIRE(workspace_bytes >= need, B2TTS_EWORKSPACE, "%s: workspace %zu B < %zu B needed", what, workspace_bytes, need);
  p.tickets = static_cast<int*>(workspace);
  p.part_acc = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + FA_TICKET_BYTES);
  p.part_ml = p.part_acc + acc_elems;

  const int group = num_heads / num_kv_heads;
  const bool eager = rounding == B2TTS_ROUND_EAGER;
  static const bool small_ok = [] { const char* e = getenv("B2TTS_FA_SMALL"); return !(e && e[0] == '0'); }();
  if (small_ok && max_ctx <= FS_MAX_CTX && group == 2 && !modality && p.nsplit == 1) {
    // a handful of cached tokens: one warp per (sequence, kv head), no ring, no split
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((batch * num_kv_heads + FS_WARPS - 1) / FS_WARPS, 1, 1);
    cfg.blockDim = dim3(FS_WARPS * 32, 1, 1);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaError_t e = eager ? cudaLaunchKernelEx(&cfg, fused_decode_attn_small_kernel<true>, p, batch)
                          : cudaLaunchKernelEx(&cfg, fused_decode_attn_small_kernel<false>, p, batch);
    count_launch();
    if (e != cudaSuccess) return cuda_fail(e, what);
    return B2TTS_OK;
  }
  void (*kern)(const FusedAttnParams) = fa_pick(group, p.nsplit > 1, num_kv_heads, eager);
  B2_REQUIRE(kern, B2TTS_EUNSUPPORTED, "%s: GQA group %d unsupported (1, 2, 4)", what, group);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e != cudaSuccess) return cuda_fail(e, what);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(batch, p.nsplit, 1);
  cfg.blockDim = dim3(32 * (num_kv_heads + 1), 1, 1);
  cfg.dynamicSmemBytes = fa_smem_bytes(num_kv_heads, num_heads);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, kern, p);
  count_launch();
  if (e != cudaSuccess) return cuda_fail(e, what);
  return B2TTS_OK;
}
