// prompt_attn_tc.cu - softmax attention of prompt portions (more than one new token of a sequence) on the 5th-generation tensor cores:
// keys and values through block tables or in rows of their own, sliding-window, chunk or causal masks with kept first keys, sinks, score
// caps, gates.  bf16 operands, float scores, weights, sums and outputs' accumulators.
//
// One CTA = 128 query rows: 128 / HPC tokens times HPC heads that share a key head.  Key tiles of 128:
//   loader    one warp; a tile's rows arrive as TMA boxes of 64 columns x R rows, R the largest power of two up to 64 that divides the
//             page (tiles start on a multiple of R, so a box never straddles a page; an issue takes about 90 cycles, so few large
//             ones; up to 16 rows a box at the list's end), one box per lane, two stages for keys and two for values (gathering rows with 16-byte asynchronous copies ran at 21 bytes a cycle and SM and was the
//             bound: 313 us for the case below).  Rows behind the last key are zeros, never what a page holds there;
//   S         tcgen05.mma 128 x 128 x 16 into one of two TMEM buffers, a tile ahead of the softmax;
//   softmax   eight warps, two threads per query row with 64 scores each in registers: maximum (exchanged through shared memory),
//             exp2, sum; the weights go back to TMEM as the A operand of the second product (never through shared memory), as
//             hi + lo pairs where 16 bits are asked for;
//   O         tcgen05.mma (weights from TMEM, the value tile MN-major as it was gathered), accumulated in TMEM over all tiles.
// The running maximum is lazy: O and the sum are rescaled only when a row's maximum has grown by more than 2^8, so the accumulator is
// almost never touched between tiles; weights are then up to 2^8, which floats and bf16 pairs hold as well as 1.
//
// Bound: per tile about 2700 cycles of softmax (1400 of them exp2 and the split into parts) beside 2700 of MMA issue (S 8 x 80, the two
// weight products 16 x 120), and about 15000 cycles of start and end per CTA, of which one runs per SM.
// 4 prompts of 2048 tokens, 16 heads over 8 of 128, window 1024 + 4 kept, element gates: 156 us (mma.sync, 64 queries per CTA: 549 us);
// causal with a score cap, 4448 tokens: 228 us the layer (662 us); 40 new tokens behind 1400 and 700 behind 20: 46 us (97 us); portions
// of 2 tokens 58 us (56 us, host-bound both).
#include <algorithm>

#include "prompt_attn.cuh"
#include "umma.cuh"

namespace b2 {
namespace row {

constexpr int PA_M = 128, PA_N = 128, PA_BOX = 128 * 128;      // a box: 128 rows of 64 bf16 columns
constexpr int PA_SOFT = 8;                                     // softmax warps
constexpr int PA_THREADS = 32 * (PA_SOFT + 2);                 // warps 0-7 softmax, 8 MMA, 9 loader

// How often a wait inside the kernel ran out (it never should); read by b2tts_prompt_attn_timeouts().
__device__ int g_prompt_attn_timeouts = 0;

// MN-major SWIZZLE_128B operand: a K index (key) is a 128-byte row of 64 columns; LBO: the next 64 columns (the second box), SBO: 8 keys
__device__ __forceinline__ uint64_t pa_desc_mn(uint32_t addr) {
  return static_cast<uint64_t>((addr & 0x3ffffu) >> 4) | (static_cast<uint64_t>(PA_BOX >> 4) << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}
// D [128 x n] (+)= A (TMEM: two bf16 per column, lane = row) B (shared memory)
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}"
      :: "r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
         "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
         "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float pa_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// within a few 2^-22 of the value: 64 of them per thread stand between the last product and the end of the CTA
__device__ __forceinline__ float pa_sigmoid(float x) { return __fdividef(1.0f, 1.0f + __expf(-x)); }
__device__ __forceinline__ int pa_mask_lo(int i, int kind, int mask) {
  if (mask <= 0) return 0;
  return kind == 0 ? max(0, i - mask + 1) : (i / mask) * mask;
}

struct PromptMaps { CUtensorMap k[2], k2[2], v[2]; };          // boxes of R rows, and of the smaller size for the list's end

// the n lowest of 32 bits (none for n <= 0, all from 32 on)
__device__ __forceinline__ uint32_t pa_below(int n) { return n <= 0 ? 0u : n >= 32 ? 0xffffffffu : (1u << n) - 1u; }

// NS: 64-column slices of q and k; NV: of v
template <int NS, int NV, bool SPLIT>
__global__ void __launch_bounds__(PA_THREADS, 1)
prompt_attn_kernel(const PromptAttnArgs a, const int hpc, const __grid_constant__ PromptMaps maps) {
  extern __shared__ uint8_t pa_smem[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(pa_smem) + 1023) & ~uintptr_t(1023));
  uint8_t* q_s = smem;
  uint8_t* k_s = q_s + NS * PA_BOX;                    // [2 stages][NS]
  uint8_t* v_s = k_s + 2 * NS * PA_BOX;                // [2 stages][NV]
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + 2 * NV * PA_BOX);
  uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = bars + 3, *v_full = bars + 5, *v_empty = bars + 7, *s_full = bars + 9,
           *s_empty = bars + 11, *p_full = bars + 13, *pv_done = bars + 14;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  float* row_x = reinterpret_cast<float*>(bars + 16);  // [2][2 halves][128]: what the two threads of a row exchange

  const int b = blockIdx.z, len = a.seq_len[b];
  const int per = PA_M / hpc;                          // tokens per CTA
  const int tile = static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x), t0 = tile * per;     // the longest rows first
  if (len <= 1 || t0 >= len) return;                   // uniform; one-token and padding rows have kernels of their own
  const int h0 = blockIdx.y * hpc, g = h0 / (a.H / a.G), gv = g % a.Gv;
  const int start = a.seq_start[b], pos0 = a.seq_pos0[b];
  const int t_last = min(len, t0 + per) - 1;
  const int j_lo = pa_mask_lo(pos0 + t0, a.mask_kind, a.mask), j_hi = pos0 + t_last;
  // the key list in whole boxes: kept first keys that the lowest bound of the CTA hides, then [j_lo, j_hi] from a multiple of R on;
  // where the boxes of the kept keys reach that bound, one run from key 0
  const int R = a.box_rows, keep_r = (a.keep_first + R - 1) & ~(R - 1);
  const bool pre = a.keep_first > 0 && keep_r <= j_lo;
  const int n_pre = pre ? a.keep_first : 0, pre_r = pre ? keep_r : 0, jl = pre || a.keep_first == 0 ? j_lo & ~(R - 1) : 0;
  const int keep_in = pre ? 0 : a.keep_first;          // kept keys that are part of the run
  const int n_keys = pre_r + j_hi - jl + 1, n_tiles = (n_keys + PA_N - 1) / PA_N;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(q_full, PA_SOFT);
    for (int s = 0; s < 2; ++s) {
      mbar_init(k_full + s, 1); mbar_init(k_empty + s, 1);
      mbar_init(v_full + s, 1); mbar_init(v_empty + s, 1);
      mbar_init(s_full + s, 1); mbar_init(s_empty + s, PA_SOFT);
    }
    mbar_init(p_full, PA_SOFT); mbar_init(pv_done, 1);
    mbar_fence_init();
  }
  if (warp == PA_SOFT) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tm_s = tmem, tm_o = tmem + 256, tm_p = tmem + 384;    // S: 2 x 128, O: 128, weights: 64 hi + 64 lo
  bool ok = true;

  if (warp > PA_SOFT) {
    // =========================== loader
    const int32_t* bt = a.block_tables != nullptr ? a.block_tables + static_cast<int64_t>(b) * a.bt_stride : nullptr;
    const int row0 = bt == nullptr ? a.key_start[b] : 0;
    auto row_of = [&](int vi) {                          // cache row of the key list's entry vi
      const int key = vi < pre_r ? vi : jl + vi - pre_r;
      if (bt == nullptr) return row0 + key;
      const int pg = a.page_shift >= 0 ? key >> a.page_shift : key / a.page;
      return bt[pg] * a.page + key - pg * a.page;
    };
    // the end of the list inside tile j behind the boxes, `n` slices at `dst` of which `width` columns exist: row by row, then zeros
    const int Rs = min(R, 16);
    auto fill_end = [&](int j, uint8_t* dst, const __nv_bfloat16* base, int64_t ld, int n, int width) {
      const int r0 = min(n_keys - j * PA_N, PA_N) / Rs * Rs;
      for (int i = lane; i < (PA_N - r0) * 8; i += 32) {
        const int ch = i & 7, r = r0 + (i >> 3);
        uint4 x[3] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
        if (j * PA_N + r < n_keys) {
          const __nv_bfloat16* src = base + static_cast<int64_t>(row_of(j * PA_N + r)) * ld + ch * 8;
#pragma unroll
          for (int s = 0; s < 3; ++s)
            if (s < n && s * 64 + ch * 8 < width) x[s] = ldg_v4(src + s * 64);
        }
#pragma unroll
        for (int s = 0; s < 3; ++s)
          if (s < n) *reinterpret_cast<uint4*>(dst + s * PA_BOX + r * 128 + ((ch ^ (r & 7)) << 4)) = x[s];
      }
    };
    // box x of tile j: whole boxes of R rows, then up to R / Rs - 1 small ones; -1 behind them
    auto box_at = [&](int j, int x, bool& big) {
      const int rows = min(n_keys - j * PA_N, PA_N), nb = rows / R;
      big = x < nb;
      const int at = big ? x * R : nb * R + (x - nb) * Rs;
      return big || at + Rs <= rows ? at : -1;
    };
    // page and offset of box `lane` (boxes beyond 32 are looked up where they are used), a tile ahead: nothing waits for the load here
    struct Slot { int pg, off; };
    auto lookup = [&](int j) {
      bool big;
      const int at = max(box_at(j, lane, big), 0), vi = j * PA_N + at, key = vi < pre_r ? vi : jl + vi - pre_r;
      Slot x{0, row0 + key};
      if (bt != nullptr) {
        const int pg = a.page_shift >= 0 ? key >> a.page_shift : key / a.page;
        x.pg = bt[min(pg, j_hi / a.page)];
        x.off = key - pg * a.page;
      }
      return x;
    };
    auto fill = [&](int j, Slot mine, uint8_t* dst, const CUtensorMap* map, int x0, int n, uint64_t* bar) {
      for (int x = lane; x < PA_N / Rs; x += 32) {
        bool big;
        const int at = box_at(j, x, big);
        if (at < 0) break;
        const int row = x == lane ? mine.pg * a.page + mine.off : row_of(j * PA_N + at);
#pragma unroll
        for (int s = 0; s < 3; ++s)
          if (s < n) tma_load_2d(dst + s * PA_BOX + at * 128, map + (big ? 0 : 1), x0 + s * 64, row, bar);
      }
      __syncwarp();
    };
    Slot cur{0, 0}, prev, next = lookup(0);
    const int n1 = min(NS, (a.d1 + 63) / 64);
    for (int j = 0; ok && j <= n_tiles; ++j) {
      prev = cur; cur = next;
      if (j < n_tiles) {
        const int st = j & 1, rows = min(n_keys - j * PA_N, PA_N) / Rs * Rs;
        uint8_t *d1 = k_s + st * NS * PA_BOX, *d2 = d1 + n1 * PA_BOX;
        if (!(ok = mbar_wait_limit(k_empty + st, ((j >> 1) & 1) ^ 1))) break;
        if (rows < PA_N) {
          fill_end(j, d1, a.k + g * a.k_head, a.k_row, n1, a.d1);
          if (n1 < NS) fill_end(j, d2, a.k2, a.k2_row, NS - n1, a.d - a.d1);
          fence_proxy_async();
        }
        __syncwarp();
        if (lane == 0) mbar_expect_tx(k_full + st, NS * rows * 128);
        __syncwarp();
        fill(j, cur, d1, maps.k, g * a.k_head, n1, k_full + st);
        if (n1 < NS) fill(j, cur, d2, maps.k2, 0, NS - n1, k_full + st);
        if (j + 1 < n_tiles) next = lookup(j + 1);
      }
      if (j > 0) {
        const int i = j - 1, st = i & 1, rows = min(n_keys - i * PA_N, PA_N) / Rs * Rs;
        uint8_t* dst = v_s + st * NV * PA_BOX;
        if (!(ok = mbar_wait_limit(v_empty + st, ((i >> 1) & 1) ^ 1))) break;
        if (rows < PA_N) {
          fill_end(i, dst, a.v + gv * a.v_head, a.v_row, NV, a.dv);
          fence_proxy_async();
        }
        __syncwarp();
        if (lane == 0) mbar_expect_tx(v_full + st, NV * rows * 128);
        __syncwarp();
        fill(i, prev, dst, maps.v, gv * a.v_head, NV, v_full + st);
      }
    }
    if (ok) {                                            // every copy has landed before the CTA leaves
      ok = mbar_wait_limit(k_full + ((n_tiles - 1) & 1), ((n_tiles - 1) >> 1) & 1) && mbar_wait_limit(v_full + ((n_tiles - 1) & 1), ((n_tiles - 1) >> 1) & 1);
    } else {
      for (int x = 0; x < 2; ++x)
        for (int ph = 0; ph < 2; ++ph) { mbar_wait_limit(k_full + x, ph); mbar_wait_limit(v_full + x, ph); }
    }
  } else if (warp == PA_SOFT) {
    // =========================== MMA issuer: S_0, S_1, O += P_0 V_0, S_2, O += P_1 V_1, ..
    const uint32_t idesc_s = umma_idesc_bf16(PA_N), idesc_o = umma_idesc_bf16(NV * 64) | (1u << 16);     // the value operand is MN-major
    const int steps = (a.d + 15) / 16;
    ok = mbar_wait_limit(q_full, 0);
    for (int j = 0; ok && j <= n_tiles; ++j) {
      const int st = j & 1;
      if (j < n_tiles) {
        if (!(ok = mbar_wait_limit(k_full + st, (j >> 1) & 1) && mbar_wait_limit(s_empty + st, ((j >> 1) & 1) ^ 1))) break;
        tc_fence_after();
        const uint32_t q_lo = umma_desc_lo_sw128(smem_u32(q_s)), k_lo = umma_desc_lo_sw128(smem_u32(k_s + st * NS * PA_BOX));
        if (elect_one()) {
#pragma unroll
          for (int s = 0; s < NS * 4; ++s)
            if (s < steps) {
              const uint32_t off = (s >> 2) * (PA_BOX >> 4) + (s & 3) * 2;
              umma_bf16_lo(tm_s + st * PA_N, q_lo + off, k_lo + off, idesc_s, s != 0);
            }
          umma_commit(s_full + st);
          umma_commit(k_empty + st);
        }
        __syncwarp();
      }
      if (j > 0) {
        const int i = j - 1, vs = i & 1;
        if (!(ok = mbar_wait_limit(v_full + vs, (i >> 1) & 1) && mbar_wait_limit(p_full, i & 1))) break;
        tc_fence_after();
        const uint32_t v_addr = smem_u32(v_s + vs * NV * PA_BOX);
        if (elect_one()) {
#pragma unroll
          for (int s = 0; s < PA_N / 16; ++s) umma_ts(tm_o, tm_p + s * 8, pa_desc_mn(v_addr + s * 2048), idesc_o, i > 0 || s > 0);
          if (SPLIT) {
#pragma unroll
            for (int s = 0; s < PA_N / 16; ++s) umma_ts(tm_o, tm_p + 64 + s * 8, pa_desc_mn(v_addr + s * 2048), idesc_o, 1);
          }
          umma_commit(pv_done);
          umma_commit(v_empty + vs);
        }
        __syncwarp();
      }
    }
  } else {
    // =========================== softmax: threads r and r + 128 own query row r (TMEM lane r), 64 columns of a tile each
    const int quarter = warp & 3, half = warp >> 2, r = quarter * 32 + lane, tk = t0 + r / hpc, h = h0 + r % hpc;
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    const int pos = pos0 + min(tk, t_last);
    const int lo = pa_mask_lo(pos, a.mask_kind, a.mask);
    constexpr float LOG2E = 1.4426950408889634f;
    constexpr int HC = PA_N / 2, OC = NV * 32;         // columns of S and of O per thread
    const float scale2 = a.scale * LOG2E, cap2 = a.softcap * LOG2E;
    // scores in the base-2 domain are f * v: the factor rides in the exponent's fma unless a cap or a sign needs it before
    const bool early = a.softcap > 0.f || !(scale2 > 0.f);
    const float f = early ? 1.f : scale2;
    float m = -1e30f, l = 0.f;
    if (a.sink != nullptr) { m = a.sink[h] * LOG2E; l = half == 0 ? 1.f : 0.f; }
    {
      // the query tile: 16 rows per warp, four rows of 128 bytes per instruction, all asked for before the first is written
      const int ch = lane & 7;
      uint4 x[4][NS];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int qr = warp * 16 + i * 4 + (lane >> 3), qt = t0 + qr / hpc;
        const __nv_bfloat16* src = a.q + static_cast<int64_t>(start + min(qt, t_last)) * a.q_tok + static_cast<int64_t>(h0 + qr % hpc) * a.q_head;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          const int c = s * 64 + ch * 8;
          x[i][s] = make_uint4(0u, 0u, 0u, 0u);
          if (qt <= t_last && c < a.d) x[i][s] = ldg_v4(src + c);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int qr = warp * 16 + i * 4 + (lane >> 3);
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          const int c = s * 64 + ch * 8;
          if (a.rot_dims > 0 && c >= a.d1) {             // turned where the rotation asks for it
            uint32_t* xp = &x[i][s].x;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int d = c - a.d1 + 2 * e;
              if (d + 1 < a.rot_dims) {
                float sn, cs;
                sincosf(static_cast<float>(pos0 + t0 + qr / hpc) * a.freq[d / 2], &sn, &cs);
                sn *= a.rot_mult; cs *= a.rot_mult;
                const float u = bf16lo(xp[e]), w = bf16hi(xp[e]);
                xp[e] = pack_bf16(u * cs - w * sn, w * cs + u * sn);
              }
            }
          }
          *reinterpret_cast<uint4*>(q_s + s * PA_BOX + qr * 128 + ((ch ^ (qr & 7)) << 4)) = x[i][s];
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(q_full);
    }
    for (int j = 0; j < n_tiles; ++j) {
      const int st = j & 1, c0 = j * PA_N + half * HC;                 // place of the thread's first column in the key list
      ok = ok && mbar_wait_limit(s_full + st, (j >> 1) & 1);           // a wait that ran out does not leave the loop: the row barrier below
      tc_fence_after();
      uint32_t v[HC];
#pragma unroll
      for (int c = 0; c < HC; c += 32) tmem_ld32(tm_s + st * PA_N + half * HC + lanes + c, v + c);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(s_empty + st);
      if (early) {
        const float fx = a.softcap > 0.f ? a.scale / a.softcap : scale2;
        float big = 0.f;
#pragma unroll
        for (int c = 0; c < HC; ++c) {
          const float x = __uint_as_float(v[c]) * fx;
          v[c] = __float_as_uint(x);
          big = fmaxf(big, fabsf(x));
        }
        if (a.softcap > 0.f) {
          // cap tanh(s / cap); while all of the warp's |s / cap| are at most 0.4 by its series (the next term is below 2e-9 of x)
          if (__all_sync(0xffffffffu, big <= 0.4f)) {
#pragma unroll
            for (int c = 0; c < HC; ++c) {
              const float x = __uint_as_float(v[c]), y = x * x;
              float t = fmaf(y, 21844.f / 6081075.f, -1382.f / 155925.f);
              t = fmaf(y, t, 62.f / 2835.f);
              t = fmaf(y, t, -17.f / 315.f);
              t = fmaf(y, t, 2.f / 15.f);
              t = fmaf(y, t, -1.f / 3.f);
              v[c] = __float_as_uint(cap2 * fmaf(x * y, t, x));
            }
          } else {
#pragma unroll
            for (int c = 0; c < HC; ++c) v[c] = __float_as_uint(cap2 * tanhf(__uint_as_float(v[c])));
          }
        }
      }
      // visible columns: of the list's front those below n_pre, behind it from `first` (or below `keep`) up to `last`
      const int j0 = c0 - pre_r + jl, last = pos - j0, first = lo - j0, keep = keep_in - j0, fr_end = pre_r - c0, fr_vis = n_pre - c0;
      if (!__all_sync(0xffffffffu, last >= HC - 1 && first <= 0 && fr_end <= 0)) {
        uint32_t see[2];
#pragma unroll
        for (int w = 0; w < 2; ++w)
          see[w] = (pa_below(fr_vis - 32 * w) & pa_below(fr_end - 32 * w)) |
                   (~pa_below(fr_end - 32 * w) & pa_below(last + 1 - 32 * w) & (~pa_below(first - 32 * w) | pa_below(keep - 32 * w)));
#pragma unroll
        for (int c = 0; c < HC; ++c)
          if (!(see[c >> 5] >> (c & 31) & 1u)) v[c] = __float_as_uint(-INFINITY);
      }
      float x0 = -INFINITY, x1 = -INFINITY, x2 = -INFINITY, x3 = -INFINITY;
#pragma unroll
      for (int c = 0; c < HC; c += 8) {
        x0 = fmaxf(x0, fmaxf(__uint_as_float(v[c]), __uint_as_float(v[c + 1])));
        x1 = fmaxf(x1, fmaxf(__uint_as_float(v[c + 2]), __uint_as_float(v[c + 3])));
        x2 = fmaxf(x2, fmaxf(__uint_as_float(v[c + 4]), __uint_as_float(v[c + 5])));
        x3 = fmaxf(x3, fmaxf(__uint_as_float(v[c + 6]), __uint_as_float(v[c + 7])));
      }
      float* ex = row_x + (j & 1) * 2 * PA_M;
      ex[half * PA_M + r] = fmaxf(fmaxf(x0, x1), fmaxf(x2, x3)) * f;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      const float mx = fmaxf(ex[r], ex[PA_M + r]);
      // ---- the running maximum moves in steps of more than 2^8
      const bool grow = mx > m + (j == 0 ? 0.f : 8.f);
      if (__any_sync(0xffffffffu, grow)) {
        const float n = fmaxf(m, mx), alpha = pa_ex2(m - n);
        m = n;
        l *= alpha;
        if (j > 0) {
          ok = ok && mbar_wait_limit(pv_done, (j - 1) & 1);
          tc_fence_after();
#pragma unroll 1
          for (int c = half * OC; ok && c < half * OC + OC; c += 32) {
            uint32_t o[32];
            tmem_ld32(tm_o + lanes + c, o);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
            tmem_st32(tm_o + lanes + c, o);
          }
          tmem_st_wait();
        }
      }
      // ---- weights, their sum, and their bf16 parts: v[0 .. 31] the rounded weights, rest[] the remainders
      float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
      uint32_t rest[SPLIT ? HC / 2 : 1];
#pragma unroll
      for (int c = 0; c < HC; c += 4) {
        const float w0 = pa_ex2(fmaf(__uint_as_float(v[c]), f, -m)), w1 = pa_ex2(fmaf(__uint_as_float(v[c + 1]), f, -m));
        const float w2 = pa_ex2(fmaf(__uint_as_float(v[c + 2]), f, -m)), w3 = pa_ex2(fmaf(__uint_as_float(v[c + 3]), f, -m));
        s0 += w0; s1 += w1; s2 += w2; s3 += w3;
        const uint32_t p0 = pack_bf16(w0, w1), p1 = pack_bf16(w2, w3);
        if constexpr (SPLIT) {
          rest[c / 2] = pack_bf16(w0 - bf16lo(p0), w1 - bf16hi(p0));
          rest[c / 2 + 1] = pack_bf16(w2 - bf16lo(p1), w3 - bf16hi(p1));
        }
        v[c / 2] = p0;
        v[c / 2 + 1] = p1;
      }
      l += (s0 + s1) + (s2 + s3);
      if (j > 0) {
        ok = ok && mbar_wait_limit(pv_done, (j - 1) & 1);              // the weights of the tile before have been read
        tc_fence_after();
      }
      tmem_st32(tm_p + half * 32 + lanes, v);
      if constexpr (SPLIT) tmem_st32(tm_p + 64 + half * 32 + lanes, rest);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    // both halves of the sum (the exchange buffer of the last tile is still being read: the other one)
    float* ex = row_x + (n_tiles & 1) * 2 * PA_M;
    ex[half * PA_M + r] = l;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    l = ex[r] + ex[PA_M + r];
    const bool live = tk <= t_last;
    const int64_t row = start + min(tk, t_last);
    float inv = 1.0f / l;
    if (a.gate != nullptr && !a.gate_el) inv *= sigmoid_f(__bfloat162float(a.gate[row * a.ldg + h]));
    const int64_t obase = (row * a.H + h) * a.dv + half * OC;
    const bool gated = a.gate != nullptr && a.gate_el;
    uint32_t gw[OC / 2];                               // the row's gates, asked for while the last products run
    if (gated) {
      const __nv_bfloat16* gr = a.gate + row * a.ldg + static_cast<int64_t>(h) * a.dv + half * OC;
      if (a.gate_vec) {
#pragma unroll
        for (int e = 0; e < OC / 2; e += 4) {
          const uint4 x = ldg_v4(gr + 2 * e);
          gw[e] = x.x; gw[e + 1] = x.y; gw[e + 2] = x.z; gw[e + 3] = x.w;
        }
      } else {                                         // pairs: the caller checked the alignment
#pragma unroll
        for (int e = 0; e < OC / 2; ++e) gw[e] = *reinterpret_cast<const uint32_t*>(gr + 2 * e);
      }
    }
    if (ok) ok = mbar_wait_limit(pv_done, (n_tiles - 1) & 1);
    tc_fence_after();
    if (ok) {
#pragma unroll
      for (int c = 0; c < OC; c += 32) {
        uint32_t o[32];
        tmem_ld32(tm_o + lanes + half * OC + c, o);
        tmem_ld_wait();
        float y[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) y[e] = __uint_as_float(o[e]) * inv;
        if (gated) {
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            y[2 * e] *= pa_sigmoid(bf16lo(gw[c / 2 + e]));
            y[2 * e + 1] *= pa_sigmoid(bf16hi(gw[c / 2 + e]));
          }
        }
        if (live && a.out_f32) {
          float* op = static_cast<float*>(a.out) + obase + c;
#pragma unroll
          for (int e = 0; e < 32; e += 4) *reinterpret_cast<float4*>(op + e) = make_float4(y[e], y[e + 1], y[e + 2], y[e + 3]);
        } else if (live) {
          __nv_bfloat16* op = static_cast<__nv_bfloat16*>(a.out) + obase + c;
#pragma unroll
          for (int e = 0; e < 32; e += 8)
            stg_v4(op + e, make_uint4(pack_bf16(y[e], y[e + 1]), pack_bf16(y[e + 2], y[e + 3]), pack_bf16(y[e + 4], y[e + 5]), pack_bf16(y[e + 6], y[e + 7])));
        }
        __syncwarp();
      }
    }
    tc_fence_before();
  }
  if (!ok && lane == 0) atomicAdd(&g_prompt_attn_timeouts, 1);
  __syncthreads();
  if (warp == PA_SOFT) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

bool prompt_attn_applies(const PromptAttnArgs& a) {
  const bool rows8 = a.q_tok % 8 == 0 && a.q_head % 8 == 0 && a.k_row % 8 == 0 && a.k_head % 8 == 0 && a.k2_row % 8 == 0 && a.v_row % 8 == 0 &&
                     a.v_head % 8 == 0;
  // a key's last slice may reach into its neighbour's columns: whole steps of 16 keep them out of the products
  return rows8 && a.d % 16 == 0 && a.d <= 192 && (a.d1 == a.d || a.d1 % 64 == 0) && (a.dv == 64 || a.dv == 128) && aligned16(a.q) &&
         aligned16(a.k) && (a.k2 == nullptr || aligned16(a.k2)) && aligned16(a.v) && aligned16(a.out) &&
         (a.gate == nullptr || !a.gate_el || (reinterpret_cast<uintptr_t>(a.gate) % 4 == 0 && a.ldg % 2 == 0));
}

template <int NS, int NV, bool SPLIT>
static int go_prompt(const char* what, PromptAttnArgs a, cudaStream_t st) {
  auto kern = prompt_attn_kernel<NS, NV, SPLIT>;
  constexpr int smem = 1024 + (NS * 3 + NV * 2) * PA_BOX + 128 + 4 * PA_M * 4;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return cuda_fail(e, what);
  a.page_shift = -1;
  for (int x = 0; x < 30; ++x)
    if (a.page == 1 << x) a.page_shift = x;
  a.gate_vec = a.gate != nullptr && aligned16(a.gate) && a.ldg % 8 == 0;
  a.box_rows = a.max_new >= 64 ? 64 : 16;              // short portions are bound by the host: two tensor maps instead of four
  while (a.block_tables != nullptr && a.page % a.box_rows) a.box_rows /= 2;
  // rows are the caller's business (slots come from its tables): the maps do not bound them
  PromptMaps maps{};
  int rc = B2TTS_OK;
  for (int x = 0; x < 2 && rc == B2TTS_OK; ++x) {
    if (x == 1 && a.box_rows <= 16) { maps.k[1] = maps.k[0]; maps.k2[1] = maps.k2[0]; maps.v[1] = maps.v[0]; break; }
    const int rows = x ? 16 : a.box_rows;
    rc = make_x_tensor_map(&maps.k[x], a.k, a.k_row, 1 << 30, static_cast<int>(a.k_row), rows, what);
    if (rc == B2TTS_OK && a.d1 < a.d) rc = make_x_tensor_map(&maps.k2[x], a.k2, a.k2_row, 1 << 30, a.d - a.d1, rows, what);
    if (rc == B2TTS_OK) rc = make_x_tensor_map(&maps.v[x], a.v, a.v_row, 1 << 30, static_cast<int>(a.v_row), rows, what);
  }
  if (rc != B2TTS_OK) return rc;
  int hpc = 1;                                         // heads of a key head that share a CTA's rows: a power of two up to 8
  while (hpc < 8 && (a.H / a.G) % (2 * hpc) == 0) hpc *= 2;
  const int per = PA_M / hpc;
  kern<<<dim3((a.max_new + per - 1) / per, a.H / hpc, a.n_seqs), PA_THREADS, smem, st>>>(a, hpc, maps);
  B2_CHECK_LAUNCH(what);
  return B2TTS_OK;
}

int launch_prompt_attn(const char* what, const PromptAttnArgs& a, cudaStream_t st) {
  const int ns = (a.d + 63) / 64;
#define PA_GO(NS, NV) return a.split_weights ? go_prompt<NS, NV, true>(what, a, st) : go_prompt<NS, NV, false>(what, a, st)
  if (a.dv == 64) {
    if (ns == 1) PA_GO(1, 1);
    if (ns == 2) PA_GO(2, 1);
    PA_GO(3, 1);
  }
  if (ns == 1) PA_GO(1, 2);
  if (ns == 2) PA_GO(2, 2);
  PA_GO(3, 2);
#undef PA_GO
}

}  // namespace row
}  // namespace b2

extern "C" int b2tts_prompt_attn_timeouts(void) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, b2::row::g_prompt_attn_timeouts, sizeof(int)) != cudaSuccess) return -1;
  return v;
}
