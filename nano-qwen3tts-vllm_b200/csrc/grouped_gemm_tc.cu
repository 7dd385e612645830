// grouped_gemm_tc.cu - the grouped products of grouped_gemm.cu on tcgen05 for prompt-sized groups (bf16).
//
// Bound: tensor cores.  A persistent CTA per SM walks (expert, 128 rows, 256 columns of W) tiles; the tiles of one expert's weight
// columns follow each other (row blocks fastest), so a weight tile is read from HBM once and then from L2.  Per 64-wide slice of K
//   rows      of consecutive pairs: one TMA box; of tokens, which lie anywhere in A: 16-byte asynchronous copies of four gather
//             warps, written where the SWIZZLE_128B operand wants them (32 TMA gathers of four rows were the bound of the
//             kernel: 18 cycles a row, 439 us for the down product below against 162 us with boxes);
//   weights   one TMA box of 256 rows (two of 128, gate and up, for gated experts);
// and four tcgen05.mma of 128 x 256 x 16, the shape that runs at the tensor pipe's pace with one issuing thread.  The float sums
// stay in TMEM, two accumulators of 256 columns: four epilogue warps empty one (activation, bf16, 16-byte stores of a thread's
// own row) while the next tile's products fill the other.  Rows behind a group's end are computed (they repeat the group's
// first row, or are the next group's) and not stored.
//
// 8192 tokens, top 2 of 16 experts, width 2048, inner size 3072: gate/up with its SiLU product 345 us (1195 TFLOP/s; on mma.sync
// 1470 us and 158 us for the product behind it), down 166 us (1240 TFLOP/s; 703 us).
#include <algorithm>

#include "grouped_gemm.cuh"
#include "umma.cuh"
#include "waits.cuh"

namespace b2 {

constexpr int TC_BM = 128, TC_BN = 256, TC_STAGES = 4, TC_THREADS = 192;
constexpr int TC_GATHER_WARPS = 4, TC_LAG = 2;     // slices a gather warp issues before it waits for the first of them
constexpr int TC_A_BYTES = TC_BM * G_BK * 2, TC_B_BYTES = TC_BN * G_BK * 2, TC_STAGE_BYTES = TC_A_BYTES + TC_B_BYTES;
constexpr size_t TC_SMEM = 1024 + static_cast<size_t>(TC_STAGES) * TC_STAGE_BYTES + 256;

// How often a wait inside the kernel ran out, see waits.cuh.
__device__ int g_grouped_tc_timeouts = 0;
__device__ __forceinline__ void report_timeout(int* word) {
  *reinterpret_cast<volatile int*>(word) = atomicAdd(&g_grouped_tc_timeouts, 1) + 1;
  __threadfence_system();
}

struct GroupedTcArgs {
  const int32_t* offsets;
  const int32_t* sorted_pair;
  __nv_bfloat16* c; int64_t ldc;
  const __nv_bfloat16* a; int64_t lda;     // rows of tokens (GATHER)
  int E, N, K, top, out_by_pair;
  int nk, nb;                              // slices of K, column blocks per expert
  float limit, alpha;
  int* timeouts;                           // host memory, see report_timeout
};

// tile -> (expert, row block, column block), for tile numbers that only grow
struct TileWalk {
  int e = 0, cum = 0, seg0, seg1;
  __device__ __forceinline__ TileWalk(const GroupedTcArgs& p) { seg0 = p.offsets[0]; seg1 = p.offsets[1]; }
  __device__ __forceinline__ bool at(const GroupedTcArgs& p, int tile, int& m0, int& n) {
    int nm = (seg1 - seg0 + TC_BM - 1) / TC_BM;
    while (tile >= cum + nm * p.nb) {
      cum += nm * p.nb;
      if (++e >= p.E) return false;
      seg0 = seg1;
      seg1 = p.offsets[e + 1];
      nm = (seg1 - seg0 + TC_BM - 1) / TC_BM;
    }
    n = (tile - cum) / nm;
    m0 = seg0 + (tile - cum - n * nm) * TC_BM;
    return true;
  }
};

template <int ACT, bool GATHER>
__global__ void __launch_bounds__(TC_THREADS + (GATHER ? TC_GATHER_WARPS * 32 : 0), 1)
grouped_gemm_tc_kernel(const GroupedTcArgs p, const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w) {
  extern __shared__ uint8_t tc_smem_dyn[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(tc_smem_dyn) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + TC_STAGES * TC_STAGE_BYTES);
  uint64_t* empty = full + TC_STAGES;
  uint64_t* acc_full = empty + TC_STAGES;          // [2]
  uint64_t* acc_empty = acc_full + 2;              // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < TC_STAGES; ++s) { mbar_init(full + s, GATHER ? 1 + TC_GATHER_WARPS : 1); mbar_init(empty + s, 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(acc_full + b, 1); mbar_init(acc_empty + b, 4); }
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  constexpr bool GATED = ACT >= GG_CLAMPED;
  constexpr int BF = GATED ? TC_BN / 2 : TC_BN;    // output columns per tile
  TileWalk walk(p);
  int m0, n;
  bool ok = true;

  if (warp == 0) {
    // =========================== producer: weights, and the rows when they are consecutive
    int it = 0;
    for (int tile = blockIdx.x; ok && walk.at(p, tile, m0, n); tile += gridDim.x) {
      const int w_row = walk.e * p.N + n * BF;
      for (int kt = 0; kt < p.nk; ++kt, ++it) {
        const int st = it % TC_STAGES;
        if (!(ok = mbar_wait_limit(empty + st, ((it / TC_STAGES) & 1) ^ 1))) break;
        uint8_t* sa = smem + st * TC_STAGE_BYTES;
        uint8_t* sb = sa + TC_A_BYTES;
        if (elect_one()) {
          mbar_expect_tx(full + st, GATHER ? TC_B_BYTES : TC_STAGE_BYTES);
          tma_load_2d(sb, &tmap_w, kt * G_BK, w_row, full + st);
          if (GATED) tma_load_2d(sb + TC_B_BYTES / 2, &tmap_w, kt * G_BK, w_row + p.N / 2, full + st);
          if (!GATHER) tma_load_2d(sa, &tmap_a, kt * G_BK, m0, full + st);
        }
        __syncwarp();
      }
    }
    if (!ok) {                                     // never expected: let this CTA's copies land before it leaves
      for (int i = max(0, it - TC_STAGES); i < it; ++i) mbar_wait_limit(full + i % TC_STAGES, (i / TC_STAGES) & 1);
    }
  } else if (warp == 1) {
    // =========================== MMA issuer
    const uint32_t idesc = umma_idesc_bf16(TC_BN);
    int it = 0, t = 0;
    for (int tile = blockIdx.x; ok && walk.at(p, tile, m0, n); tile += gridDim.x, ++t) {
      const int b = t & 1;
      if (!(ok = mbar_wait_limit(acc_empty + b, ((t >> 1) & 1) ^ 1))) break;
      tc_fence_after();
      for (int kt = 0; kt < p.nk; ++kt, ++it) {
        const int st = it % TC_STAGES;
        if (!(ok = mbar_wait_limit(full + st, (it / TC_STAGES) & 1))) break;
        tc_fence_after();
        const uint32_t a_lo = umma_desc_lo_sw128(smem_u32(smem + st * TC_STAGE_BYTES));
        const uint32_t b_lo = umma_desc_lo_sw128(smem_u32(smem + st * TC_STAGE_BYTES + TC_A_BYTES));
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < G_BK / 16; ++k) umma_bf16_lo(tmem + b * TC_BN, a_lo + 2 * k, b_lo + 2 * k, idesc, kt > 0 || k > 0);
          umma_commit(empty + st);
          if (kt == p.nk - 1) umma_commit(acc_full + b);
        }
        __syncwarp();
      }
    }
    // every commit of this warp has arrived (and with it every product) before the CTA gives up its TMEM and shared memory
    for (int i = max(0, it - TC_STAGES); i < it; ++i) ok = mbar_wait_limit(empty + i % TC_STAGES, (i / TC_STAGES) & 1) && ok;
  } else if (GATHER && warp >= TC_THREADS / 32) {
    // =========================== gather: warp w copies rows 32 w .. + 31 of the tile, four rows of 128 bytes per instruction
    const int w = warp - TC_THREADS / 32, ch = lane & 7;
    uint32_t dst[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = w * 32 + i * 4 + (lane >> 3);
      dst[i] = r * 128 + ((ch ^ (r & 7)) << 4);
    }
    int it = 0;
    auto hand_over = [&](int done) {               // the copies of slice `done` have landed: visible to the tensor core, then signalled
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(full + done % TC_STAGES);
    };
    for (int tile = blockIdx.x; ok && walk.at(p, tile, m0, n); tile += gridDim.x) {
      const __nv_bfloat16* src[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int s = m0 + w * 32 + i * 4 + (lane >> 3);
        src[i] = p.a + static_cast<int64_t>(p.sorted_pair[s < walk.seg1 ? s : m0] / p.top) * p.lda;
      }
      for (int kt = 0; kt < p.nk; ++kt, ++it) {
        const int st = it % TC_STAGES;
        if (!(ok = mbar_wait_limit(empty + st, ((it / TC_STAGES) & 1) ^ 1))) break;
        uint8_t* sa = smem + st * TC_STAGE_BYTES;
        const int k = kt * G_BK + ch * 8;
#pragma unroll
        for (int i = 0; i < 8; ++i) cp_async_16(sa + dst[i], src[i] + (k < p.K ? k : 0), k < p.K);
        cp_async_commit();
        if (it >= TC_LAG) {
          cp_async_wait<TC_LAG>();
          hand_over(it - TC_LAG);
        }
      }
    }
    cp_async_wait<0>();
    for (int i = max(0, it - TC_LAG); ok && i < it; ++i) hand_over(i);
  } else {
    // =========================== epilogue: thread r owns row r (TMEM lane r)
    const int quarter = warp & 3, r = quarter * 32 + lane;
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    const int cols = GATED ? p.N / 2 : p.N;
    int t = 0;
    for (int tile = blockIdx.x; ok && walk.at(p, tile, m0, n); tile += gridDim.x, ++t) {
      const int b = t & 1, s = m0 + r;
      int orow = -1;
      if (s < walk.seg1) orow = p.out_by_pair ? p.sorted_pair[s] : s;
      if (!(ok = mbar_wait_limit(acc_full + b, (t >> 1) & 1))) break;
      tc_fence_after();
      __nv_bfloat16* crow = p.c + static_cast<int64_t>(orow) * p.ldc + n * BF;
      const int left = cols - n * BF;              // columns of this tile that exist
#pragma unroll 1
      for (int c = 0; c < min(BF, left); c += 32) {
        uint32_t v[32], u[GATED ? 32 : 1];
        tmem_ld32(tmem + lanes + b * TC_BN + c, v);
        if constexpr (GATED) tmem_ld32(tmem + lanes + b * TC_BN + TC_BN / 2 + c, u);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float x = __uint_as_float(v[i + e]);
            if constexpr (GATED) f[e] = gated_value<ACT>(x, __uint_as_float(u[i + e]), p.limit, p.alpha);
            else if constexpr (ACT == GG_RELU_SQ) { const float z = fmaxf(x, 0.f); f[e] = z * z; }
            else f[e] = x;
          }
          if (orow >= 0 && c + i < left)           // whole groups of eight: the output's column count is a multiple of eight
            stg_v4(crow + c + i, make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7])));
        }
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty + b);
    }
  }
  if (!ok && lane == 0) report_timeout(p.timeouts);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// Where this kernel is the faster one.  A tile costs it about 4 us of start and end (gathered rows 5, gated sums 10: one warp a
// scheduler forms 128 columns of them) and then little per slice of K; the kernels of grouped_gemm.cu start in 3 us and pay more per
// slice, and more when their 128-row tiles are mostly empty.  So what decides is K, and with a short K how many of their 128-column
// tiles there are to spread over the GPU.  Measured over 4 to 256 experts, K 64 to 4096, 64 to 6144 rows of W and 13 to 1024 rows an
// expert (4566 shapes, weights cold): always this kernel is 10 % from the faster of the two on average, this rule 0.7 %.  Some of the
// lines, here / there in us:
//   more than 16 rows an expert   gated     16 experts, 256 rows of W, 32 rows     K 256 14 / 9      K 1024 20 / 22    K 2048 34 / 41
//                                           64 experts, 1024 rows of W, 128 rows   K 64 36 / 27      K 256 37 / 40     K 1024 53 / 107
//                                 gathered  64 experts, 512 rows of W, 17 rows     K 64 13 / 9       K 256 14 / 13     K 1024 22 / 33
//   13 to 16 rows (32-row tiles)  gated     16 experts, 6144 rows of W             K 2048 102 / 84   (128 experts, 1536 rows of W, K 768: 80 / 98)
//                                 gathered  16 experts, 2048 rows of W             K 1024 21 / 18    K 2048 32 / 31
//                                 in order  16 experts, 6144 rows of W             K 1024 39 / 45    K 2048 70 / 82
// Sizes that do not fill 16-byte output vectors, rows of W that a copy's 32-bit coordinates cannot name and rows shorter than one
// slice stay there too.
bool grouped_tc_applies(int n_pairs, int experts, int w_rows, int k, bool gated, bool in_by_token, int64_t ldc, const void* c) {
  const int64_t e = experts, col_tiles = (w_rows + 127) / 128;
  if (n_pairs <= 12 * e || k < G_BK || (gated ? w_rows / 2 : w_rows) % 8 != 0 || ldc % 8 != 0 || !aligned16(c) || e * w_rows >= (1ll << 31))
    return false;
  if (n_pairs <= 16 * e) {
    const int64_t tiles = (e + n_pairs / 32) * col_tiles;
    if (gated) return e >= 128 && tiles >= 1200;
    return in_by_token ? (e >= 64 && tiles >= 700) || (k >= 1536 && tiles <= 70) : k > 640 || tiles >= 600;
  }
  const int64_t tiles = (e + n_pairs / 128) * col_tiles;
  if (gated) return k >= 768 || (k >= 128 && tiles * k >= 280000) || (w_rows <= 64 && n_pairs > 24 * e);
  return k >= 192 || tiles * k >= 40000;
}

int grouped_tc_check(const char* what) { return wait_check(WAITS_GROUPED, what); }

template <int ACT, bool GATHER>
static int go(const char* what, const GroupedTcArgs& p, const CUtensorMap& ma, const CUtensorMap& mw, int tiles, cudaStream_t st) {
  auto kern = grouped_gemm_tc_kernel<ACT, GATHER>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(TC_SMEM));
  if (e != cudaSuccess) return cuda_fail(e, what);
  kern<<<std::min(tiles, sm_count()), TC_THREADS + (GATHER ? TC_GATHER_WARPS * 32 : 0), TC_SMEM, st>>>(p, ma, mw);
  B2_CHECK_LAUNCH(what);
  return B2TTS_OK;
}

int launch_grouped_tc(const char* what, const void* a, int64_t lda, const void* w, void* c, int64_t ldc, const int32_t* offsets,
                      const int32_t* sorted_pair, int n_pairs, int experts, int n, int k, int top, int in_by_token, int out_by_pair,
                      int act, float limit, float alpha, cudaStream_t st) {
  int* word = wait_word(WAITS_GROUPED);
  B2_REQUIRE(word != nullptr, B2TTS_ECUDA, "%s: no host memory for the kernel's status", what);
  const bool gated = act >= GG_CLAMPED;
  CUtensorMap ma{}, mw;
  int rc = make_x_tensor_map(&mw, w, k, experts * n, k, gated ? TC_BN / 2 : TC_BN, what);
  if (rc == B2TTS_OK && !in_by_token) rc = make_x_tensor_map(&ma, a, lda, n_pairs, k, TC_BM, what);
  if (rc != B2TTS_OK) return rc;
  GroupedTcArgs p{};
  p.offsets = offsets; p.sorted_pair = sorted_pair;
  p.a = static_cast<const __nv_bfloat16*>(a); p.lda = lda;
  p.c = static_cast<__nv_bfloat16*>(c); p.ldc = ldc;
  p.E = experts; p.N = n; p.K = k; p.top = top; p.out_by_pair = out_by_pair;
  p.nk = (k + G_BK - 1) / G_BK;
  const int cols = gated ? n / 2 : n, bf = gated ? TC_BN / 2 : TC_BN;
  p.nb = (cols + bf - 1) / bf;
  p.limit = limit; p.alpha = alpha;
  p.timeouts = word;
  const int64_t tiles = (static_cast<int64_t>(n_pairs + TC_BM - 1) / TC_BM + experts) * p.nb;
  const int most = static_cast<int>(std::min<int64_t>(tiles, 1 << 20));
#define GT_GO(ACT) return in_by_token ? go<ACT, true>(what, p, ma, mw, most, st) : go<ACT, false>(what, p, ma, mw, most, st)
  switch (act) {
    case GG_NONE: GT_GO(GG_NONE);
    case GG_RELU_SQ: GT_GO(GG_RELU_SQ);
    case GG_CLAMPED: return go<GG_CLAMPED, true>(what, p, ma, mw, most, st);     // gated products read tokens
    default: return go<GG_SILU, true>(what, p, ma, mw, most, st);
  }
#undef GT_GO
}

}  // namespace b2

extern "C" int b2tts_grouped_gemm_timeouts(void) {
  return b2::wait_count(b2::WAITS_GROUPED);
}
extern "C" int b2tts_grouped_gemm_check(void) {
  for (int k = 0; k < b2::WAITS_KINDS; ++k) {
    const int rc = b2::wait_check(k, "check_waits");
    if (rc != B2TTS_OK) return rc;
  }
  return B2TTS_OK;
}

namespace b2 {
// One wait of the kind that the kernel has, on a barrier that nothing arrives at, with a short limit.
__global__ void grouped_tc_lost_wait_kernel(int* word) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) { mbar_init(&bar, 1); mbar_fence_init(); }
  __syncwarp();
  if (!mbar_wait_limit(&bar, 0, 64) && threadIdx.x == 0) report_timeout(word);
}
}  // namespace b2

extern "C" int b2tts_grouped_gemm_lose_wait(void* stream) {
  using namespace b2;
  int* word = wait_word(WAITS_GROUPED);
  B2_REQUIRE(word != nullptr, B2TTS_ECUDA, "grouped_gemm_lose_wait: no host memory");
  grouped_tc_lost_wait_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(word);
  B2_CHECK_LAUNCH("grouped_gemm_lose_wait");
  return B2TTS_OK;
}
