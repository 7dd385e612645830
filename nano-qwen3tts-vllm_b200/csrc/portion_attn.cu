// portion_attn.cu - attention of prompt portions (more than one new token of a sequence) on the 5th-generation tensor cores:
// keys and values through block tables or in rows of their own, sliding-window, chunk or causal masks with kept first keys, sinks, score
// caps, gates; or sigmoid weights with a logarithmic distance bias in a window.  bf16 operands; scores, weights, sums and the outputs'
// accumulators are float.
//
// A persistent CTA per SM takes items of one or two row tiles.  A row tile is 128 query rows: 128 / HPC tokens times HPC heads that share
// a key head; the two tiles of an item are neighbouring tokens and share the key tiles (128 keys) that pass through one ring of
// 16 KiB slots (128 rows x 64 columns).  Twenty warps:
//   softmax   two groups of eight, a group per row tile, two threads of a warp per row: each takes 64 scores from TMEM, and gives the weights
//             back in the same columns as the A operand of the second product, a bf16 pair hi + lo each (16 bits);
//   MMA       S = Q K^T (128 x 128 x d), O += P V (128 x dv x 128, twice: hi and lo) for the tiles in turn, so that one tile's products run
//             while the other tile's weights are formed.  A tile's next S overwrites its weights: the products of one thread
//             run in the order of their issue;
//   loader    queries (one box of 64 columns x HPC heads x tokens per slice), keys and values as boxes of R rows inside pages;
//   cleaner   zeros the value rows of a tile that no query of the item sees (behind the last key, before the window): their weights are
//             zero, but what a page holds there may be infinite.
// A row's maximum is the running one: where one key has most of the weight, its weight is then 1 and carries no rounding.  (A lazy one, moved in steps
// of 2^8, left it a weight with a rounding of its own: outputs of 2000 peaked keys 1.21 times as far from 64 bits with weights
// rounded once, 1.9 times with pairs in float.  O is scaled more often for it: layers 2 % longer, single tiles 10 %.)  The sum is that of the weights as the
// products see them, rounded, so that what rounding adds to all of them cancels.
//
// Bound: the issue of the tensor core's products.  A key tile of a row tile is 24 of them of 64 cycles (1536); the issuer's own instructions and
// barriers between two tiles make that about 2300, and the weights (64 exponents, splits and sums a thread) are ready before that.  An item
// starts and ends in about 12000 cycles (first key tile under a mask, last products, division and gates).  Two threads a row and 64 scores
// each in two passes over TMEM keep everything in 96 registers: spilled ones went through L2, since shared memory leaves L1 next to nothing
// (one thread a row with 40 spilled registers: 143 us for the case below; one barrier per slot of the ring instead of per tile: 20 us more).
// 4 prompts of 2048 tokens, 16 heads over 8 of 128, window 1024 + 4 kept, element gates: 131 us (mma.sync, 64 queries per CTA: 547 us; 31 at
// the tensor core's rate; 123 with the lazy maximum); causal with a score cap, 4448 tokens: 133 us (579 us); latent
// heads of 192 over expanded keys, 4 x 2048 causal: 150 us; prompts that are their own keys, weights rounded once, 4096 + 1531 causal: 114 us (152 us
// one query tile a CTA).  Sigmoid weights (two special-function results and a table's number a pair), window 1024, 4138 tokens: 77 us (143 us).
//
// Values that a query does not see have a weight of zero, and zero times infinity is not a number: an infinite value that some query of an item sees
// reaches the others that share its key tile, up to two row tiles of tokens (256 / HPC) in front of it.  On mma.sync that is up to 78 tokens.
//
// Every copy is bounded: maps have the true extents of their tensors, so a row that a block table should not name reads zeros.  Every
// commit of the last products is waited for before the CTA leaves.  tests/test_portion_bookkeeping.py plays the items, ring and barriers on the CPU.
#include <algorithm>

#include "portion_attn.cuh"
#include "umma.cuh"
#include "waits.cuh"

namespace b2 {
namespace row {

constexpr int PO_N = 128, PO_SLOT = 128 * 128;         // keys per tile; bytes of a slot: 128 rows of 64 bf16 columns
constexpr int PO_SOFT = 16, PO_THREADS = 640, PO_ITEMS = 48;           // softmax warps; items a CTA takes at most
constexpr int PO_MMA = 16, PO_LOADER = 17, PO_CLEANER = 18, PO_LISTER = 19;
__device__ int g_portion_timeouts = 0;                 // see waits.cuh
__device__ __forceinline__ void po_report(int* word) {
  *reinterpret_cast<volatile int*>(word) = atomicAdd(&g_portion_timeouts, 1) + 1;
  __threadfence_system();
}

// Low word of an MN-major SWIZZLE_128B operand: a K index (key) is a 128-byte row of 64 columns; LBO: the next 64 columns (the next slot),
// SBO: 8 keys.  The high word is that of the K-major operands.
__device__ __forceinline__ uint32_t po_desc_mn_lo(uint32_t addr) { return ((addr & 0x3ffffu) >> 4) | (static_cast<uint32_t>(PO_SLOT >> 4) << 16); }
// D [128 x n] (+)= A (TMEM: two bf16 per column, lane = row) B (shared memory)
__device__ __forceinline__ void po_umma_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b64 db;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t"
      "}"
      :: "r"(d), "r"(a), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(UMMA_DESC_HI_SW128) : "memory");
}
// 32 columns of 16 lanes for lanes 0 .. 15 of the warp and 32 columns of the same lanes, SPLIT columns further, for the others
template <int SPLIT>
__device__ __forceinline__ void po_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x32bx2.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32], %33;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
        "=r"(r[31])
      : "r"(taddr), "n"(SPLIT));
}
template <int SPLIT>
__device__ __forceinline__ void po_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x32bx2.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16], %17;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr), "n"(SPLIT));
}
template <int SPLIT>
__device__ __forceinline__ void po_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x32bx2.x16.b32 [%0], %17, {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
         "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "n"(SPLIT) : "memory");
}
template <int SPLIT>
__device__ __forceinline__ void po_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x32bx2.x32.b32 [%0], %33, {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
        "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]),
        "n"(SPLIT) : "memory");
}
__device__ __forceinline__ void po_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float po_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 1 / (1 + 2^x): about 2 ulp; 2^big = inf and 1 / inf = 0
__device__ __forceinline__ float po_sigmoid(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(1.0f + po_ex2(x)));
  return y;
}
__device__ __forceinline__ int po_mask_lo(int i, int kind, int mask) {
  if (mask <= 0) return 0;
  return kind == 0 ? max(0, i - mask + 1) : (i / mask) * mask;
}
// the n lowest of 32 bits (none for n <= 0, all from 32 on)
__device__ __forceinline__ uint32_t po_below(int n) { return n <= 0 ? 0u : n >= 32 ? 0xffffffffu : (1u << n) - 1u; }

// Columns of a row tile's weights of 16 keys: step s < 8 the rounded weights of keys 16 s .., s >= 8 the remainders of keys 16 (s - 8) ..  32 keys
// have the 32 columns where their scores were: 16 of rounded weights, 16 of remainders.
__device__ __forceinline__ constexpr int po_weights_at(int s) { return (s >> 1 & 3) * 32 + (s >> 3) * 16 + (s & 1) * 8; }

struct PortionPlan { int hpc, hpc_shift, sms, few, box_rows, page_shift, gate_vec, tab_row; int* timeouts; };    // set by the launch
struct PortionMaps { CUtensorMap q, k, k2, v; };
struct PortionEntry { int t0, end, b, hg, start, pos0; };       // tokens t0 .. end - 1 of sequence b, heads of group hg

// What every role knows of an item.  The key list: kept first keys that the lowest bound of the item hides, in whole boxes, then
// [jl, j_hi] from a multiple of R on; where the boxes of the kept keys reach that bound, one run from key 0.
struct PortionItem {
  int b, t0, end, start, pos0, h0, j_lo, j_hi, jl, pre_r, n_pre, keep_in, n_keys, n_tiles, per;
  __device__ __forceinline__ PortionItem(const PortionArgs& a, const PortionPlan& p, const PortionEntry& e) {
    per = 128 >> p.hpc_shift;
    b = e.b;
    t0 = e.t0; end = e.end;
    start = e.start; pos0 = e.pos0;
    h0 = e.hg << p.hpc_shift;
    const int R = p.box_rows, keep_r = (a.keep_first + R - 1) & ~(R - 1);
    j_lo = po_mask_lo(pos0 + t0, a.mask_kind, a.mask);
    j_hi = pos0 + end - 1;
    const bool pre = a.keep_first > 0 && keep_r <= j_lo;
    n_pre = pre ? a.keep_first : 0;
    pre_r = pre ? keep_r : 0;
    jl = pre || a.keep_first == 0 ? j_lo & ~(R - 1) : 0;
    keep_in = pre ? 0 : a.keep_first;                  // kept keys that are part of the run
    n_keys = pre_r + j_hi - jl + 1;
    n_tiles = (n_keys + PO_N - 1) / PO_N;
  }
  __device__ __forceinline__ bool has(int g) const { return t0 + g * per < end; }
};

// The key tiles of which some row of row tile g sees a key: those of the kept keys, [0, front), and [first, last]
struct PortionSpan {
  int front = 0, first = 0, last = -1;
  PortionSpan() = default;
  __device__ __forceinline__ PortionSpan(const PortionArgs& a, const PortionItem& m, int g) {
    if (!m.has(g)) return;
    const int t = m.t0 + g * m.per, lo = po_mask_lo(m.pos0 + t, a.mask_kind, a.mask);
    first = (max(lo - m.jl, 0) + m.pre_r) / PO_N;
    last = (m.pos0 + min(m.end, t + m.per) - 1 - m.jl + m.pre_r) / PO_N;
    front = min((m.n_pre + m.keep_in + PO_N - 1) / PO_N, last + 1);
  }
  __device__ __forceinline__ bool has(int j) const { return j < front || (j >= first && j <= last); }
};

// softmax weights as bf16 pairs, or rounded once; sigmoid weights as pairs
enum { PO_PAIRS = 0, PO_ROUNDED = 1, PO_SIGMOID = 2 };
// slots of the ring; sigmoid weights need room for their tables beside it
template <int NS, int MODE> constexpr int po_slots() { return MODE == PO_SIGMOID ? 8 : NS == 1 ? 12 : NS == 2 ? 10 : 8; }
constexpr int PO_DEEP = 8, PO_BAR_BYTES = 512, PO_TAIL = PO_BAR_BYTES + PO_ITEMS * 24, PO_SMEM = 232448;
template <int NS, int MODE> constexpr int po_smem() { return 1024 + (2 * NS + po_slots<NS, MODE>()) * PO_SLOT + PO_TAIL; }
static_assert(po_smem<1, PO_PAIRS>() <= PO_SMEM && po_smem<2, PO_PAIRS>() <= PO_SMEM && po_smem<3, PO_PAIRS>() <= PO_SMEM, "shared memory of a CTA");

// NS: 64-column slices of q and k; NV: of v
template <int NS, int NV, int MODE>
__global__ void __launch_bounds__(PO_THREADS, 1)
portion_attn_kernel(const PortionArgs a, const PortionPlan p, const __grid_constant__ PortionMaps maps) {
  constexpr int SLOTS = po_slots<NS, MODE>(), PER_TILE = NS + NV;
  constexpr bool SIG = MODE == PO_SIGMOID;
  constexpr int STEPS = PO_N / 16 * (MODE == PO_ROUNDED ? 1 : 2);        // products of a tile's weights and values
  static_assert(2 * NS + NV <= SLOTS, "a tile's values beside two tiles of keys");
  static_assert(SLOTS / PER_TILE + 1 < PO_DEEP, "tiles in the ring at once");
  extern __shared__ uint8_t po_smem_dyn[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(po_smem_dyn) + 1023) & ~uintptr_t(1023));
  uint8_t* q_s = smem;                                 // [2 tiles][NS]
  uint8_t* ring = q_s + 2 * NS * PO_SLOT;              // keys of tile 0, values of tile 0, keys of tile 1, ..
  // key tile t of the CTA, counted over its items, at t % PO_DEEP: keys there, values there, values cleaned; its
  // keys and the values of the tile before given back
  uint64_t* k_full = reinterpret_cast<uint64_t*>(ring + SLOTS * PO_SLOT);
  uint64_t *v_full = k_full + PO_DEEP, *clean = v_full + PO_DEEP, *empty = clean + PO_DEEP;
  uint64_t *q_full = empty + PO_DEEP, *q_empty = q_full + 2, *s_full = q_empty + 2, *p_full = s_full + 2;
  uint64_t *o_full = p_full + 2, *t_full = o_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(t_full + 2);
  int* n_items_s = reinterpret_cast<int*>(tmem_slot + 1);
  PortionEntry* list = reinterpret_cast<PortionEntry*>(reinterpret_cast<uint8_t*>(k_full) + PO_BAR_BYTES);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  if (warp == PO_LISTER) {
    // The CTA's items: number i of the valid (tile, sequence, heads), late tiles first (they are the longest under a causal mask), for
    // i = c, 2 G - 1 - c, 3 G - 1 - c, 3 G + c, 4 G + c, ..: who begins with a long one gets the short ones, and a round that is not full goes to
    // those with the least so far
    const int per_shift = 7 - p.hpc_shift, per = 1 << per_shift, groups = a.H >> p.hpc_shift, c = blockIdx.x;
    auto len_of = [&](int b) { return a.cu != nullptr ? a.cu[b + 1] - a.cu[b] : a.seq_len[b]; };
    auto pos_of = [&](int b) { return a.cu != nullptr ? 0 : a.seq_pos0[b]; };
    auto start_of = [&](int b) { return a.cu != nullptr ? a.cu[b] : a.seq_start[b]; };
    const bool here = lane < a.n_seqs;                 // the first 32 sequences' numbers stay in registers
    const int len0 = here ? len_of(lane) : 0, pos00 = here ? pos_of(lane) : 0, start0 = here ? start_of(lane) : 0, least = a.one_token ? 1 : 2;
    // f(tokens, position of the first) of each sequence, summed over the step's
    auto over_sequences = [&](auto f) {
      int n = 0;
      for (int b = lane; b < a.n_seqs; b += 32) {
        const int len = b < 32 ? len0 : len_of(b);
        if (len >= least) n += f(len, b < 32 ? pos00 : pos_of(b));
      }
      return __reduce_add_sync(0xffffffffu, n);
    };
    // One row tile an item, or two.  An item of two takes a third longer than one of one, so it is the better one once some multiprocessor gets two single
    // tiles of two thirds of the longest's keys: two where they fill the chip, or where there are more such long single tiles than
    // multiprocessors.  The host knows the longest portion only, and beside decoded tokens that says little: every CTA counts, with the
    // same result.  16 heads over 8 of 128, window of 1024, one / two in us: 1500 tokens 34 / 43, 2048 52 / 43, 6 x 200 behind 800 50 / 38.
    int span = per, G = gridDim.x;
    if (!p.few) {
      int keys = 0;
      int64_t items = static_cast<int64_t>(groups) * over_sequences([&](int len, int pos0) {
        keys = max(keys, pos0 + len);
        return (len + 2 * per - 1) >> (per_shift + 1);
      });
      span = 2 * per;
      if (items < p.sms) {
        keys = __reduce_max_sync(0xffffffffu, keys);
        const int far = (a.mask > 0 ? min(keys, a.mask) : keys) / 3 * 2;
        const int n_long = over_sequences([&](int len, int pos0) { return max(((len + per - 1) >> per_shift) - (max(far - pos0, 0) >> per_shift), 0); });
        if (static_cast<int64_t>(groups) * n_long <= p.sms) {
          span = per;
          items = static_cast<int64_t>(groups) * over_sequences([&](int len, int) { return (len + per - 1) >> per_shift; });
        }
      }
      // the CTAs that have a part in it: the others were launched for portions that are not there
      G = static_cast<int>(max(min(items, static_cast<int64_t>(p.sms)), (items + PO_ITEMS - 1) / PO_ITEMS));
    }
    int k = 0, cum = 0, want = c < G ? c : 0x7fffffff;
    for (int tile = (a.max_new + span - 1) / span - 1; tile >= 0 && k < PO_ITEMS; --tile) {
      for (int base = 0; base < a.n_seqs && k < PO_ITEMS; base += 32) {
        const int len = base == 0 ? len0 : base + lane < a.n_seqs ? len_of(base + lane) : 0;
        const unsigned live = __ballot_sync(0xffffffffu, len >= least && tile * span < len);
        const int cnt = __popc(live) * groups;
        while (k < PO_ITEMS && want < cum + cnt) {
          const int at = want - cum, rank = at / groups;
          const int at_b = static_cast<int>(__fns(live, 0, rank + 1));
          if (lane == at_b)
            list[k] = PortionEntry{tile * span, min(len, (tile + 1) * span), base + lane, at - rank * groups, base == 0 ? start0 : start_of(base + lane),
                                   base == 0 ? pos00 : pos_of(base + lane)};
          ++k;
          want = k * G + ((k + 1) >> 1 & 1 ? G - 1 - c : c);
        }
        cum += cnt;
      }
    }
    if (lane == 0) *n_items_s = k;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < PO_DEEP; ++s) {
      mbar_init(k_full + s, 1); mbar_init(v_full + s, 1); mbar_init(clean + s, 1); mbar_init(empty + s, 1);
    }
    for (int g = 0; g < 2; ++g) {
      mbar_init(q_full + g, 1); mbar_init(q_empty + g, 1); mbar_init(s_full + g, 1); mbar_init(p_full + g, PO_SOFT / 2); mbar_init(o_full + g, 1);
      mbar_init(t_full + g, PO_SOFT / 2);
    }
    mbar_fence_init();
  }
  if (warp == PO_MMA) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;                    // S and weights of tile g: columns 128 g; O: 256 + 128 g
  const int n_items = *n_items_s;
  bool ok = true;

  if (warp >= PO_SOFT) {
    if (warp == PO_LOADER) {
      // =========================== loader
      int t = 0, slot = 0, q_uses[2] = {0, 0};         // the tile, the next slot, query tiles loaded so far
      for (int x = 0; ok && x < n_items; ++x) {
        const PortionItem m(a, p, list[x]);
        const int g = m.h0 / (a.H / a.G), gv = g % a.Gv, R = p.box_rows;
        const int32_t* bt = a.block_tables != nullptr ? a.block_tables + static_cast<int64_t>(m.b) * a.bt_stride : nullptr;
        const int row0 = bt != nullptr ? 0 : a.cu != nullptr ? m.start : a.key_start[m.b];
        const int n1 = min(NS, (a.d1 + 63) / 64);
        // lane = box * 4 + slice; row of the lane's box of tile j, a tile ahead: nothing waits for the load of the page's number here
        const int box = lane >> 2, sl = lane & 3, boxes = PO_N / R;
        struct Row { int pg, off; };
        auto row_of = [&](int j) {
          const int vi = j * PO_N + box * R;
          if (box >= boxes || vi >= m.n_keys) return Row{0, 0};
          const int key = vi < m.pre_r ? vi : m.jl + vi - m.pre_r;
          if (bt == nullptr) return Row{0, row0 + key};
          const int pg = p.page_shift >= 0 ? key >> p.page_shift : key / a.page;
          return Row{bt[pg], key - pg * a.page};
        };
        // the next n slots: keys or values of tile t, columns x0 ..
        auto fill = [&](int j, Row r, int n, bool keys, int x0) {
          // what lay there: the ring holds SLOTS slots, given back in order, values with the keys of the tile behind them
          const int old = t * PER_TILE + (keys ? 0 : NS) + n - 1 - SLOTS, ot = (old + NV) / PER_TILE;
          if (old >= 0) ok = mbar_wait_limit(empty + (ot & (PO_DEEP - 1)), (ot / PO_DEEP) & 1);
          if (!ok) return;
          const int nb = (min(m.n_keys - j * PO_N, PO_N) + R - 1) / R;
          uint64_t* bar = (keys ? k_full : v_full) + (t & (PO_DEEP - 1));
          if (lane == 0) mbar_expect_tx(bar, n * nb * R * 128);
          __syncwarp();
          if (box < nb && sl < n) {
            const int at = slot + sl < SLOTS ? slot + sl : slot + sl - SLOTS, row = r.pg * a.page + r.off;
            uint8_t* dst = ring + at * PO_SLOT + box * R * 128;
            if (keys && sl >= n1) tma_load_2d(dst, &maps.k2, (sl - n1) * 64, row, bar);
            else tma_load_2d(dst, keys ? &maps.k : &maps.v, x0 + sl * 64, row, bar);
          }
          __syncwarp();
          slot = slot + n < SLOTS ? slot + n : slot + n - SLOTS;
        };
        Row cur = row_of(0);
        for (int j = 0; ok && j < m.n_tiles; ++j, ++t) {
          fill(j, cur, NS, true, g * a.d1);
          for (int tg = 0; ok && j == 0 && tg < 2; ++tg) {
            if (!m.has(tg)) continue;
            if (!(ok = mbar_wait_limit(q_empty + tg, (q_uses[tg] & 1) ^ 1))) break;
            if (lane == 0) mbar_expect_tx(q_full + tg, NS * PO_SLOT);
            __syncwarp();
            if (lane < NS) tma_load_3d(q_s + (tg * NS + lane) * PO_SLOT, &maps.q, lane * 64, m.h0, m.start + m.t0 + tg * m.per, q_full + tg);
            __syncwarp();
            ++q_uses[tg];
          }
          const Row mine = cur;
          if (j + 1 < m.n_tiles) cur = row_of(j + 1);
          if (ok) fill(j, mine, NV, false, gv * a.dv);
        }
      }
      // every copy has landed before the CTA leaves
      for (int i = max(0, t - PO_DEEP); i < t; ++i)
        ok = mbar_wait_limit(k_full + (i & (PO_DEEP - 1)), (i / PO_DEEP) & 1) && mbar_wait_limit(v_full + (i & (PO_DEEP - 1)), (i / PO_DEEP) & 1) && ok;
      for (int tg = 0; tg < 2; ++tg)
        if (q_uses[tg] > 0) ok = mbar_wait_limit(q_full + tg, (q_uses[tg] - 1) & 1) && ok;
    } else if (warp == PO_CLEANER) {
      // =========================== cleaner: value rows that nothing sees
      int t = 0, slot = 0;                             // of the tile's keys
      for (int x = 0; ok && x < n_items; ++x) {
        const PortionItem m(a, p, list[x]);
        for (int j = 0; ok && j < m.n_tiles; ++j, ++t) {
          const int v0 = slot + NS < SLOTS ? slot + NS : slot + NS - SLOTS;
          slot = slot + PER_TILE < SLOTS ? slot + PER_TILE : slot + PER_TILE - SLOTS;
          if (!(ok = mbar_wait_limit(v_full + (t & (PO_DEEP - 1)), (t / PO_DEEP) & 1))) break;
          bool wrote = false;
#pragma unroll
          for (int i = 0; i < PO_N / 32; ++i) {
            const int r = i * 32 + lane, vi = j * PO_N + r, key = m.jl + vi - m.pre_r;
            const bool keep = vi < m.n_pre || (vi >= m.pre_r && vi < m.n_keys && (key >= m.j_lo || key < m.keep_in));
            if (!keep) {
              wrote = true;
#pragma unroll
              for (int s = 0; s < NV; ++s) {
                uint4* row = reinterpret_cast<uint4*>(ring + (v0 + s < SLOTS ? v0 + s : v0 + s - SLOTS) * PO_SLOT + r * 128);
#pragma unroll
                for (int c = 0; c < 8; ++c) row[(c + lane) & 7] = make_uint4(0u, 0u, 0u, 0u);
              }
            }
          }
          if (wrote) fence_proxy_async();
          __syncwarp();
          if (lane == 0) mbar_arrive(clean + (t & (PO_DEEP - 1)));
        }
      }
    } else if (warp == PO_MMA) {
      // =========================== MMA issuer: per key tile j and row tile g: O_g += P_g(j - 1) V(j - 1), then S_g(j)
      const uint32_t idesc_s = umma_idesc_bf16(PO_N), idesc_half = umma_idesc_bf16(64) | (1u << 16),
                     idesc_o = umma_idesc_bf16(NV * 64) | (1u << 16);                   // the value operand is MN-major
      const uint32_t ring_k = umma_desc_lo_sw128(smem_u32(ring)), ring_v = po_desc_mn_lo(smem_u32(ring)), q_lo = umma_desc_lo_sw128(smem_u32(q_s));
      constexpr uint32_t SLOT_LO = PO_SLOT >> 4;
      int t = 0, slot = 0, q_uses[2] = {0, 0}, p_uses[2] = {0, 0}, o_uses[2] = {0, 0};
      for (int x = 0; ok && x < n_items; ++x) {
        const PortionItem m(a, p, list[x]);
        const PortionSpan span[2] = {PortionSpan(a, m, 0), PortionSpan(a, m, 1)};
        int v_slot = 0;                                // of the tile before
        bool was[2] = {false, false}, begun[2] = {false, false};
        for (int j = 0; ok && j <= m.n_tiles; ++j) {
          // everything but the weights is waited for in front: what the issuer does between two products leaves the tensor core idle
          const int at = t & (PO_DEEP - 1), before = (t - 1) & (PO_DEEP - 1);
          if (j > 0) ok = mbar_wait_limit(clean + before, ((t - 1) / PO_DEEP) & 1);
          if (ok && j < m.n_tiles) ok = mbar_wait_limit(k_full + at, (t / PO_DEEP) & 1);
          const uint32_t v_lo = ring_v + v_slot * SLOT_LO;
          // values in the ring's last and first slot (rings whose length no whole tiles make up come to that): 64 columns at a time
          const bool apart = NV == 2 && SLOTS % PER_TILE != 0 && (NS + NV) % 2 != 0 && v_slot == SLOTS - 1;
          uint32_t k_lo[NS];
#pragma unroll
          for (int sl = 0; sl < NS; ++sl) k_lo[sl] = ring_k + (slot + sl < SLOTS ? slot + sl : slot + sl - SLOTS) * SLOT_LO;
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const uint32_t tm_o = tmem + 256 + g * 128, tm_p = tmem + g * 128;
            const bool now = j < m.n_tiles && span[g].has(j), last_s = j == span[g].last, last_o = j - 1 == span[g].last;
            if (ok && was[g]) {
              ok = mbar_wait_limit(p_full + g, p_uses[g] & 1);
              ++p_uses[g];
            }
            if (ok && now && !begun[g]) ok = mbar_wait_limit(q_full + g, q_uses[g] & 1);
            if (ok && (was[g] || now)) {
              tc_fence_after();
              if (elect_one()) {
                if (was[g]) {
                  if (!apart) {
                    po_umma_ts(tm_o, tm_p, v_lo, idesc_o, begun[g]);
#pragma unroll
                    for (int s = 1; s < STEPS; ++s) po_umma_ts(tm_o, tm_p + po_weights_at(s), v_lo + (s & 7) * 128, idesc_o, 1);
                  } else {
#pragma unroll 1
                    for (int half = 0; half < 2; ++half)
#pragma unroll
                      for (int s = 0; s < STEPS; ++s)
                        po_umma_ts(tm_o + half * 64, tm_p + po_weights_at(s), (half ? ring_v : v_lo) + (s & 7) * 128, idesc_half, begun[g] || s);
                  }
                  if (last_o) umma_commit(o_full + g);
                }
                if (now) {
#pragma unroll
                  for (int sl = 0; sl < NS; ++sl)
#pragma unroll
                    for (int s = 0; s < 4; ++s) umma_bf16_lo(tm_p, q_lo + (g * NS + sl) * SLOT_LO + 2 * s, k_lo[sl] + 2 * s, idesc_s, sl | s);
                  umma_commit(s_full + g);
                  if (last_s) umma_commit(q_empty + g);
                }
                if (g == 1 && j < m.n_tiles) umma_commit(empty + at);
              }
              __syncwarp();
              begun[g] = begun[g] || was[g];
              o_uses[g] += was[g] && last_o;
              q_uses[g] += now && last_s;
            } else if (g == 1 && j < m.n_tiles) {
              if (ok && elect_one()) umma_commit(empty + at);
              __syncwarp();
            }
            was[g] = now;
          }
          if (j < m.n_tiles) {
            v_slot = slot + NS < SLOTS ? slot + NS : slot + NS - SLOTS;
            slot = slot + PER_TILE < SLOTS ? slot + PER_TILE : slot + PER_TILE - SLOTS;
            ++t;
          }
        }
      }
      // every commit of this warp has arrived (and with it every product) before the CTA gives up its TMEM and shared memory
      for (int i = max(0, t - PO_DEEP); i < t; ++i)
        ok = mbar_wait_limit(empty + (i & (PO_DEEP - 1)), (i / PO_DEEP) & 1) && ok;
      for (int g = 0; g < 2; ++g) {
        if (q_uses[g] > 0) ok = mbar_wait_limit(q_empty + g, (q_uses[g] - 1) & 1) && ok;
        if (o_uses[g] > 0) ok = mbar_wait_limit(o_full + g, (o_uses[g] - 1) & 1) && ok;
      }
    }
  } else {
    // =========================== softmax: lanes i and i + 16 of a warp share row r (TMEM lane r), 64 keys of a tile each
    const int tg = warp >> 3, r0 = (warp & 3) * 32 + (warp & 4) * 4, half = lane >> 4, r = r0 + (lane & 15);
    const uint32_t tm_s = tmem + (static_cast<uint32_t>(r0) << 16) + tg * 128, tm_o = tm_s + 256;
    constexpr int HK = PO_N / 2, OC = NV * 32;         // keys and output columns of a thread
    constexpr float LOG2E = 1.4426950408889634f;
    const float scale2 = a.scale * LOG2E, cap2 = a.softcap * LOG2E;
    // scores in the base-2 domain are f * v: the factor rides in the exponent's fma unless a cap or a sign needs it before
    const bool early = a.softcap > 0.f || !(scale2 > 0.f);
    const float f = early ? 1.f : scale2;
    const bool gated = a.gate != nullptr && a.gate_el;
    // SIG: log2(e) (r1 ln(1 + r2 x) - pb) of the distances x, a table per head, for each half of the lanes its own copy (rows of p.tab_row floats, which
    // puts the 32 numbers that a warp reads at once into different banks)
    float* tab = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(k_full) + PO_TAIL) + tg * 2 * p.hpc * p.tab_row;
    const float* my_tab = tab + (half * p.hpc + (r & (p.hpc - 1))) * p.tab_row;
    int s_uses = 0, o_uses = 0, t_uses = 0;
    for (int x = 0; ok && x < n_items; ++x) {
      // What an item needs in its masked tiles and in the end is formed there again: the loop over whole tiles has no registers for it
      float m = -1e30f, l = 0.f;
      PortionSpan span;
      int whole0, whole1;                              // key tiles that all rows of the warp see whole
      {
        const PortionItem it(a, p, list[x]);
        if (!it.has(tg)) continue;
        span = PortionSpan(a, it, tg);
        if (!SIG && a.sink != nullptr) {
          const float s = a.sink[it.h0 + (r & (p.hpc - 1))] * LOG2E;
          m = s < m ? m : s;                           // a sink that is off (-inf, the lowest float) leaves the maximum finite: its weight is 0 behind the first key
          l = half == 0 ? 1.f : 0.f;
        }
        const int t_first = it.t0 + tg * it.per, t_last = min(it.end, t_first + it.per) - 1;
        const int lo = po_mask_lo(it.pos0 + min(t_first + ((r0 + 15) >> p.hpc_shift), t_last), a.mask_kind, a.mask);    // the highest of its rows
        whole0 = (max(lo - it.jl, 0) + it.pre_r + PO_N - 1) / PO_N;
        whole1 = (it.pos0 + min(t_first + (r0 >> p.hpc_shift), t_last) + 1 - it.jl + it.pre_r) / PO_N;
        if (gated)                                     // read in the end, far from any cache by then
          asm volatile("prefetch.global.L2 [%0];" :: "l"(a.gate + static_cast<int64_t>(it.start + min(t_first + (r >> p.hpc_shift), t_last)) * a.ldg +
                                                         static_cast<int64_t>(it.h0 + (r & (p.hpc - 1))) * a.dv + half * OC));
      }
      if constexpr (SIG) {                             // nobody reads the last item's table any more: its last weights are all there
        const int h0 = list[x].hg << p.hpc_shift;
        for (int i = threadIdx.x & 255; i < p.hpc * a.mask; i += 256) {
          const int h = i / a.mask, dist = i - h * a.mask;
          const float y = LOG2E * (a.r1[h0 + h] * log1pf(a.r2[h0 + h] * static_cast<float>(dist)) - a.pb[h0 + h]);
          tab[h * p.tab_row + dist] = y;
          tab[(p.hpc + h) * p.tab_row + dist] = y;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(t_full + tg);
        if (!(ok = mbar_wait_limit(t_full + tg, t_uses & 1))) break;
        ++t_uses;
      }
      bool first = true;
      for (int j = 0; ok && j <= span.last; ++j) {
        if (!span.has(j)) continue;
        if (!(ok = mbar_wait_limit(s_full + tg, s_uses & 1))) break;
        ++s_uses;
        tc_fence_after();
        const bool masked = j < whole0 || j >= whole1;
        if (early || masked) {                         // scores are put right where they lie
          // visible columns, counted from the thread's first: of the list's front those below fr_vis, behind it from `from` (or below `keep`) to `to`
          const PortionItem it(a, p, list[x]);
          const int t_first = it.t0 + tg * it.per, pos = it.pos0 + min(t_first + (r >> p.hpc_shift), min(it.end, t_first + it.per) - 1);
          const int c0 = j * PO_N + half * HK, j0 = c0 - it.pre_r + it.jl;
          int to = pos - j0, from = po_mask_lo(pos, a.mask_kind, a.mask) - j0, keep = it.keep_in - j0, fr_end = it.pre_r - c0, fr_vis = it.n_pre - c0;
#pragma unroll 1
          for (int c = 0; c < HK; c += 32) {
            uint32_t v[32];
            po_ld32<HK>(tm_s + c, v);
            tmem_ld_wait();
            if (early) {
              const float fx = a.softcap > 0.f ? a.scale / a.softcap : scale2;
              float big = 0.f;
#pragma unroll
              for (int e = 0; e < 32; ++e) {
                const float y = __uint_as_float(v[e]) * fx;
                v[e] = __float_as_uint(y);
                big = fmaxf(big, fabsf(y));
              }
              if (a.softcap > 0.f) {
                // cap tanh(s / cap); while all of the warp's |s / cap| are at most 0.4 by its series (the next term is below 2e-9 of it)
                if (__all_sync(0xffffffffu, big <= 0.4f)) {
#pragma unroll
                  for (int e = 0; e < 32; ++e) {
                    const float z = __uint_as_float(v[e]), y = z * z;
                    float t = fmaf(y, 21844.f / 6081075.f, -1382.f / 155925.f);
                    t = fmaf(y, t, 62.f / 2835.f);
                    t = fmaf(y, t, -17.f / 315.f);
                    t = fmaf(y, t, 2.f / 15.f);
                    t = fmaf(y, t, -1.f / 3.f);
                    v[e] = __float_as_uint(cap2 * fmaf(z * y, t, z));
                  }
                } else {
#pragma unroll
                  for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(cap2 * tanhf(__uint_as_float(v[e])));
                }
              }
            }
            if (SIG && masked) {                       // the exponent's argument, from the other side, while the distance is at hand
              const int dist = pos - j0 - c;
#pragma unroll
              for (int e = 0; e < 32; ++e)
                v[e] = __float_as_uint(fmaf(__uint_as_float(v[e]), f, -my_tab[min(max(dist - e, 0), a.mask - 1)]));
            }
            if (masked) {
              const uint32_t see = (po_below(fr_vis) & po_below(fr_end)) | (~po_below(fr_end) & po_below(to + 1) & (~po_below(from) | po_below(keep)));
#pragma unroll
              for (int e = 0; e < 32; ++e)
                if (!(see & (1u << e))) v[e] = __float_as_uint(-INFINITY);
              to -= 32; from -= 32; keep -= 32; fr_end -= 32; fr_vis -= 32;
            }
            po_st32<HK>(tm_s + c, v);
          }
          po_st_wait();
        }
        if constexpr (!SIG) {
          // two passes over the scores, which stay in TMEM meanwhile: a thread has no registers for all of them beside the weights' parts
          float mx;
          {
            uint32_t v[HK];
            po_ld32<HK>(tm_s, v);
            po_ld32<HK>(tm_s + 32, v + 32);
            tmem_ld_wait();
            float x0 = -INFINITY, x1 = -INFINITY, x2 = -INFINITY, x3 = -INFINITY;
#pragma unroll
            for (int c = 0; c < HK; c += 8) {
              x0 = fmaxf(x0, fmaxf(__uint_as_float(v[c]), __uint_as_float(v[c + 1])));
              x1 = fmaxf(x1, fmaxf(__uint_as_float(v[c + 2]), __uint_as_float(v[c + 3])));
              x2 = fmaxf(x2, fmaxf(__uint_as_float(v[c + 4]), __uint_as_float(v[c + 5])));
              x3 = fmaxf(x3, fmaxf(__uint_as_float(v[c + 6]), __uint_as_float(v[c + 7])));
            }
            mx = fmaxf(fmaxf(x0, x1), fmaxf(x2, x3));
          }
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16)) * f;
          // ---- the running maximum.  These scores were issued behind the last weight products, so O is at rest
          const bool grow = mx > m;
          if (__any_sync(0xffffffffu, grow)) {
            const float n = grow ? mx : m, alpha = po_ex2(m - n);
            m = n;
            l *= alpha;
            if (!first) {
#pragma unroll 1
              for (int c = 0; c < OC; c += 32) {
                uint32_t o[32];
                po_ld32<OC>(tm_o + c, o);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
                po_st32<OC>(tm_o + c, o);
              }
            }
          }
          first = false;
        }
        // ---- weights, their bf16 parts in place of the scores, and the sum of those: pairs' remainders in sb, minus the rounded weights in sa
        const uint64_t f2 = f2_pack(f, f), m2 = f2_pack(-m, -m);
        uint64_t sa = 0, sb = 0;
#pragma unroll 1
        for (int part = 0; part < HK; part += 32) {
          uint32_t v[32], hi[16], rest[16];
          po_ld32<HK>(tm_s + part, v);
          tmem_ld_wait();
          if constexpr (SIG) {
            if (masked) {
#pragma unroll
              for (int c = 0; c < 32; ++c) v[c] = __float_as_uint(-__uint_as_float(v[c]));
            } else {
              const PortionEntry& e = list[x];
              const int tk = e.t0 + tg * (128 >> p.hpc_shift) + (r >> p.hpc_shift), pos = e.pos0 + min(tk, e.end - 1);
              const PortionItem it(a, p, e);
              const float* at = my_tab + (pos - (j * PO_N + half * HK + it.jl) - part);
#pragma unroll
              for (int c = 0; c < 32; ++c) v[c] = __float_as_uint(fmaf(__uint_as_float(v[c]), -f, at[-c]));
            }
          }
#pragma unroll
          for (int c = 0; c < 32; c += 4) {
            const uint32_t* vv = v + c;
            float w0, w1, w2, w3, r0, r1, r2, r3;
            if constexpr (SIG) {
              w0 = po_sigmoid(__uint_as_float(vv[0])); w1 = po_sigmoid(__uint_as_float(vv[1]));
              w2 = po_sigmoid(__uint_as_float(vv[2])); w3 = po_sigmoid(__uint_as_float(vv[3]));
            } else {
              f2_unpack(f2_fma(f2_pack(__uint_as_float(vv[0]), __uint_as_float(vv[1])), f2, m2), w0, w1);
              f2_unpack(f2_fma(f2_pack(__uint_as_float(vv[2]), __uint_as_float(vv[3])), f2, m2), w2, w3);
              w0 = po_ex2(w0); w1 = po_ex2(w1); w2 = po_ex2(w2); w3 = po_ex2(w3);
            }
            const uint64_t wa = f2_pack(w0, w1), wb = f2_pack(w2, w3);
            const uint32_t p0 = pack_bf16(w0, w1), p1 = pack_bf16(w2, w3);
            if constexpr (MODE != PO_ROUNDED) {
              const uint32_t n0 = p0 ^ 0x80008000u, n1 = p1 ^ 0x80008000u;
              const uint64_t h0 = f2_pack(bf16lo(n0), bf16hi(n0)), h1 = f2_pack(bf16lo(n1), bf16hi(n1));
              f2_unpack(f2_add(wa, h0), r0, r1);
              f2_unpack(f2_add(wb, h1), r2, r3);
              const uint32_t q0 = pack_bf16(r0, r1), q1 = pack_bf16(r2, r3);
              if constexpr (!SIG) {
                sa = f2_add(f2_add(sa, h0), h1);
                sb = f2_add(f2_add(sb, f2_pack(bf16lo(q0), bf16hi(q0))), f2_pack(bf16lo(q1), bf16hi(q1)));
              }
              rest[c / 2] = q0;
              rest[c / 2 + 1] = q1;
            } else {
              sa = f2_add(sa, f2_pack(bf16lo(p0), bf16hi(p0)));
              sb = f2_add(sb, f2_pack(bf16lo(p1), bf16hi(p1)));
            }
            hi[c / 2] = p0;
            hi[c / 2 + 1] = p1;
          }
          po_st16<HK>(tm_s + part, hi);
          if constexpr (MODE != PO_ROUNDED) po_st16<HK>(tm_s + part + 16, rest);
        }
        float s0, s1;
        f2_unpack(f2_add(MODE == PO_PAIRS ? sa ^ 0x8000000080000000ull : sa, sb), s0, s1);
        l += s0 + s1;
        po_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full + tg);
      }
      if (!ok) break;
      const PortionItem it(a, p, list[x]);
      const int t_first = it.t0 + tg * it.per, t_last = min(it.end, t_first + it.per) - 1, tk = t_first + (r >> p.hpc_shift), h = it.h0 + (r & (p.hpc - 1));
      const int64_t row = it.start + min(tk, t_last), obase = (row * a.H + h) * a.dv + half * OC;
      // 16 columns at a time, their gates a step ahead
      const __nv_bfloat16* gr = gated ? a.gate + row * a.ldg + static_cast<int64_t>(h) * a.dv + half * OC : nullptr;
      uint4 g0 = make_uint4(0u, 0u, 0u, 0u), g1 = g0;
      auto gates = [&](int c) {
        if (p.gate_vec) { g0 = ldg_v4(gr + c); g1 = ldg_v4(gr + c + 8); return; }
        const uint32_t* gw = reinterpret_cast<const uint32_t*>(gr + c);                    // pairs: the caller checked the alignment
        g0 = make_uint4(gw[0], gw[1], gw[2], gw[3]);
        g1 = make_uint4(gw[4], gw[5], gw[6], gw[7]);
      };
      if (gated) gates(0);
      l += __shfl_xor_sync(0xffffffffu, l, 16);
      float inv = SIG ? 1.f : 1.0f / l;
      if (a.gate != nullptr && !a.gate_el) inv *= sigmoid_f(__bfloat162float(a.gate[row * a.ldg + h]));
      if (!(ok = mbar_wait_limit(o_full + tg, o_uses & 1))) break;
      ++o_uses;
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < OC; c += 16) {
        uint32_t o[16];
        po_ld16<OC>(tm_o + c, o);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * inv);
        if (gated) {
          const uint32_t w[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
          if (c + 16 < OC) gates(c + 16);
          if (a.out_f32) {
#pragma unroll
            for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * sigmoid_f(e & 1 ? bf16hi(w[e >> 1]) : bf16lo(w[e >> 1])));
          } else {                                     // rounded to bf16 behind it: 203 us the window layer below, 208 with exact divisions
#pragma unroll
            for (int e = 0; e < 16; ++e)
              o[e] = __float_as_uint(__uint_as_float(o[e]) * sigmoid_for<__nv_bfloat16>(e & 1 ? bf16hi(w[e >> 1]) : bf16lo(w[e >> 1])));
          }
        }
        if (tk <= t_last && a.out_f32) {
          float* op = static_cast<float*>(a.out) + obase + c;
#pragma unroll
          for (int e = 0; e < 16; e += 4) *reinterpret_cast<uint4*>(op + e) = make_uint4(o[e], o[e + 1], o[e + 2], o[e + 3]);
        } else if (tk <= t_last) {
          __nv_bfloat16* op = static_cast<__nv_bfloat16*>(a.out) + obase + c;
#pragma unroll
          for (int e = 0; e < 16; e += 8) {
            const float* y = reinterpret_cast<const float*>(o + e);
            stg_v4(op + e, make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7])));
          }
        }
        __syncwarp();
      }
      tc_fence_before();                               // the next item's first weights tell the issuer that O may be overwritten
    }
  }
  if (!ok && lane == 0) po_report(p.timeouts);
  tc_fence_before();
  __syncthreads();
  if (warp == PO_MMA) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// One wait of the kernel's kind, on a barrier that nothing arrives at, with a short limit, and its report.
__global__ void portion_lost_wait_kernel(int* word) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) { mbar_init(&bar, 1); mbar_fence_init(); }
  __syncwarp();
  if (!mbar_wait_limit(&bar, 0, 64) && threadIdx.x == 0) po_report(word);
}

// floats of a row of the distance tables: the rows' tokens, heads and halves of a warp fall into different banks
static int po_tab_row(int window, int hpc) { return (window + 31) / 32 * 32 + 16 / hpc; }
// heads of a key head that share a row tile: a power of two up to 8; for sigmoid weights as many as have room for their tables (0: none)
static int po_heads(const PortionArgs& a) {
  int hpc = 1;
  while (hpc < 8 && (a.H / a.G) % (2 * hpc) == 0) hpc *= 2;
  if (a.r1 == nullptr) return hpc;
  const int room = PO_SMEM - (a.d == 64 ? po_smem<1, PO_SIGMOID>() : po_smem<2, PO_SIGMOID>());
  while (hpc > 0 && static_cast<int64_t>(4) * hpc * po_tab_row(a.mask, hpc) * 4 > room) hpc /= 2;
  return hpc;
}

// Whole slices of 64 columns (a box is never wider than a row), rows that copies can name and pages in whole boxes of 16 rows.
bool portion_attn_applies(const PortionArgs& a) {
  const bool rows8 = a.q_tok % 8 == 0 && a.q_head % 8 == 0 && a.k_row % 8 == 0 && a.k2_row % 8 == 0 && a.v_row % 8 == 0;
  return rows8 && a.d % 64 == 0 && a.d <= 192 && a.d1 % 64 == 0 && a.d1 <= a.d && (a.dv == 64 || a.dv == 128) && aligned16(a.q) &&
         aligned16(a.k) && (a.k2 == nullptr || aligned16(a.k2)) && aligned16(a.v) && aligned16(a.out) && a.n_rows > 0 &&
         a.n_rows < (1ll << 31) && (a.block_tables == nullptr || a.page % 16 == 0) && a.k_row >= static_cast<int64_t>(a.G) * a.d1 &&
         a.v_row >= static_cast<int64_t>(a.Gv) * a.dv &&
         (a.r1 == nullptr || (a.d == a.dv && a.d <= 128 && a.mask > 0 && a.mask_kind == 0 && a.keep_first == 0 && a.softcap == 0.f && po_heads(a) > 0)) &&
         (a.gate == nullptr || !a.gate_el || (reinterpret_cast<uintptr_t>(a.gate) % 4 == 0 && a.ldg % 2 == 0));
}

static unsigned long long g_portion_launches = 0;

template <int NS, int NV, int MODE>
static int go_portion(const char* what, const PortionArgs& a, const PortionPlan& p, const PortionMaps& maps, int grid, cudaStream_t st) {
  auto kern = portion_attn_kernel<NS, NV, MODE>;
  const int smem = po_smem<NS, MODE>() + (MODE == PO_SIGMOID ? 4 * p.hpc * p.tab_row * 4 : 0);
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return cuda_fail(e, what);
  kern<<<grid, PO_THREADS, smem, st>>>(a, p, maps);
  B2_CHECK_LAUNCH(what);
  __atomic_add_fetch(&g_portion_launches, 1ull, __ATOMIC_RELAXED);
  return B2TTS_OK;
}

int launch_portion_attn(const char* what, const PortionArgs& a, cudaStream_t st) {
  int rc = wait_check(WAITS_PORTIONS, what);
  if (rc != B2TTS_OK) return rc;
  PortionPlan p{};
  p.timeouts = wait_word(WAITS_PORTIONS);
  B2_REQUIRE(p.timeouts != nullptr, B2TTS_ECUDA, "%s: no host memory for the kernel's status", what);
  p.hpc = po_heads(a);
  while (1 << p.hpc_shift < p.hpc) ++p.hpc_shift;
  if (a.r1 != nullptr) p.tab_row = po_tab_row(a.mask, p.hpc);
  p.page_shift = -1;
  for (int x = 0; x < 30; ++x)
    if (a.page == 1 << x) p.page_shift = x;
  p.box_rows = 64;
  while (a.block_tables != nullptr && a.page % p.box_rows) p.box_rows /= 2;
  p.gate_vec = a.gate != nullptr && aligned16(a.gate) && a.ldg % 8 == 0;
  // A CTA per multiprocessor, or as many as their lists have room for; the kernel counts the items that there are
  const int per = 128 >> p.hpc_shift;
  auto items = [&](int tiles) { return static_cast<int64_t>((a.max_new + tiles * per - 1) / (tiles * per)) * (a.H / p.hpc) * a.n_seqs; };
  p.sms = sm_count();
  p.few = items(1) <= p.sms;                           // single tiles with a multiprocessor each, as long as the portions may be
  const int grid = static_cast<int>(std::max<int64_t>(std::min<int64_t>(items(1), p.sms), (items(2) + PO_ITEMS - 1) / PO_ITEMS));
  PortionMaps maps{};
  {
    const int64_t dims[3] = {a.d, a.H, a.n_tokens}, strides[2] = {a.q_head, a.q_tok};
    const int box[3] = {64, p.hpc, per};
    rc = make_tensor_map(&maps.q, a.q, 3, dims, strides, box, what);
  }
  const int box[2] = {64, p.box_rows};
  {
    const int64_t dims[2] = {static_cast<int64_t>(a.G) * a.d1, a.n_rows};
    if (rc == B2TTS_OK) rc = make_tensor_map(&maps.k, a.k, 2, dims, &a.k_row, box, what);
  }
  if (a.d1 < a.d) {
    const int64_t dims[2] = {a.d - a.d1, a.n_rows};
    if (rc == B2TTS_OK) rc = make_tensor_map(&maps.k2, a.k2, 2, dims, &a.k2_row, box, what);
  }
  {
    const int64_t dims[2] = {static_cast<int64_t>(a.Gv) * a.dv, a.n_rows};
    if (rc == B2TTS_OK) rc = make_tensor_map(&maps.v, a.v, 2, dims, &a.v_row, box, what);
  }
  if (rc != B2TTS_OK) return rc;
  const int ns = a.d / 64;
  if (a.r1 != nullptr) return ns == 1 ? go_portion<1, 1, PO_SIGMOID>(what, a, p, maps, grid, st) : go_portion<2, 2, PO_SIGMOID>(what, a, p, maps, grid, st);
  if (a.round_weights && ns == 2 && a.dv == 128) return go_portion<2, 2, PO_ROUNDED>(what, a, p, maps, grid, st);
#define PO_GO(NS, NV) return go_portion<NS, NV, PO_PAIRS>(what, a, p, maps, grid, st)
  if (a.dv == 64) {
    if (ns == 1) PO_GO(1, 1);
    if (ns == 2) PO_GO(2, 1);
    PO_GO(3, 1);
  }
  if (ns == 1) PO_GO(1, 2);
  if (ns == 2) PO_GO(2, 2);
  PO_GO(3, 2);
#undef PO_GO
}

}  // namespace row
}  // namespace b2

extern "C" int b2tts_latent_portions_attn(const void* q, int64_t q_tok, int64_t q_head, const void* k, int64_t k_row, const void* kr,
                                          int64_t kr_row, const void* v, int64_t v_row, int64_t n_rows, const int32_t* key_start, void* out,
                                          const float* sink, const void* gate, int64_t ldg, int gate_el, const int32_t* seq_start,
                                          const int32_t* seq_pos0, const int32_t* seq_len, int n_tokens, int n_seqs, int max_new, int heads,
                                          int dim, int rot_dim, int vdim, int window, float scale, void* stream) {
  using namespace b2;
  using namespace b2::row;
  B2_REQUIRE(n_tokens >= 0 && n_seqs >= 0 && max_new >= 0 && heads > 0 && dim > 0 && rot_dim >= 0 && vdim > 0 && window >= 0, B2TTS_EINVAL,
             "latent_portions_attn: bad sizes");
  B2_REQUIRE(heads <= 65535 && n_seqs <= 65535, B2TTS_EUNSUPPORTED, "latent_portions_attn: %d heads, %d sequences", heads, n_seqs);
  if (n_tokens == 0 || n_seqs == 0 || max_new <= 1) return B2TTS_OK;
  B2_REQUIRE(q && k && v && key_start && out && seq_start && seq_pos0 && seq_len && (rot_dim == 0 || kr), B2TTS_EINVAL,
             "latent_portions_attn: null pointer");
  using B = __nv_bfloat16;
  PortionArgs p{};
  p.q = static_cast<const B*>(q); p.q_tok = q_tok; p.q_head = q_head; p.n_tokens = n_tokens;
  p.k = static_cast<const B*>(k); p.k_row = k_row; p.d1 = dim;
  p.k2 = rot_dim > 0 ? static_cast<const B*>(kr) : nullptr; p.k2_row = rot_dim > 0 ? kr_row : 0;
  p.v = static_cast<const B*>(v); p.v_row = v_row;
  p.n_rows = n_rows;
  p.key_start = key_start; p.page = 1;
  p.seq_start = seq_start; p.seq_pos0 = seq_pos0; p.seq_len = seq_len;
  p.sink = sink; p.gate = static_cast<const B*>(gate); p.ldg = ldg; p.gate_el = gate_el;
  p.out = out;
  p.H = heads; p.G = heads; p.Gv = heads; p.d = dim + rot_dim; p.dv = vdim;
  p.mask = window; p.scale = scale;
  p.n_seqs = n_seqs; p.max_new = max_new;
  B2_REQUIRE(portion_attn_applies(p), B2TTS_EUNSUPPORTED, "latent_portions_attn: dim=%d rot_dim=%d vdim=%d or a row alignment", dim, rot_dim, vdim);
  return launch_portion_attn("latent_portions_attn", p, static_cast<cudaStream_t>(stream));
}

extern "C" int b2tts_portion_attn_timeouts(void) { return b2::wait_count(b2::WAITS_PORTIONS); }
extern "C" unsigned long long b2tts_portion_attn_launches(void) { return __atomic_load_n(&b2::row::g_portion_launches, __ATOMIC_RELAXED); }
extern "C" int b2tts_portion_attn_lose_wait(void* stream) {
  using namespace b2;
  int* word = wait_word(WAITS_PORTIONS);
  B2_REQUIRE(word != nullptr, B2TTS_ECUDA, "portion_attn_lose_wait: no host memory");
  row::portion_lost_wait_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(word);
  B2_CHECK_LAUNCH("portion_attn_lose_wait");
  return B2TTS_OK;
}
