// Prefill multi-LoRA in one launch (bf16, tcgen05): a cluster takes a block of rows and a range of the columns, shrinks the rows (for
// the slices in its range) with K split over its CTAs, and takes its output tiles in turn.
//
//   ADD    : y[rows, :] += delta (reduce-add), or y = delta
//   LINEAR : y[rows, :]  = x . W^T (+ bias) + delta
//
// What bounds the pair it replaces (sgmv_shrink_kernel, then tc_tile_kernel) is the way between its launches: both fill an SM's
// shared memory, so the second one's set-up, its wait for the first and the trip of the intermediate through the L2 are all
// serial with the K loop: 9 to 13 us a shrink of 1000 rows whose loads take 2. Here
//   * one set-up (barriers, TMEM, table of the slots) and one wait for the launch ahead;
//   * partial sums go straight from tensor memory to the CTA that owns their columns, which sends the 16-bit values straight into
//     the MMA operand tile of every CTA (st.async both times): no scratch, no barrier of the cluster between the halves;
//   * the tiles' B operands are on their way before that exchange is over, and y's rows are on their way to the L2;
//   * eight epilogue warps in two sets, each with two output buffers, and few TMA instructions: 1.35 us a tile of 128 x 256 (2.3).
// us per projection (qkv, o, gate_up, down), the pair / this kernel: 8000 rows of 14 prompts, 2048-wide, rank 64: 40 / 38, 32 / 23, 92 / 88,
// 49 / 39; 1000 rows of them 18.7 / 16.8, 14.5 / 10.4, 22 / 17.5, 17 / 12.9. What is left of gate_up's 88 (HBM time 66): a kernel that only
// reads, adds to and writes these rows takes 73 to 80, and the blocks that hold a request boundary end 8 us after the others. Of the 9.9
// of o: 1.4 from the end of the launch before to its first CTA's wait, 1.3 more to the last CTA's, K loop 2.4, exchange 2.5, tile and
// store 2.
// Rows of a block may use different slots: the MMA of the rows of one slot updates these rows only (its lane mask), so
// the operand needs no masked copy per slot. Rows without adapter: -0.0 in ADD launches (x + (-0.0) == x bit for bit), the base
// result in LINEAR ones.
#pragma once

#include "gemm_tc.cuh"

namespace b200lora {

constexpr int kPcThreads = 320;   // warp 0 TMA, warp 1 MMA + TMEM owner, warps 2-9 epilogue
constexpr int kPcEpi = 256;
constexpr int kPcShrinkStages = 12;
constexpr int kPcTileStages = 4;   // ADD
constexpr int kPcMaxTileStages = 8;
constexpr int kPcSmem = 224 * 1024;
constexpr int kPcBox = 64;        // rows of a W or lora_B box

struct PcArgs {
  __nv_bfloat16* y; int64_t y_ld;
  const __nv_bfloat16* bias;                // LINEAR, may be null
  int T, in_dim, n_total, S, r, n;
  int out[B200_LORA_MAX_SLICES], col[B200_LORA_MAX_SLICES];
  const int32_t* token_to_slot;
  const float* scale_per_slot; float scaling;
  int groups, group_cols;                   // clusters of a block of rows, each with a range of the columns (a multiple of 64)
  int cta_cols, tile_cols;                  // columns of y per CTA and per tile (multiples of 64, a tile at most 256)
  int overwrite;                            // ADD: store the delta (-0.0 in rows without adapter) instead of adding it
  int bm, ck;                               // rows of a block (a multiple of 8, 64 to 128), CTAs of a cluster
  int gmax;                                 // lots (slots of a block) whose K loops share one pass over x
  int stages, stage_bytes;                  // ring of the tiles: lora_B tiles (LINEAR: or x and W tiles)
  int out_bufs, off_out, off_tmp;           // output buffers of each epilogue set; byte offsets
  int part_cols, off_part;                  // columns of partial sums exchanged at a time, where they arrive
};
struct PcMaps {
  CUtensorMap x;                            // [T, in]           box bm x 64
  CUtensorMap w;                            // [n_total, in]     box 64 x 64 (LINEAR)
  CUtensorMap y;                            // [T, n_total]      box bm x 64
  CUtensorMap a[B200_LORA_MAX_SLICES];      // [S*r, in]         box r x 64
  CUtensorMap b[B200_LORA_MAX_SLICES];      // [S*out_s, r]      box 64 x r
};

// 16-byte piece c of row `row` inside an operand tile with rows of `row_bytes` (the TMA swizzle of that span)
__device__ __forceinline__ uint32_t swizzled_piece(int row, int c, int row_bytes) {
  const int x = row_bytes == 128 ? (row & 7) : (row_bytes == 64 ? (row >> 1) & 3 : (row >> 2) & 1);
  return (uint32_t)(row * row_bytes + ((c ^ x) << 4));
}

// one arrival, when the MMAs issued so far are complete, at the barrier of this offset in each of the cluster's CTAs in `ctas`
__device__ __forceinline__ void umma_commit_cluster_elected(uint32_t bar, uint16_t ctas, uint32_t leader) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %2;\n\t}"
      ::"r"(bar), "r"(leader), "h"(ctas)
      : "memory");
}

template <bool kLinear>
__global__ void __launch_bounds__(kPcThreads, 1)
prefill_cluster_kernel(const __grid_constant__ PcMaps maps, const __grid_constant__ PcArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ int16_t s_slot[kSgmvBM], lot_slot[kSgmvBM];
  __shared__ uint8_t row_lot[kSgmvBM];  // the lot of a row (255: no adapter)
  __shared__ int nlots_s;
  __shared__ __align__(8) uint64_t bar_words[2 * kPcShrinkStages + 2 * kPcMaxTileStages + 9];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_flag;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int CK = a.ck, ck = CK > 1 ? (int)cluster_ctarank() : 0, blk = (int)blockIdx.x / (CK * a.groups);
  // This cluster's columns, and the slices that they touch: n of them from s0 on
  const int g_lo = ((int)blockIdx.x / CK - blk * a.groups) * a.group_cols, g_hi = min(g_lo + a.group_cols, a.n_total);
  int s0 = 0, n = a.n;
  if (a.groups > 1) {  // (the slices lie one behind the other)
    while (a.col[s0] + a.out[s0] <= g_lo) ++s0;
    n = 1;
    while (s0 + n < a.n && a.col[s0 + n] < g_hi) ++n;
  }
  const int r = a.r, width = n * r, row_bytes = r * 2, bm = a.bm, row0 = blk * bm;
  griddep_launch_dependents();
  const uint32_t smem_base = smem_u32(smem);
  if ((smem_base & 1023u) != 0) {  // (the swizzled tiles need it; the same in every CTA)
    if (tid == 0) atomicOr(&g_b200_status, kStatusBadSmemBase);
    return;
  }
  const uint32_t bar0 = smem_u32(bar_words);
  // ring of the shrink (ADD launches), ring of the tiles
  auto s_full = [&](int s) { return bar0 + 8u * (uint32_t)s; };
  auto s_empty = [&](int s) { return bar0 + 8u * (uint32_t)(kPcShrinkStages + s); };
  auto t_full = [&](int s) { return bar0 + 8u * (uint32_t)(2 * kPcShrinkStages + s); };
  auto t_empty = [&](int s) { return bar0 + 8u * (uint32_t)(2 * kPcShrinkStages + kPcMaxTileStages + s); };
  const uint32_t bar1 = bar0 + 8u * (2 * kPcShrinkStages + 2 * kPcMaxTileStages);
  auto acc_full = [&](int b) { return bar1 + 8u * (uint32_t)b; };
  auto acc_empty = [&](int b) { return bar1 + 16u + 8u * (uint32_t)b; };
  const uint32_t s_acc_full = bar1 + 32u, s_acc_empty = bar1 + 40u;
  const uint32_t part_ready = bar1 + 48u;                          // every CTA of the cluster has room for partial sums
  const uint32_t part_full = bar1 + 56u;                           // the partial sums of this CTA's columns have arrived
  const uint32_t tmp_full = bar1 + 64u;                            // every CTA's share of the intermediate has arrived

  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_s), 512u);
    tc_fence_before_sync();
  }
  if (warp == 0 && elect_one()) {
    tma_prefetch_desc(&maps.x); tma_prefetch_desc(&maps.y);
    if (kLinear) tma_prefetch_desc(&maps.w);
    for (int s = s0; s < s0 + n; ++s) { tma_prefetch_desc(&maps.a[s]); tma_prefetch_desc(&maps.b[s]); }
  }
  if (warp == 2) {
    // ---- lots: the block's rows of one slot each, wherever they lie, in the order of their first rows. (By runs of equal slot, every row
    // of a decode batch over few adapters, which the host cannot tell from whole prompts, was a run, and every one to four runs a pass
    // over x: an add of 333 rows over 8 adapters, 4096-wide, rank 64, took 352 us a layer, by lots 86. One warp finds them by itself: a
    // table of runs that four warps made between barriers kept a launch of 500 to 6000 rows 0.2 to 0.7 us, fused linears 0.1 to 0.5.)
    int slot[4], lot[4], n_lots = 0;  // of rows lane, 32 + lane, ...
    unsigned left[4];                 // rows that have none yet
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const int i = 32 * w + lane;
      slot[w] = i < bm && row0 + i < a.T ? a.token_to_slot[row0 + i] : -1;
      (void)B200_IN_BOUNDS(slot[w] >= -1 && slot[w] < a.S);  // ids outside [-1, S) are treated as "no adapter"; the checked build reports them
      if (slot[w] >= a.S || slot[w] < -1) slot[w] = -1;
      lot[w] = 255;
    }
#pragma unroll
    for (int w = 0; w < 4; ++w) left[w] = __ballot_sync(0xffffffffu, slot[w] >= 0);
    while ((left[0] | left[1] | left[2] | left[3]) != 0) {
      const int w = left[0] != 0 ? 0 : left[1] != 0 ? 1 : left[2] != 0 ? 2 : 3;
      const unsigned rows = w == 0 ? left[0] : w == 1 ? left[1] : w == 2 ? left[2] : left[3];
      const int v = __shfl_sync(0xffffffffu, w == 0 ? slot[0] : w == 1 ? slot[1] : w == 2 ? slot[2] : slot[3], __ffs(rows) - 1);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (slot[q] == v) lot[q] = n_lots;
        left[q] &= ~__ballot_sync(0xffffffffu, slot[q] == v);
      }
      if (lane == 0) lot_slot[n_lots] = (int16_t)v;
      ++n_lots;
    }
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      s_slot[32 * w + lane] = (int16_t)slot[w];
      row_lot[32 * w + lane] = (uint8_t)lot[w];
    }
    if (lane == 0) nlots_s = n_lots;
  }
  if (warp == 3 && elect_one()) {
    for (int s = 0; s < kPcShrinkStages; ++s) { mbar_init(s_full(s), 1); mbar_init(s_empty(s), 1); }
    for (int s = 0; s < kPcMaxTileStages; ++s) { mbar_init(t_full(s), 1); mbar_init(t_empty(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), kPcEpi / 32); }
    mbar_init(s_acc_full, 1);
    mbar_init(s_acc_empty, kPcEpi / 32);
    mbar_init(part_ready, (uint32_t)CK);
    mbar_init(part_full, 1);
    mbar_init(tmp_full, 1);
    abort_flag = 0;
    mbar_fence_init();
    mbar_arrive_expect_tx(tmp_full, (uint32_t)(bm * width * 2));
  }
  __syncthreads();
  tc_fence_after_sync();
  if (CK > 1) { cluster_arrive(); cluster_wait(); }  // the barriers of every CTA of the cluster are initialised
  // Everything above may overlap the previous launch of the stream; x and y are final from here on. (Warp 0 waits ahead of its first load.)
  if (warp != 0) griddep_wait();

  const uint32_t tmem_base = tmem_base_s;
  const int nlots = nlots_s;
  // This CTA's columns of y and its tiles of up to 256 of them: a range, or, in ADD launches, tiles dealt to the CTAs in turn, so that a
  // cluster updates neighbouring pieces of the same rows (8172 rows, 2048-wide, rank 64, a layer 192.1 -> 190.7 us). Not an odd number
  // of tiles to two CTAs, of which one would have more columns than by range (1024 -> 1280, 4300 to 8000 rows, in turn / by range: rank
  // 16 13.1 / 12.6 us, rank 64 17.7 / 17.3). Ten tiles to four CTAs stay dealt (2048 -> 2560, rank 64, 3300 rows 20.1 / 20.7). An ADD
  // launch has nothing to add to a block without any adapter row.
  const int c_begin = min(g_lo + ck * a.cta_cols, g_hi), c_end = min(c_begin + a.cta_cols, g_hi);
  const int all_tiles = (g_hi - g_lo + a.tile_cols - 1) / a.tile_cols;
  const bool in_turn = !kLinear && (CK != 2 || all_tiles % 2 == 0);
  const int my_tiles = !kLinear && nlots == 0 && !a.overwrite ? 0 : in_turn ? (all_tiles - ck + CK - 1) / CK : (c_end - c_begin + a.tile_cols - 1) / a.tile_cols;
  const int t_lo = in_turn ? g_lo + ck * a.tile_cols : c_begin, t_hi = in_turn ? g_hi : c_end, t_step = in_turn ? CK * a.tile_cols : a.tile_cols;
  auto tile_lo = [&](int i) { return t_lo + i * t_step; };
  auto tile_hi = [&](int i) { return min(t_lo + i * t_step + a.tile_cols, t_hi); };
  const uint32_t tmp_base = smem_base + (uint32_t)a.off_tmp, tmp_tile = (uint32_t)(kSgmvBM * row_bytes);
  // ---- the shrink's passes over x: up to G lots share one
  const int nk_all = a.in_dim / kSgmvBK, nk_per = (nk_all + CK - 1) / CK;
  const int kc0 = min(ck * nk_per, nk_all), nk = min(nk_per, nk_all - kc0);  // this CTA's K steps (at least one: see the launch)
  const int G = min(a.gmax, max(nlots, 1)), npass = (nlots + G - 1) / G;
  const uint32_t x_tile = (uint32_t)bm * kSgmvBK * 2, a_tile = (uint32_t)r * kSgmvBK * 2;
  const uint32_t x_span = kSgmvBM * kSgmvBK * 2;  // (the MMA reads 128 rows; those beyond bm give rows that nobody reads)
  const uint32_t s_stage = kLinear ? (uint32_t)a.stage_bytes : x_span + (uint32_t)(G * n) * a_tile;
  // ADD: the partial sums have a place of their own where that leaves the K loop enough stages
  const bool apart = kLinear || a.off_part / (int)s_stage >= min(nk_per, 4);
  // ADD: the MMAs of a pass read its K loop's ring and begin when this CTA has read the sums of the pass before, so their completion tells
  // the cluster that this CTA has room for sums. (Told by the epilogue, whose arrival has to release those reads: qkv of 4300 to 8000 rows,
  // rank 64, 1024-wide 18.5 / 18.1 us, 2048-wide 32.1 / 31.4.) Not where nobody would wait for it: a CTA may leave before its peers arrive.
  const bool told = !kLinear && CK > 1 && (!apart || npass > 1);
  const int s_stages = kLinear ? a.stages : min(kPcShrinkStages, (apart ? a.off_part : a.off_tmp) / (int)s_stage);
  const uint32_t s_tmem = tmem_base + (kLinear ? kSgmvBN : 0);  // (LINEAR: the first tile's sums lie in front)
  const uint32_t part_base = smem_base + (uint32_t)a.off_part;
  const int nk_base = kLinear ? nk_all : 0;

  // slice s inside tile i: its columns [lo, hi) of y
  auto part_of = [&](int s, int i, int& lo, int& hi) {
    lo = max(a.col[s], tile_lo(i));
    hi = min(a.col[s] + a.out[s], tile_hi(i));
    return lo < hi;
  };

  if (warp == 0) {
    // =========================== TMA
    const uint32_t leader = elect_one();
    int st = 0, round = 0;
    if (npass == 0) griddep_wait();
    for (int pi = 0; pi < npass; ++pi) {
      // (ADD: the partial sums of a pass lie where the ring is)
      if (!kLinear && pi > 0) mbar_wait_bounded(s_acc_empty, (uint32_t)((pi - 1) & 1), &abort_flag);
      const int u0 = pi * G, g = min(G, nlots - u0);
      int row[4];  // first lora_A row of each lot of the pass (G <= 4)
#pragma unroll
      for (int ui = 0; ui < 4; ++ui) row[ui] = uniform(ui < g ? lot_slot[u0 + ui] * r : 0);
      // (lora_A of the first stages asked for ahead of this wait puts x behind it: us a launch, with / without, means over 1072 adds of 64 to
      // 8000 rows: up to 450 rows 5.99 / 5.99, to 800 8.65 / 8.50, to 2112 11.45 / 11.17, to 4224 18.3 / 17.9, to 4736 24.6 / 23.9, to 8000
      // 29.0 / 28.5; slabs that are not in the L2 the same way; fused linears 0 to 1 %.)
      if (pi == 0) griddep_wait();
      for (int kc = 0; kc < nk; ++kc) {
        const uint32_t full = kLinear ? t_full(st) : s_full(st), empty = kLinear ? t_empty(st) : s_empty(st);
        if (round > 0) mbar_wait_bounded(empty, (uint32_t)((round & 1) ^ 1), &abort_flag);
        if (leader) {
          uint32_t dst = smem_base + (uint32_t)st * s_stage;
          mbar_arrive_expect_tx(full, x_tile + (uint32_t)(g * n) * a_tile);
          tma_load_2d(dst, &maps.x, (kc0 + kc) * kSgmvBK, row0, full);
          dst += x_span;
#pragma unroll
          for (int ui = 0; ui < 4; ++ui)
            if (ui < g)
              for (int s = 0; s < n; ++s, dst += a_tile) tma_load_2d(dst, &maps.a[s0 + s], (kc0 + kc) * kSgmvBK, row[ui], full);
        }
        __syncwarp();
        if (++st == s_stages) { st = 0; ++round; }
      }
    }
    if (!kLinear) {
      st = round = 0;
      if (npass > 0) mbar_wait_bounded(s_acc_full, (uint32_t)((npass - 1) & 1), &abort_flag);  // the ring changes its use
    }
    bool exchanged = kLinear;
    const uint64_t w_policy = l2_policy_evict_last();
    // The reduce-add reads y at the L2: the rows of a tile are asked for together with its lora_B tiles, as many tiles ahead as the
    // ring has stages (one tile further ahead 2 to 8 % slower), the first ones while the sums of the shrink are exchanged. By box:
    // 128 bulk prefetches of a row piece each kept the TMA unit busy for 2.3 us a tile.
    auto ask_y = [&](int i) {
      if (kLinear || a.overwrite || !leader || i >= my_tiles) return;
      for (int c = tile_lo(i); c < tile_hi(i); c += kGemmOutChunk) tma_prefetch_2d(&maps.y, c, row0);
    };
    for (int i = 0; i < my_tiles; ++i) {
      ask_y(i);
      const int w_boxes = (tile_hi(i) - tile_lo(i) + kPcBox - 1) / kPcBox;
      for (int kc = 0; kc < nk_base; ++kc) {
        if (round > 0) mbar_wait_bounded(t_empty(st), (uint32_t)((round & 1) ^ 1), &abort_flag);
        if (leader) {
          const uint32_t base = smem_base + (uint32_t)(st * a.stage_bytes), full = t_full(st);
          mbar_arrive_expect_tx(full, x_tile + (uint32_t)(w_boxes * kPcBox * kSgmvBK * 2));
          tma_load_2d(base, &maps.x, kc * kSgmvBK, row0, full);
          for (int q = 0; q < w_boxes; ++q)
            tma_load_2d_hint(base + x_span + (uint32_t)(q * kPcBox * kSgmvBK * 2), &maps.w, kc * kSgmvBK, tile_lo(i) + q * kPcBox, full, w_policy);
        }
        __syncwarp();
        if (++st == a.stages) { st = 0; ++round; }
      }
      for (int u = 0; u < nlots; ++u) {
        const int slot = uniform(lot_slot[u]);
        for (int s = s0; s < s0 + n; ++s) {
          int lo, hi;
          if (!part_of(s, i, lo, hi)) continue;
          if (round > 0) mbar_wait_bounded(t_empty(st), (uint32_t)((round & 1) ^ 1), &abort_flag);
          const uint32_t base = smem_base + (uint32_t)(st * a.stage_bytes), full = t_full(st);
          // (ADD: a stage that lies where the partial sums are waits until every CTA has read them, that is, has sent its share)
          if (!exchanged && base + (uint32_t)a.stage_bytes > part_base) {
            mbar_wait_bounded_acquire_cluster(tmp_full, 0u, &abort_flag);
            fence_proxy_async_smem();
            exchanged = true;
          }
          if (leader) {
            const int boxes = (hi - lo + kPcBox - 1) / kPcBox;
            mbar_arrive_expect_tx(full, (uint32_t)(boxes * kPcBox * row_bytes));
            for (int q = 0; q < boxes; ++q)
              tma_load_2d(base + (uint32_t)(q * kPcBox * row_bytes), &maps.b[s], 0, slot * a.out[s] + (lo - a.col[s]) + q * kPcBox, full);
          }
          __syncwarp();
          if (++st == a.stages) { st = 0; ++round; }
        }
      }
    }
  } else if (warp == 1) {
    // =========================== MMA
    const uint32_t leader = elect_one();
    const uint64_t desc_x = umma_smem_desc(smem_base, 128), desc_t = umma_smem_desc(smem_base, row_bytes);
    const uint32_t hi_x = (uint32_t)(desc_x >> 32), hi_t = (uint32_t)(desc_t >> 32), lo0 = (uint32_t)desc_x;
    const uint32_t idesc_s = umma_idesc_bf16(kSgmvBM, width);
    int st = 0, round = 0;
    for (int pi = 0; pi < npass; ++pi) {
      const int jobs = uniform(min(G, nlots - pi * G));
      if (pi > 0) mbar_wait_bounded(s_acc_empty, (uint32_t)((pi - 1) & 1), &abort_flag);
      tc_fence_after_sync();
      for (int kc = 0; kc < nk; ++kc) {
        mbar_wait_bounded(kLinear ? t_full(st) : s_full(st), (uint32_t)(round & 1), &abort_flag);
        tc_fence_after_sync();
        const uint32_t xl = lo0 + ((uint32_t)st * s_stage >> 4);
        uint32_t al = xl + (x_span >> 4), d = s_tmem;
        for (int q = 0; q < jobs; ++q, al += (uint32_t)n * a_tile >> 4, d += (uint32_t)width) {  // lots of the pass
#pragma unroll
          for (int k4 = 0; k4 < kSgmvBK / 16; ++k4) umma_elected(d, xl + 2u * k4, al + 2u * k4, hi_x, idesc_s, (kc > 0 || k4 > 0) ? 1u : 0u, leader);
        }
        umma_commit_elected(kLinear ? t_empty(st) : s_empty(st), leader);  // stage reusable once these MMAs have read it
        if (++st == s_stages) { st = 0; ++round; }
      }
      umma_commit_elected(s_acc_full, leader);
      if (told) umma_commit_cluster_elected(part_ready, (uint16_t)((1 << CK) - 1), leader);
    }
    if (!kLinear) st = round = 0;
    bool have_tmp = false;
    int my_lot[4];  // of rows lane, 32 + lane, ...
#pragma unroll
    for (int w = 0; w < 4; ++w) my_lot[w] = row_lot[32 * w + lane];
    for (int job = 0; job < my_tiles; ++job) {
      const int buf = job & 1, c_lo = tile_lo(job);
      const uint32_t idesc_w = umma_idesc_bf16(kSgmvBM, (tile_hi(job) - c_lo + 15) & ~15);
      const uint32_t d_tmem = tmem_base + (uint32_t)(buf * kSgmvBN);
      // (the shrink's sums: in LINEAR launches where the second tile's will be, in ADD ones read before the intermediate was sent)
      if (kLinear && job == 1 && npass > 0) mbar_wait_bounded(s_acc_empty, (uint32_t)((npass - 1) & 1), &abort_flag);
      if (job >= 2) mbar_wait_bounded(acc_empty(buf), (uint32_t)(((job >> 1) - 1) & 1), &abort_flag);
      tc_fence_after_sync();
      for (int kc = 0; kc < nk_base; ++kc) {
        mbar_wait_bounded(t_full(st), (uint32_t)(round & 1), &abort_flag);
        tc_fence_after_sync();
        const uint32_t xl = lo0 + ((uint32_t)(st * a.stage_bytes) >> 4), wl = xl + (x_span >> 4);
#pragma unroll
        for (int k4 = 0; k4 < kSgmvBK / 16; ++k4) umma_elected(d_tmem, xl + 2u * k4, wl + 2u * k4, hi_x, idesc_w, (kc > 0 || k4 > 0) ? 1u : 0u, leader);
        umma_commit_elected(t_empty(st), leader);
        if (++st == a.stages) { st = 0; ++round; }
      }
      for (int u = 0; u < nlots; ++u) {
        uint32_t off[4];  // lanes that are not of the lot
#pragma unroll
        for (int w = 0; w < 4; ++w) off[w] = __ballot_sync(0xffffffffu, my_lot[w] != u);
        for (int s = s0; s < s0 + n; ++s) {
          int lo, hi;
          if (!part_of(s, job, lo, hi)) continue;
          if (!have_tmp) {
            mbar_wait_bounded_acquire_cluster(tmp_full, 0u, &abort_flag);
            fence_proxy_async_smem();  // (it came by plain stores)
            if (!kLinear) mbar_wait_bounded(s_acc_empty, (uint32_t)((npass - 1) & 1), &abort_flag);  // this CTA's own sums have been read
            have_tmp = true;
            tc_fence_after_sync();
          }
          mbar_wait_bounded(t_full(st), (uint32_t)(round & 1), &abort_flag);
          tc_fence_after_sync();
          const uint32_t bl = lo0 + ((uint32_t)(st * a.stage_bytes) >> 4), tl = lo0 + (((uint32_t)a.off_tmp + (uint32_t)(s - s0) * tmp_tile) >> 4);
          const uint32_t idesc = umma_idesc_bf16(kSgmvBM, (hi - lo + 15) & ~15);
#pragma unroll
          for (int k4 = 0; k4 < 4; ++k4)
            if (16 * k4 < r)
              umma_rows_elected(d_tmem + (uint32_t)(lo - c_lo), tl + 2u * k4, bl + 2u * k4, hi_t, idesc, kLinear || k4 > 0 ? 1u : 0u, leader, off);
          umma_commit_elected(t_empty(st), leader);
          if (++st == a.stages) { st = 0; ++round; }
        }
      }
      umma_commit_elected(acc_full(buf), leader);
    }
  } else {
    // =========================== epilogue: eight warps; a warp may only touch its own quarter of the 128 TMEM lanes
    const int quarter = warp & 3, set = (warp - 2) >> 2, etid = tid - 64, row_in_blk = quarter * 32 + lane;
    // ---- the shrink's sums: every CTA sends its partial sums to the CTA that owns their columns (eight at a time are a piece, the
    // pieces are dealt in ranges), which adds them up, rounds and sends the values to every CTA's operand tile. Everything travels by
    // st.async: with plain remote stores and an arrival that releases them a layer of 300 to 5000 rows takes 4 to 10 % longer, the
    // release alone 1 us. (Before: written to shared memory, read by the owners across the cluster behind a barrier.)
    int exchange = 0;
    const int my_slot = s_slot[row_in_blk], my_lot = row_lot[row_in_blk];
    const float my_scale = my_slot < 0 ? 0.f : a.scaling * (a.scale_per_slot != nullptr ? a.scale_per_slot[my_slot] : 1.0f);
    const uint32_t row_off = (uint32_t)row_in_blk * 16u, quad = (uint32_t)bm * 16u;  // [sender][piece][half of it][row] of 16 bytes
    for (int pi = 0; pi < npass; ++pi) {
      const int u0 = pi * G, g = min(G, nlots - u0);
      int rows = 0;  // of this pass
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const int of = row_lot[32 * w + lane];
        rows += __popc(__ballot_sync(0xffffffffu, of >= u0 && of < u0 + g));
      }
      const bool live = my_lot >= u0 && my_lot < u0 + g;
      const bool zero = my_slot < 0 && pi == 0 && row_in_blk < bm;  // rows without adapter
      mbar_wait_bounded(s_acc_full, (uint32_t)(pi & 1), &abort_flag);
      tc_fence_after_sync();
      for (int c0 = 0; c0 < width; c0 += a.part_cols, ++exchange) {
        const int cols = min(a.part_cols, width - c0), pieces = cols >> 3, per = (pieces + CK - 1) / CK;
        const int mine = min(max(pieces - ck * per, 0), per);
        // (Not before every thread has seen the exchange before complete: one of no bytes is complete at once, and a wait that is two
        // phases behind takes the parity for that of the phase to come.)
        if (exchange > 0) named_bar_sync(2, kPcEpi);
        if (etid == 0) mbar_arrive_expect_tx(part_full, (uint32_t)((CK - 1) * rows * mine * 32));
        // Room for them in every CTA: the K loop whose ring lies there is over, the sums of the exchange before have been read.
        // LINEAR: nothing lies there ahead of the first one; the arrival releases, since peers may write only behind these reads.
        if (kLinear && exchange > 0) {
          if (etid < CK) mbar_arrive_remote_release(mapa_shared(part_ready, (uint32_t)etid));
          mbar_wait_bounded_acquire_cluster(part_ready, (uint32_t)((exchange - 1) & 1), &abort_flag);
        }
        const bool ahead = !apart || pi > 0;  // of the sends
        if (told && ahead) mbar_wait_bounded_acquire_cluster(part_ready, (uint32_t)(pi & 1), &abort_flag);
        // (A TMEM load is a warp-wide operation on one column range: a warp with rows of two lots reads both lots' columns.)
        for (int ui = 0; ui < g; ++ui) {
          const bool here = my_lot == u0 + ui;
          if (!__any_sync(0xffffffffu, here)) continue;
          for (int c = 16 * set; c < cols; c += 32) {
            uint32_t v[16];
            tmem_ld_32x16(s_tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ui * width + c0 + c), v);
            tmem_ld_wait();
            if (here) {
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int p = (c >> 3) + h, owner = p / per;
                const uint32_t at = part_base + (uint32_t)((ck * per + p - owner * per) * 2) * quad + row_off;
                const uint4 v0 = make_uint4(v[8 * h], v[8 * h + 1], v[8 * h + 2], v[8 * h + 3]);
                const uint4 v1 = make_uint4(v[8 * h + 4], v[8 * h + 5], v[8 * h + 6], v[8 * h + 7]);
                if (owner == ck) {  // (this thread reads them again)
                  sts128(at, v0);
                  sts128(at + quad, v1);
                } else {
                  const uint32_t dst = mapa_shared(at, (uint32_t)owner), bar = mapa_shared(part_full, (uint32_t)owner);
                  st_async_b32x4(dst, v0, bar);
                  st_async_b32x4(dst + quad, v1, bar);
                }
              }
            }
          }
        }
        tc_fence_before_sync();
        if (kLinear && c0 + cols == width) {  // the second tile's sums may go where these were
          __syncwarp();
          if (lane == 0) mbar_arrive(s_acc_empty);
        }
        mbar_wait_bounded_acquire_cluster(part_full, (uint32_t)(exchange & 1), &abort_flag);
        // (Every phase is waited for, ahead of the arrival that lets this CTA's next pass begin: the next phase may be complete soon after
        // that, and its parity is the one of the phase before.)
        if (told && !ahead) mbar_wait_bounded_acquire_cluster(part_ready, (uint32_t)(pi & 1), &abort_flag);
        auto add_up = [&](auto parts) {
          constexpr int kParts = decltype(parts)::value;
          if (!live && !zero) return;
          for (int lp = 0; lp < mine; ++lp) {
            if ((((ck * per + lp) >> 1) & 1) != set) continue;
            uint4 packed = make_uint4(0, 0, 0, 0);
            if (live) {
              uint4 w[kParts][2];
#pragma unroll
              for (int q = 0; q < kParts; ++q)
#pragma unroll
                for (int h = 0; h < 2; ++h) w[q][h] = lds128(part_base + (uint32_t)((q * per + lp) * 2 + h) * quad + row_off);
              float sum[2][4];
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                sum[h][0] = __uint_as_float(w[0][h].x); sum[h][1] = __uint_as_float(w[0][h].y);
                sum[h][2] = __uint_as_float(w[0][h].z); sum[h][3] = __uint_as_float(w[0][h].w);
#pragma unroll
                for (int q = 1; q < kParts; ++q) {
                  sum[h][0] += __uint_as_float(w[q][h].x); sum[h][1] += __uint_as_float(w[q][h].y);
                  sum[h][2] += __uint_as_float(w[q][h].z); sum[h][3] += __uint_as_float(w[q][h].w);
                }
              }
              packed = make_uint4(pack_bf16x2(sum[0][0] * my_scale, sum[0][1] * my_scale), pack_bf16x2(sum[0][2] * my_scale, sum[0][3] * my_scale),
                                  pack_bf16x2(sum[1][0] * my_scale, sum[1][1] * my_scale), pack_bf16x2(sum[1][2] * my_scale, sum[1][3] * my_scale));
            }
            const int col = c0 + 8 * (ck * per + lp), s = col / r, c = col - s * r;
            const uint32_t dst = tmp_base + (uint32_t)s * tmp_tile + swizzled_piece(row_in_blk, c >> 3, row_bytes);
            for (int q = 0; q < CK; ++q) st_async_b32x4(mapa_shared(dst, (uint32_t)q), packed, mapa_shared(tmp_full, (uint32_t)q));
          }
        };
        if (CK == 8) add_up(std::integral_constant<int, 8>{});
        else if (CK == 4) add_up(std::integral_constant<int, 4>{});
        else if (CK == 2) add_up(std::integral_constant<int, 2>{});
        else add_up(std::integral_constant<int, 1>{});
      }
      if (!kLinear) {
        fence_proxy_async_smem();  // the ring is filled again where the partial sums were
        __syncwarp();
        if (lane == 0) mbar_arrive(s_acc_empty);
      }
    }
    // ---- the tiles: set 0 takes the first and third 64-column chunk of a tile, set 1 the others
    const uint32_t out_bytes = (uint32_t)bm * kGemmOutChunk * 2;
    const uint32_t out_set = smem_base + (uint32_t)a.off_out + (uint32_t)(set * a.out_bufs) * out_bytes;
    const bool issuer = tid == 64 + 128 * set, in_block = quarter * 32 < bm;
    const bool neg_zero_row = !kLinear && s_slot[row_in_blk] < 0;
    int chunk_no = 0;
    // Every CTA has read the partial sums that lie where the output buffers are. (A CTA without tiles waits too: it may not leave
    // while a peer still reads from it or sends to it.)
    if (npass > 0) mbar_wait_bounded_acquire_cluster(tmp_full, 0u, &abort_flag);
    for (int job = 0; job < my_tiles; ++job) {
      const int buf = job & 1, c_lo = tile_lo(job), cols = tile_hi(job) - c_lo;
      mbar_wait_bounded(acc_full(buf), (uint32_t)((job >> 1) & 1), &abort_flag);
      tc_fence_after_sync();
      for (int c = kGemmOutChunk * set; c < cols; c += 2 * kGemmOutChunk, ++chunk_no) {
        const int col0 = c_lo + c;
        const uint32_t obuf = out_set + (uint32_t)(chunk_no % a.out_bufs) * out_bytes;
        if (issuer) {  // the store that last used this buffer must have finished reading it
          if (a.out_bufs == 2) bulk_wait_group_read<1>();
          else bulk_wait_group_read<0>();
        }
        named_bar_sync(3 + (uint32_t)set, 128);
        if (in_block) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t v[32];
            tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * kSgmvBN + c + 32 * h), v);
            tmem_ld_wait();
            if (kLinear && a.bias != nullptr) {
#pragma unroll
              for (int q = 0; q < 32; ++q) {
                const int cc = col0 + 32 * h + q;
                v[q] = __float_as_uint(__uint_as_float(v[q]) + (cc < a.n_total ? __bfloat162float(a.bias[cc]) : 0.f));
              }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint4 o;
              o.x = pack_bf16x2(__uint_as_float(v[8 * q + 0]), __uint_as_float(v[8 * q + 1]));
              o.y = pack_bf16x2(__uint_as_float(v[8 * q + 2]), __uint_as_float(v[8 * q + 3]));
              o.z = pack_bf16x2(__uint_as_float(v[8 * q + 4]), __uint_as_float(v[8 * q + 5]));
              o.w = pack_bf16x2(__uint_as_float(v[8 * q + 6]), __uint_as_float(v[8 * q + 7]));
              if (neg_zero_row) o = make_uint4(0x80008000u, 0x80008000u, 0x80008000u, 0x80008000u);
              if (row_in_blk < bm) sts128(obuf + swizzled_piece(row_in_blk, 4 * h + q, 128), o);
            }
          }
        }
        fence_proxy_async_smem();
        named_bar_sync(3 + (uint32_t)set, 128);
        if (issuer) {
          if (!kLinear && !a.overwrite) tma_reduce_add_2d(&maps.y, obuf, col0, row0);
          else tma_store_2d_hint(&maps.y, obuf, col0, row0, l2_policy_evict_first());
          bulk_commit_group();
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty(buf));
    }
    if (issuer) bulk_wait_group_read<0>();
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 512u);
  if (tid == 0 && abort_flag != 0) atomicOr(&g_b200_status, kStatusWaitGaveUp);
}

// ------------------------------------------------------------------ host side
// Clusters of 1, 2, 4 and 8 CTAs with an SM each that are resident at a time (what cudaOccupancyMaxActiveClusters says: the SMs
// of a cluster lie in one GPC). One cluster more is a second wave.
inline int clusters_resident(int ck) { return ck == 1 ? 148 : (ck == 2 ? 74 : (ck == 4 ? 33 : 15)); }
// Slices that one of the groups of `group_cols` columns touches, at most (a group with more than one holds the first column of one)
inline int prefill_cluster_need(const PcArgs& a, int n, int group_cols) {
  int most = 1;
  for (int k = 1; k < n; ++k) {
    const int lo = a.col[k] / group_cols * group_cols, hi = lo + group_cols;
    int here = 0;
    for (int s = 0; s < n; ++s) here += a.col[s] < hi && a.col[s] + a.out[s] > lo;
    most = std::max(most, here);
  }
  return most;
}

// Lots (the rows of a slot) of a block that share a pass over x (`width` rank rows each). ADD: sums in 512 TMEM columns, two stages of the ring; LINEAR: in
// 256, lora_A tiles where a stage has its W tile.
inline int prefill_cluster_lots(bool linear, int width, int room) {
  int lots = 1;
  for (int g = 2; g <= 4; ++g)
    if (linear ? g * width <= kSgmvBN && g * width * kSgmvBK * 2 <= room : g * width <= 512 && room / (kSgmvBM * kSgmvBK * 2 + g * width * kSgmvBK * 2) >= 2)
      lots = g;
  return lots;
}

// LINEAR: bytes of a stage and stages of its ring (of which at least three and one output buffer of each epilogue set must fit; 0 if not)
inline int prefill_cluster_linear_stages(int tile_cols, int width, int off_tmp, int out_buf, int* stage_bytes) {
  *stage_bytes = kSgmvBM * kSgmvBK * 2 + std::max(tile_cols, width) * kSgmvBK * 2;
  if (width > kSgmvBN || off_tmp - 3 * *stage_bytes < 2 * out_buf) return 0;
  int stages = 3;
  while (stages < kPcMaxTileStages && off_tmp - (stages + 1) * *stage_bytes >= 4 * out_buf) ++stages;
  return stages;
}

// K parts (the CTAs of a cluster), groups of columns and rows of a block: of those splits whose clusters are resident at once, the one
// of the least time in us, which is returned (negative: none fits). `in_groups`: the slices lie one behind the other.
//   ADD: a sum of the K loop at 70 KB a us, the exchange, the output tiles, less than half of the SMs (the launch behind then sets itself
//   up beside this one), passes over x that fewer than four lots can share. A fit to 210 measured points (15 projections, 1024- and
//   2048-wide, rank 16 to 64; 200 to 11000 rows of up to eight prompts, every K split with 1 to 16 groups): it loses 1.0 % to the best
//   split of each, at most 17; one group and the largest K split 7.1; over 465 later points (1000 to 8000 rows, three widths) 0.7. us, that / the split taken: 2048 -> 2 x 6144, rank 64, 300, 700, 2000,
//   4000 rows 22.5 / 13.6, 22.0 / 15.1, 29.5 / 27.9, 51.9 / 47.2; 2048 -> 2560 300 and 700 20.0 / 12.6, 19.4 / 15.4; 1024 -> 1024, rank 32,
//   300 and 2000 7.9 / 7.4, 8.8 / 8.8. (A CTA's tiles, 1.1 us each, were half of the time where a block had one cluster: with groups a
//   block can be 128 rows high and its columns still go to 16 CTAs and more.)
//   LINEAR: set-up, the shrink's steps (more where one or two lots share a pass), the base product's (their latency over the stages of
//   the ring, then the bytes that all CTAs take), the exchange, the tiles: a regression over 3820 measured splits (12 projections as
//   above, 64 to 4500 rows) that meets them within 8 %. Below that the sum does not tell, so the most K parts with one group stay
//   unless another split promises 13 % less.
inline double prefill_cluster_split(bool linear, bool in_groups, int T, int in_dim, int n, int n_total, int r, PcArgs* a) {
  const int nk = in_dim / kSgmvBK;
  // Rows that are too many for clusters of four and fill the chip with 64-row blocks of clusters of two, and a y that is updated at the rate
  // of the HBM: blocks of 128 rows in two groups of columns are slower, although the sum has them equal. us, two groups / one, 24 points
  // of 4300 to 4700 rows 43.4 / 40.6: 1024 -> 8192, rank 32, 35.7 / 32.5, 2048 -> 12288, rank 64, 51.6 / 47.0. (A y of less than half of the L2
  // keeps its groups: 1024 -> 4096, rank 32, 15.0 / 17.3.)
  const bool one_group_only = !linear && ceil_div_i(T, kSgmvBM) > clusters_resident(4) && ceil_div_i(T, 64) <= clusters_resident(2) &&
                              2 * (int64_t)T * n_total > 56 * 1000 * 1000;
  double least = -1.0, one_group = -1.0;
  int one_group_ck = 0, one_group_bm = 0;
  for (int ck = 1; ck <= 8; ck *= 2) {
    const int nk_part = ceil_div_i(nk, ck);
    if (ck > 1 && nk_part * (ck - 1) >= nk) break;  // every K part at least one step
    // columns of a CTA in units of 64: all, then fewer and fewer, in about ten sizes
    int last = 0;
    for (int unit = ceil_div_i(n_total, 64 * ck); unit >= 1; unit = unit > 4 ? (unit + 1) * 3 / 4 : unit - 1) {
      const int groups = unit * ck * 64 >= n_total ? 1 : ceil_div_i(n_total, unit * ck * 64);
      if (groups == last) continue;
      if (groups > clusters_resident(ck) || (groups > 1 && (!in_groups || one_group_only))) break;
      last = groups;
      const int bm = std::max(64, round_up_i(ceil_div_i(T, clusters_resident(ck) / groups), 8)), rows = std::min(bm, kSgmvBM);
      if (bm > kSgmvBM && (ck > 1 || groups > 1)) break;
      const int group_cols = groups > 1 ? round_up_i(ceil_div_i(n_total, groups), 64) : n_total;
      if (group_cols * (groups - 1) >= n_total) continue;
      const int width = (groups > 1 ? prefill_cluster_need(*a, n, group_cols) : n) * r, off_tmp = kPcSmem - width * kSgmvBM * 2;
      const int cols = round_up_i(ceil_div_i(group_cols, ck), 64), tiles = ceil_div_i(cols, kSgmvBN), tile_cols = round_up_i(ceil_div_i(cols, tiles), 64);
      const int ctas = ck * groups * ceil_div_i(T, rows);
      const double exchange = rows * width * 4 / 1024.0;
      double cost;
      if (linear) {
        int stage;
        const int stages = prefill_cluster_linear_stages(tile_cols, width, off_tmp, rows * kGemmOutChunk * 2, &stage);
        if (stages == 0) continue;
        const int lots = prefill_cluster_lots(true, width, std::max(tile_cols, width) * kSgmvBK * 2);
        const double high = (double)rows / kSgmvBM, kb = (rows + tile_cols) * 0.128;
        cost = 3.6 + nk_part * (0.27 + high * (0.06 + (lots == 1 ? 0.44 : lots == 2 ? 0.1 : 0.0))) +
               tiles * nk * (0.042 + 0.87 / stages + kb * (0.0009 + 0.0015 * ctas / 148)) + 0.044 * exchange + tiles * (0.28 + 0.65 * tile_cols / kSgmvBN * high);
      } else {
        cost = nk_part * (rows + width) * (kSgmvBK * 2 / 70e3) + 0.05 * exchange + 0.35 * tiles + 0.1 * cols / kSgmvBN + (ctas > 74 ? 0.3 : 0.0) +
               3.0 * (4 - prefill_cluster_lots(false, width, off_tmp));
      }
      if (groups == 1) { one_group = cost; one_group_ck = ck; one_group_bm = rows; }  // (the most K parts come last)
      if (least < 0.0 || cost < least) {
        least = cost;
        a->ck = ck; a->groups = groups; a->bm = rows; a->group_cols = group_cols;
      }
    }
  }
  if (linear && one_group >= 0.0 && least > 0.87 * one_group) {
    least = one_group;
    a->ck = one_group_ck; a->groups = 1; a->bm = one_group_bm; a->group_cols = n_total;
  }
  return least;
}

// bytes of the partial sums that a CTA gets of `cols` columns
inline int prefill_cluster_part_bytes(const PcArgs& a, int cols) { return a.ck * ceil_div_i(cols / 8, a.ck) * 8 * a.bm * 4; }

// Split, tiles and shared memory (ring of the tiles, output buffers, the intermediate as MMA operand; ADD launches shrink through a
// ring over the first two) of a problem with `n` slices; false: too many rank rows for them. `time`: what the split is expected to take.
inline bool prefill_cluster_plan(const SgmvProblem& b, int n, int n_total, bool linear, PcArgs* a, double* time = nullptr) {
  bool in_groups = true;  // slices that cover the columns one behind the other
  for (int s = 0, k = 0, pos = 0; s < b.st.n; ++s)
    if (b.st.out[s] > 0) {
      in_groups = in_groups && b.st.col[s] == pos;
      pos += b.st.out[s];
      a->out[k] = b.st.out[s]; a->col[k] = b.st.col[s]; ++k;
      if (k == n) in_groups = in_groups && pos == n_total;
    }
  const double cost = prefill_cluster_split(linear, in_groups, b.T, b.in_dim, n, n_total, b.r_max, a);
  if (cost < 0.0) return false;
  if (time != nullptr) *time = cost;
  a->cta_cols = round_up_i(ceil_div_i(a->group_cols, a->ck), 64);
  a->tile_cols = round_up_i(ceil_div_i(a->cta_cols, ceil_div_i(a->cta_cols, kSgmvBN)), 64);
  const int width = (a->groups > 1 ? prefill_cluster_need(*a, n, a->group_cols) : n) * b.r_max, out_buf = a->bm * kGemmOutChunk * 2;
  a->off_tmp = kPcSmem - width * kSgmvBM * 2;
  if (linear) {
    // stages of an x and a W tile (or, ahead of the tiles, of the lora_A tiles of up to gmax lots), then output buffers
    a->stages = prefill_cluster_linear_stages(a->tile_cols, width, a->off_tmp, out_buf, &a->stage_bytes);
    a->gmax = prefill_cluster_lots(true, width, a->stage_bytes - kSgmvBM * kSgmvBK * 2);
    a->out_bufs = std::min(2, (a->off_tmp - a->stages * a->stage_bytes) / (2 * out_buf));
    a->part_cols = width;
    while (prefill_cluster_part_bytes(*a, a->part_cols) > 2 * a->out_bufs * out_buf) a->part_cols -= 16;  // (16 always fit)
  } else {
    a->stages = kPcTileStages;
    a->stage_bytes = a->tile_cols * b.r_max * 2;
    a->out_bufs = 2;
    while (a->stages > 2 && a->off_tmp - a->stages * a->stage_bytes < 2 * a->out_bufs * out_buf) --a->stages;
    a->gmax = prefill_cluster_lots(false, width, a->off_tmp);
    a->part_cols = width;
  }
  a->off_out = a->stages * a->stage_bytes;
  a->off_part = linear ? a->off_out : (a->off_tmp - prefill_cluster_part_bytes(*a, width)) & ~1023;
  return true;
}

// y += delta or y = delta (weight == nullptr), or y = x . W^T (+ bias) + delta, of a problem that sgmv_supported takes and that
// prefill_cluster_plan has planned in `a`.
inline int prefill_cluster_launch(const SgmvProblem& b, PcArgs a, const void* weight, int64_t w_ld, int n_total, const void* bias, bool overwrite, cudaStream_t stream) {
  const bool linear = weight != nullptr;
  PcMaps maps;
  if (b.S > 32767) return fail(B200_LORA_EUNSUPPORTED, "prefill kernel: more than 32767 adapter slots");
  a.y = static_cast<__nv_bfloat16*>(b.y); a.y_ld = b.y_ld; a.bias = static_cast<const __nv_bfloat16*>(bias);
  a.T = b.T; a.in_dim = b.in_dim; a.n_total = n_total; a.S = b.S; a.r = b.r_max;
  a.token_to_slot = b.token_to_slot; a.scale_per_slot = b.scale_per_slot; a.scaling = b.scaling; a.overwrite = overwrite ? 1 : 0;
  for (int s = 0; s < b.st.n; ++s) {
    if (b.st.out[s] == 0) continue;
    if (int rc = make_tmap_2d(&maps.a[a.n], b.st.a[s], (uint64_t)b.S * b.r_max, (uint64_t)b.in_dim, (uint64_t)b.in_dim, (uint32_t)b.r_max, kSgmvBK)) return rc;
    if (int rc = make_tmap_2d(&maps.b[a.n], b.st.b[s], (uint64_t)b.S * b.st.out[s], (uint64_t)b.r_max, (uint64_t)b.r_max, kPcBox, (uint32_t)b.r_max)) return rc;
    ++a.n;
  }
  for (int s = a.n; s < B200_LORA_MAX_SLICES; ++s) { maps.a[s] = maps.a[0]; maps.b[s] = maps.b[0]; }
  if (int rc = make_tmap_2d(&maps.x, b.x, (uint64_t)b.T, (uint64_t)b.in_dim, (uint64_t)b.x_ld, (uint32_t)a.bm, kSgmvBK)) return rc;
  if (int rc = make_tmap_2d(&maps.y, b.y, (uint64_t)b.T, (uint64_t)n_total, (uint64_t)b.y_ld, (uint32_t)a.bm, kGemmOutChunk)) return rc;
  maps.w = maps.x;
  if (linear)
    if (int rc = make_tmap_2d(&maps.w, weight, (uint64_t)n_total, (uint64_t)b.in_dim, (uint64_t)w_ld, kPcBox, kSgmvBK)) return rc;
  const auto kernel = linear ? prefill_cluster_kernel<true> : prefill_cluster_kernel<false>;
  if (int rc = sgmv_set_smem(reinterpret_cast<const void*>(kernel), kPcSmem)) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ceil_div_i(b.T, a.bm) * a.groups * a.ck), 1, 1);
  cfg.blockDim = dim3(kPcThreads, 1, 1);
  cfg.dynamicSmemBytes = kPcSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)a.ck;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = bgmv_options().pdl ? 2 : 1;  // B200_LORA_OPT_PDL = 0: strict stream order
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, maps, a);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(B200_LORA_ECUDA, "prefill_cluster_kernel launch: %s", cudaGetErrorString(e));
  }
  return B200_LORA_OK;
}

// Whether the kernel takes an ADD launch: slices that tile the output in 64-column units, a block of rows per SM at most.
inline bool prefill_cluster_add_ok(const SgmvProblem& b) {
  int n = 0, pos = 0;
  for (int s = 0; s < b.st.n; ++s) {
    if (b.st.out[s] == 0) continue;
    if (b.st.col[s] != pos || b.st.out[s] % kGemmOutChunk != 0) return false;
    pos += b.st.out[s];
    ++n;
  }
  return n * b.r_max <= 256 && ceil_div_i(b.T, kSgmvBM) <= kTileSMs;
}

// y += LoRA delta for a prefill batch (overwrite: y = delta). Scratch is for the two launches of what the kernel does not take.
inline int prefill_add(const SgmvProblem& b, void* workspace, size_t workspace_bytes, cudaStream_t stream, bool overwrite = false) {
  const char* why = nullptr;
  if (!prefill_cluster_add_ok(b)) return prefill_add_launch(b, workspace, workspace_bytes, stream, overwrite);
  if (!sgmv_supported(b, &why)) return fail(B200_LORA_EUNSUPPORTED, "prefill kernels: %s", why);
  int n = 0, n_total = 0;
  for (int s = 0; s < b.st.n; ++s) {
    n += b.st.out[s] > 0;
    if (b.st.out[s] > 0) n_total = std::max(n_total, b.st.col[s] + b.st.out[s]);
  }
  PcArgs a = {};
  if (!prefill_cluster_plan(b, n, n_total, false, &a)) return fail(B200_LORA_EUNSUPPORTED, "prefill kernel: too many rank rows");
  return prefill_cluster_launch(b, a, nullptr, 0, n_total, nullptr, overwrite, stream);
}

}  // namespace b200lora
