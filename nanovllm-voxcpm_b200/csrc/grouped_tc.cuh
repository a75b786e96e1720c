// Multi-LoRA add for bucketed batches on the Blackwell tensor cores, two launches: shrink (x . A^T, fp32 partial sums to
// scratch) and expand (tmp . B^T, added to y), both in the weight-stationary form D^T = W . act^T: the adapter's rows are
// the 128-row operand of tcgen05.mma and the bucket's tokens its N operand (16 or 32 columns).
//
// Why this form. A bucket's weights are fetched once per 32 tokens, by CTAs that share the tiles of all buckets evenly. The
// fused decode kernel (bgmv_fused.cuh) gives every 16 tokens a cluster of its own, which fetches the adapter again and takes
// as long as its slowest cluster; it stays the kernel of most batches, because its single launch is shorter than two
// (grouped_preferred has the line between them).
//
// Both kernels are persistent, one CTA per SM: every CTA builds the list of (bucket, 32-token chunk) pairs in use from the
// index arrays (graph buffers carry one bucket per slot, most of them empty) and takes items of it in turn:
//   shrink item = (chunk, group of slices whose rank rows fit the 128 rows, K part)
//   expand item = (chunk, slice, run of 128-row output tiles)
// Under programmatic dependent launch a CTA builds its list and fills its ring of weight tiles (TMA, 128 / 64 / 32-byte
// swizzle) before it waits for the previous kernel. Its ring is 84 KB, so that the CTA of the next launch is resident beside
// it, or 196 KB where a launch streams many bytes (grouped_ring_bytes).
//
// Precision: tmp stays fp32 between the launches and is multiplied as the sum of two 16-bit numbers (hi + lo), the K parts
// are added in fp32, and y is read, added to in fp32 and rounded once - what the per-token kernels compute. Where the fused
// decode kernel rounds the delta to bf16 and adds it at the L2, the delta is rounded here too (round_delta) and needs hi only.
#pragma once

#include "bgmv_fused.cuh"
#include "tc_common.cuh"

namespace b200lora {

constexpr int kGrpTok = 32;            // tokens per chunk (N of an MMA)
constexpr int kGrpRows = 128;          // weight rows per tile (M of an MMA)
constexpr int kGrpBK = 64;             // K columns per shrink panel (one 128-byte swizzle row)
constexpr int kGrpMaxChunks = 2560;    // entries of the chunk list
constexpr int kGrpMaxBuckets = 2048;
constexpr int kGrpMaxSplit = 8;        // K parts of the shrink
constexpr int kGrpShrinkThreads = 256; // warp 0 lora_A, warp 1 MMA, warps 2-5 epilogue, warps 6-7 x rows (every other stage)
constexpr int kGrpExpandThreads = 416; // warp 0 lora_B, warps 1 / 12 MMA of even / odd tiles, 2-9 epilogue (4 + 4), 10-11 tmp rows
constexpr int kGrpAcc = 4;             // expand: accumulators of 32 columns in TMEM
constexpr int kGrpMaxStages = 12;
constexpr int kGrpSMs = 148;

struct GroupedArgs {
  uint8_t* y; int64_t y_ld;            // 16-bit elements
  int T, in_dim, S, r, n;
  int out[B200_LORA_MAX_SLICES], col[B200_LORA_MAX_SLICES];
  const int32_t *sorted_idx, *slot_ids, *counts, *offsets;
  const int32_t* rank_per_slot; const float* scale_per_slot;
  int n_buckets;
  float scaling;
  int f16;                             // fp16 instead of bf16
  float* tmp;                          // shrink result / expand input [parts, n, T, r]
  int parts, k_part;                   // K parts and their width (multiple of kGrpBK)
  int panels, w_bytes;                 // shrink: 64-column panels per stage, bytes of its lora_A part
  int whole_stage;                     // shrink: one slice per operand, its panels of a stage arrive in one copy (3-D map)
  int spg, m_groups;                   // shrink: slices per 128-row operand, number of such groups
  int tile_cost;                       // expand: cost of fetching a weight tile, in units of one 16-token epilogue block
  int round_delta;                     // expand: add the delta rounded to bf16 with a reduction at the L2 (y is not read)
  int stages;                          // ring stages
};

struct GroupedMaps {
  CUtensorMap x;                       // shrink: [T, in], box 1 x 64 (rows are gathered)
  CUtensorMap w[B200_LORA_MAX_SLICES]; // shrink: lora_A [S*r, in], box r x 64; expand: lora_B [S*out, r], box 128 x r
};

// kind::f16 instruction descriptor for bf16 or fp16 operands (both of one type)
__device__ __forceinline__ uint32_t umma_idesc_16bit(int M, int N, int f16) {
  const uint32_t t = f16 ? 0u : 1u;
  return (1u << 4) | (t << 7) | (t << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ uint16_t to_16bit(float v, int f16) {
  return f16 ? __half_as_ushort(__float2half_rn(v)) : __bfloat16_as_ushort(__float2bfloat16_rn(v));
}
__device__ __forceinline__ float from_16bit(uint16_t v, int f16) {
  return f16 ? __half2float(__ushort_as_half(v)) : __bfloat162float(__ushort_as_bfloat16(v));
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst_smem, const CUtensorMap* tmap, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst_smem), "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}
// Four rows y0..y3 of a 2-D map (box one row high), 64 columns from c0, to 4 x 128 consecutive bytes (swizzled)
__device__ __forceinline__ void tma_gather4(uint32_t dst_smem, const CUtensorMap* tmap, int c0, int y0, int y1, int y2, int y3, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
      ::"r"(dst_smem), "l"(tmap), "r"(c0), "r"(y0), "r"(y1), "r"(y2), "r"(y3), "r"(bar)
      : "memory");
}

// Cost of the output tiles of a chunk of `cnt` tokens, per tile: the fetch of its weights and its epilogue blocks.
__device__ __forceinline__ int grouped_tile_cost(const GroupedArgs& a, int cnt) { return a.tile_cost + ((cnt + 15) >> 4); }

// Chunks in use: list[i] = bucket | chunk << 16. Every thread of the CTA calls this; returns the number of entries.
// (A bucket whose id, rank or row range is unusable has no chunks; both kernels see the same list.)
// With `cost` != nullptr cost[i] = sum of the tile costs of the chunks before i (one tile each), *total the sum of all.
template <int THREADS>
__device__ __forceinline__ int grouped_chunk_list(const GroupedArgs& a, int* list, int* cost, int (*scan)[2], int* total) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kWarps = THREADS / 32;
  const int full = grouped_tile_cost(a, kGrpTok);
  int base = 0, base_cost = 0;
  for (int b0 = 0; b0 < a.n_buckets; b0 += THREADS) {
    const int b = b0 + tid;
    int k = 0, w = 0;
    if (b < a.n_buckets) {
      const int slot = a.slot_ids[b], cnt = a.counts[b], start = a.offsets[b];
      if (cnt > 0 && slot >= 0) (void)B200_IN_BOUNDS(slot < a.S && start >= 0 && start <= a.T - cnt);
      const bool ok = slot >= 0 && slot < a.S && cnt > 0 && start >= 0 && start <= a.T - cnt &&
                      (a.rank_per_slot == nullptr || a.rank_per_slot[slot] > 0);
      if (ok) {
        k = (cnt + kGrpTok - 1) / kGrpTok;
        w = (k - 1) * full + grouped_tile_cost(a, cnt - (k - 1) * kGrpTok);
      }
    }
    int incl = k, incl_w = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o), u = __shfl_up_sync(0xffffffffu, incl_w, o);
      if (lane >= o) { incl += v; incl_w += u; }
    }
    if (lane == 31) { scan[warp][0] = incl; scan[warp][1] = incl_w; }
    __syncthreads();
    int before = base, before_w = base_cost, sum = 0, sum_w = 0;
#pragma unroll
    for (int v = 0; v < kWarps; ++v) {
      if (v < warp) { before += scan[v][0]; before_w += scan[v][1]; }
      sum += scan[v][0]; sum_w += scan[v][1];
    }
    before += incl - k; before_w += incl_w - w;
    for (int i = 0; i < k; ++i)
      if (before + i < kGrpMaxChunks) {
        list[before + i] = b | (i << 16);
        if (cost != nullptr) cost[before + i] = before_w + i * full;
      }
    base += sum; base_cost += sum_w;
    __syncthreads();
  }
  *total = base_cost;
  return min(base, kGrpMaxChunks);
}

// ============================================================================ shrink
__global__ void __launch_bounds__(kGrpShrinkThreads, 1)
grouped_shrink_kernel(const __grid_constant__ GroupedMaps maps, const GroupedArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ int list[kGrpMaxChunks];
  __shared__ int scan[kGrpShrinkThreads / 32][2];
  __shared__ __align__(8) uint64_t bars[2 * kGrpMaxStages + 4];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t smem_base = (smem_u32(smem) + 1023u) & ~1023u;
  constexpr uint32_t kXPanel = kGrpTok * kGrpBK * 2;
  const int P = a.panels, NS = a.stages, step = P * kGrpBK;
  const uint32_t w_bytes = (uint32_t)a.w_bytes, stage = w_bytes + (uint32_t)P * kXPanel;
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * (uint32_t)s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (uint32_t)(kGrpMaxStages + s); };
  auto acc_full = [&](int b) { return bar0 + 8u * (uint32_t)(2 * kGrpMaxStages + b); };
  auto acc_empty = [&](int b) { return bar0 + 8u * (uint32_t)(2 * kGrpMaxStages + 2 + b); };
  if (tid == 0) {
    for (int s = 0; s < NS; ++s) { mbar_init(full_bar(s), 2); mbar_init(empty_bar(s), 1); }  // full: lora_A and x
    for (int b = 0; b < 2; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 128); }
    abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_s), 2 * kGrpTok);
    tc_fence_before_sync();
  }
  int cost_sum;
  const int n_chunks = grouped_chunk_list<kGrpShrinkThreads>(a, list, nullptr, scan, &cost_sum);
  __syncthreads();
  griddep_launch_dependents();  // only now that this CTA holds its tensor memory
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  const int per_chunk = a.m_groups * a.parts;
  const int items = n_chunks * per_chunk;
  struct Item { int bucket, chunk, g0, gn, part, k0, nk; };
  auto item_at = [&](int i) {
    Item t;
    const int c = i / per_chunk, rest = i - c * per_chunk;
    t.bucket = list[c] & 0xffff; t.chunk = list[c] >> 16;
    const int mg = rest / a.parts;
    t.part = rest - mg * a.parts;
    t.g0 = mg * a.spg; t.gn = min(a.spg, a.n - t.g0);
    t.k0 = t.part * a.k_part;
    t.nk = (min(a.k_part, a.in_dim - t.k0) + step - 1) / step;
    return t;
  };

  // The producers run converged too (see umma_elected): a TMA instruction issued from divergent code costs 130 cycles.
  if (warp == 0) {
    // lora_A panels. The weights do not depend on the previous kernel of the stream.
    const uint32_t leader = elect_one();
    if (leader)
      for (int s = 0; s < a.n; ++s) tma_prefetch_desc(&maps.w[s]);
    int st = 0, round = 0;
    for (int i = blockIdx.x; i < items; i += gridDim.x) {
      const Item t = item_at(i);
      const int row = uniform(a.slot_ids[t.bucket] * a.r), gn = uniform(t.gn), g0 = uniform(t.g0), nk = uniform(t.nk);
      int col = uniform(t.k0);
      const uint32_t slice_bytes = (uint32_t)(a.r * kGrpBK * 2);
      for (int kc = 0; kc < nk; ++kc, col += step) {
        if (round > 0) mbar_wait_bounded(empty_bar(st), (uint32_t)((round & 1) ^ 1), &abort_flag);
        if (leader) {
          const uint32_t base = smem_base + (uint32_t)st * stage, bar = full_bar(st);
          mbar_arrive_expect_tx(bar, (uint32_t)(P * gn) * slice_bytes);
          // stage = [panel][slice][rank row]; a panel beyond the end of the rows arrives as zeros
          if (a.whole_stage) {
            tma_load_3d(base, &maps.w[g0], 0, row, col / kGrpBK, bar);
          } else {
            for (int p = 0; p < P; ++p)
              for (int s = 0; s < gn; ++s)
                tma_load_2d(base + (uint32_t)(p * gn + s) * slice_bytes, &maps.w[g0 + s], col + p * kGrpBK, row, bar);
          }
        }
        __syncwarp();
        if (++st == NS) { st = 0; ++round; }
      }
    }
    griddep_wait();  // a launch never ends before its predecessor
  } else if (warp >= 6) {
    // x rows of the chunk's tokens, four per copy; the two warps take every other stage
    const uint32_t leader = elect_one();
    if (leader) tma_prefetch_desc(&maps.x);
    const int mine = warp - 6;
    int st = 0, round = 0, n = 0;
    bool waited = false;
    for (int i = blockIdx.x; i < items; i += gridDim.x) {
      const Item t = item_at(i);
      const int first = a.offsets[t.bucket] + t.chunk * kGrpTok;
      const int cnt = min(kGrpTok, a.counts[t.bucket] - t.chunk * kGrpTok), quads = uniform((cnt + 15) >> 4) * 4;
      int tok = a.sorted_idx[first + min(lane, cnt - 1)];  // columns beyond the count repeat the last token and are not read
      (void)B200_IN_BOUNDS(tok >= 0 && tok < a.T);
      if (tok < 0 || tok >= a.T) tok = 0;
      const int nk = uniform(t.nk);
      int col = uniform(t.k0);
      if (!waited) { griddep_wait(); waited = true; }  // x is final from here on (the index arrays were before)
      for (int kc = 0; kc < nk; ++kc, ++n, col += step) {
        if ((n & 1) == mine) {
          if (round > 0) mbar_wait_bounded(empty_bar(st), (uint32_t)((round & 1) ^ 1), &abort_flag);
          const uint32_t xs = smem_base + (uint32_t)st * stage + w_bytes, bar = full_bar(st);
          if (leader) mbar_arrive_expect_tx(bar, (uint32_t)(P * quads) * 512u);
          __syncwarp();
          for (int q = 0; q < quads; ++q) {
            const int y0 = __shfl_sync(0xffffffffu, tok, 4 * q), y1 = __shfl_sync(0xffffffffu, tok, 4 * q + 1);
            const int y2 = __shfl_sync(0xffffffffu, tok, 4 * q + 2), y3 = __shfl_sync(0xffffffffu, tok, 4 * q + 3);
            if (leader)
              for (int p = 0; p < P; ++p)
                tma_gather4(xs + (uint32_t)p * kXPanel + (uint32_t)q * 512u, &maps.x, col + p * kGrpBK, y0, y1, y2, y3, bar);
          }
          __syncwarp();
        }
        if (++st == NS) { st = 0; ++round; }
      }
    }
  } else if (warp == 1) {
    const uint32_t leader = elect_one();
    const uint64_t desc0 = umma_smem_desc(smem_base, 128);
    const uint32_t hi = (uint32_t)(desc0 >> 32), lo0 = (uint32_t)desc0;
    int st = 0, round = 0, job = 0;
    for (int i = blockIdx.x; i < items; i += gridDim.x, ++job) {
      const Item t = item_at(i);
      const int nk = uniform(t.nk);
      const uint32_t panel = (uint32_t)uniform(t.gn * a.r * kGrpBK * 2) >> 4;
      const uint32_t idesc = (uint32_t)uniform((int)umma_idesc_16bit(kGrpRows, (min(kGrpTok, a.counts[t.bucket] - t.chunk * kGrpTok) + 15) & ~15, a.f16));
      const int buf = job & 1;
      const uint32_t d = tmem_base + (uint32_t)(buf * kGrpTok);
      if (job >= 2) mbar_wait_bounded(acc_empty(buf), (uint32_t)(((job >> 1) - 1) & 1), &abort_flag);
      tc_fence_after_sync();
      for (int kc = 0; kc < nk; ++kc) {
        mbar_wait_bounded(full_bar(st), (uint32_t)(round & 1), &abort_flag);
        tc_fence_after_sync();
        // (rows of a tile beyond the rank rows hold whatever lies there; their accumulator rows are not read)
        uint32_t w = lo0 + ((uint32_t)st * stage >> 4), xr = w + (w_bytes >> 4);
        for (int p = 0; p < P; ++p) {
#pragma unroll
          for (int k4 = 0; k4 < kGrpBK / 16; ++k4)
            umma_elected(d, w + 2u * k4, xr + 2u * k4, hi, idesc, (kc > 0 || p > 0 || k4 > 0) ? 1u : 0u, leader);
          w += panel; xr += kXPanel >> 4;
        }
        umma_commit_elected(empty_bar(st), leader);
        if (++st == NS) { st = 0; ++round; }
      }
      umma_commit_elected(acc_full(buf), leader);
    }
  } else {
    // epilogue: lane <-> stacked rank row, column <-> token
    const int quarter = warp & 3, q = quarter * 32 + lane;
    griddep_wait();  // the previous launch may still read the scratch
    int job = 0;
    for (int i = blockIdx.x; i < items; i += gridDim.x, ++job) {
      const Item t = item_at(i);
      const int slot = a.slot_ids[t.bucket], first = a.offsets[t.bucket] + t.chunk * kGrpTok;
      const int cnt = min(kGrpTok, a.counts[t.bucket] - t.chunk * kGrpTok);
      const int s = t.g0 + q / a.r, j = q % a.r;
      const bool mine = q < t.gn * a.r;
      float sc = a.scaling * (a.scale_per_slot != nullptr ? a.scale_per_slot[slot] : 1.0f);
      const int rank = a.rank_per_slot != nullptr ? a.rank_per_slot[slot] : a.r;
      const int tok = lane < cnt ? a.sorted_idx[first + lane] : -1;
      const int buf = job & 1;
      mbar_wait_bounded(acc_full(buf), (uint32_t)((job >> 1) & 1), &abort_flag);
      tc_fence_after_sync();
      const int64_t plane = ((int64_t)t.part * a.n + s) * a.T;
      if (quarter * 32 < t.gn * a.r) {  // warp-uniform
#pragma unroll
        for (int c = 0; c < kGrpTok; c += 16) {
          if (c < cnt) {
            uint32_t v[16];
            tmem_ld_32x16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * kGrpTok + c), v);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const int row = __shfl_sync(0xffffffffu, tok, c + e);
              if (mine && row >= 0 && row < a.T) a.tmp[(plane + row) * a.r + j] = j < rank ? __uint_as_float(v[e]) * sc : 0.f;
            }
          }
        }
      }
      tc_fence_before_sync();
      mbar_arrive_relaxed(acc_empty(buf));
    }
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 2 * kGrpTok);
  if (tid == 0 && abort_flag != 0) atomicOr(&g_b200_status, kStatusWaitGaveUp);
}

// ============================================================================ expand
__global__ void __launch_bounds__(kGrpExpandThreads, 1)
grouped_expand_kernel(const __grid_constant__ GroupedMaps maps, const GroupedArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ int list[kGrpMaxChunks];
  __shared__ int scan[kGrpExpandThreads / 32][2];
  __shared__ int cost[kGrpMaxChunks];
  __shared__ int first_chunk_s;
  __shared__ int rows_s[2][kGrpTok];                       // token row of every column, -1 beyond the count
  __shared__ __align__(8) uint64_t bars[2 * kGrpMaxStages + 2 * kGrpAcc + 4];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t smem_base = (smem_u32(smem) + 1023u) & ~1023u;
  const int r = a.r, row_bytes = r * 2, NS = a.stages;
  const uint32_t stage_bytes = (uint32_t)(kGrpRows * row_bytes);
  const uint32_t half_bytes = (uint32_t)(kGrpTok * row_bytes);  // one of hi / lo
  const uint32_t tmp_base = smem_base + (uint32_t)NS * stage_bytes;
  const int halves = a.round_delta ? 1 : 2;  // (a delta that is rounded anyway does not need the low half)
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * (uint32_t)s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (uint32_t)(kGrpMaxStages + s); };
  auto acc_full = [&](int b) { return bar0 + 8u * (uint32_t)(2 * kGrpMaxStages + b); };
  auto acc_empty = [&](int b) { return bar0 + 8u * (uint32_t)(2 * kGrpMaxStages + kGrpAcc + b); };
  auto tmp_full = [&](int b) { return bar0 + 8u * (uint32_t)(2 * kGrpMaxStages + 2 * kGrpAcc + b); };
  auto tmp_empty = [&](int b) { return bar0 + 8u * (uint32_t)(2 * kGrpMaxStages + 2 * kGrpAcc + 2 + b); };
  if (tid == 0) {
    for (int s = 0; s < NS; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int b = 0; b < kGrpAcc; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 128); }
    for (int b = 0; b < 2; ++b) { mbar_init(tmp_full(b), 64); mbar_init(tmp_empty(b), 2 + 256); }  // MMA warps, epilogue (row table)
    abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_s), kGrpAcc * kGrpTok);
    tc_fence_before_sync();
  }
  int cost_sum;
  const int n_chunks = grouped_chunk_list<kGrpExpandThreads>(a, list, cost, scan, &cost_sum);
  __syncthreads();
  griddep_launch_dependents();  // only now that this CTA holds its tensor memory
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  // The tiles of all chunks, chunk by chunk and slice by slice, are dealt to the CTAs in contiguous ranges of equal cost
  // (a chunk of 32 tokens costs more than one of three: with equal numbers of tiles the CTAs of a popular adapter finished
  // last by a factor). An item is the part of the range inside one slice of one chunk.
  int tile_end[B200_LORA_MAX_SLICES], per_chunk = 0;
#pragma unroll
  for (int s = 0; s < B200_LORA_MAX_SLICES; ++s) {
    if (s < a.n) per_chunk += ceil_div_i(a.out[s], kGrpRows);
    tile_end[s] = per_chunk;
  }
  const int64_t all = (int64_t)cost_sum * per_chunk;
  const int64_t range_lo = all * blockIdx.x / gridDim.x, range_hi = all * (blockIdx.x + 1) / gridDim.x;
  if (tid == 0) first_chunk_s = 0;
  __syncthreads();
  for (int c = tid; c < n_chunks; c += kGrpExpandThreads)  // last chunk that starts at or before the range
    if ((int64_t)cost[c] * per_chunk <= range_lo) atomicMax(&first_chunk_s, c);
  __syncthreads();
  const int first_chunk = first_chunk_s;
  struct Item { int bucket, chunk, cnt, s, out, col, tile0, tiles; };
  // cursor: chunk c, next tile of it; false when the range is used up
  auto next_item = [&](int& c, int& tile, int& stop, Item& t) {
    while (tile >= stop) {  // next chunk
      if (++c >= n_chunks) return false;
      const int64_t at = (int64_t)cost[c] * per_chunk;
      if (at >= range_hi) return false;
      const int bucket = list[c] & 0xffff;
      const int w = grouped_tile_cost(a, min(kGrpTok, a.counts[bucket] - (list[c] >> 16) * kGrpTok));
      tile = at >= range_lo ? 0 : (int)((range_lo - at + w - 1) / w);
      stop = (int)min((int64_t)per_chunk, (range_hi - at + w - 1) / w);
    }
    t.bucket = list[c] & 0xffff; t.chunk = list[c] >> 16;
    t.cnt = min(kGrpTok, a.counts[t.bucket] - t.chunk * kGrpTok);
    int before = 0, end = tile_end[0];
    t.s = 0; t.out = a.out[0]; t.col = a.col[0];
#pragma unroll
    for (int s = 1; s < B200_LORA_MAX_SLICES; ++s)
      if (s < a.n && tile >= tile_end[s - 1]) { t.s = s; t.out = a.out[s]; t.col = a.col[s]; before = tile_end[s - 1]; end = tile_end[s]; }
    t.tile0 = tile - before;
    t.tiles = min(end, stop) - tile;
    tile += t.tiles;
    return true;
  };
#define B200_FOR_EACH_ITEM(t) \
  Item t;                     \
  for (int c_ = first_chunk - 1, tile_ = 0, stop_ = 0; next_item(c_, tile_, stop_, t);)

  if (warp == 0) {
    const uint32_t leader = elect_one();
    if (leader)
      for (int s = 0; s < a.n; ++s) tma_prefetch_desc(&maps.w[s]);
    int st = 0, round = 0;
    B200_FOR_EACH_ITEM(t) {
      int row = uniform(a.slot_ids[t.bucket] * t.out + t.tile0 * kGrpRows);
      const int tiles = uniform(t.tiles), s = uniform(t.s);
      for (int j = 0; j < tiles; ++j, row += kGrpRows) {
        if (round > 0) mbar_wait_bounded(empty_bar(st), (uint32_t)((round & 1) ^ 1), &abort_flag);
        if (leader) {
          mbar_arrive_expect_tx(full_bar(st), stage_bytes);
          tma_load_2d(smem_base + (uint32_t)st * stage_bytes, &maps.w[s], 0, row, full_bar(st));
        }
        __syncwarp();
        if (++st == NS) { st = 0; ++round; }
      }
    }
    griddep_wait();
  } else if (warp == 1 || warp == 12) {
    // two issuing warps, one for the even and one for the odd tiles of the CTA: waits and issue of a tile take 500 cycles
    const uint32_t leader = elect_one();
    const uint64_t desc0 = umma_smem_desc(smem_base, row_bytes);
    const uint32_t hi = (uint32_t)(desc0 >> 32), lo0 = (uint32_t)desc0, tmp_lo0 = lo0 + ((tmp_base - smem_base) >> 4);
    const int turn = warp == 12;
    int st = 0, round = 0, job = 0, it = 0;
    B200_FOR_EACH_ITEM(t) {
      const uint32_t idesc = (uint32_t)uniform((int)umma_idesc_16bit(kGrpRows, (t.cnt + 15) & ~15, a.f16));
      const int tiles = uniform(t.tiles), tb = it & 1;
      mbar_wait_bounded(tmp_full(tb), (uint32_t)((it >> 1) & 1), &abort_flag);
      tc_fence_after_sync();
      const uint32_t tmp_lo = tmp_lo0 + ((uint32_t)(2 * tb) * half_bytes >> 4);
      for (int j = 0; j < tiles; ++j, ++job, st = st + 1 == NS ? 0 : st + 1, round += st == 0) {
        if ((job & 1) != turn) continue;
        const int buf = job % kGrpAcc;
        const uint32_t d = tmem_base + (uint32_t)(buf * kGrpTok), w = lo0 + ((uint32_t)st * stage_bytes >> 4);
        if (job >= kGrpAcc) mbar_wait_bounded(acc_empty(buf), (uint32_t)((job / kGrpAcc - 1) & 1), &abort_flag);
        mbar_wait_bounded(full_bar(st), (uint32_t)(round & 1), &abort_flag);
        tc_fence_after_sync();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (h >= halves) break;
          const uint32_t tl = tmp_lo + (uint32_t)h * (half_bytes >> 4);
#pragma unroll
          for (int k4 = 0; k4 < 4; ++k4)
            if (16 * k4 < r) umma_elected(d, w + 2u * k4, tl + 2u * k4, hi, idesc, (h > 0 || k4 > 0) ? 1u : 0u, leader);
        }
        umma_commit_elected(empty_bar(st), leader);
        umma_commit_elected(acc_full(buf), leader);
      }
      umma_commit_elected(tmp_empty(tb), leader);
      ++it;
    }
  } else if (warp == 10 || warp == 11) {
    // rank-r rows of the chunk's tokens: sum of the K parts, as hi + lo 16-bit numbers in the swizzle of the operand tile
    const int lt = tid - 320;
    int it = 0;
    bool waited = false;
    B200_FOR_EACH_ITEM(t) {
      const int first = a.offsets[t.bucket] + t.chunk * kGrpTok;
      const int cnt = t.cnt, rows = (cnt + 15) & ~15;
      const int tb = it & 1;
      if (it >= 2) mbar_wait_bounded(tmp_empty(tb), (uint32_t)(((it >> 1) - 1) & 1), &abort_flag);
      const uint32_t hi = tmp_base + (uint32_t)(2 * tb) * half_bytes, lo = hi + half_bytes;
      if (lt < kGrpTok) {
        int tok = lt < cnt ? a.sorted_idx[first + lt] : -1;
        if (lt < cnt) (void)B200_IN_BOUNDS(tok >= 0 && tok < a.T);
        rows_s[tb][lt] = tok >= 0 && tok < a.T ? tok : -1;
      }
      const int pieces = r >> 3;  // 8 ranks per piece
      named_bar_sync(1, 64);  // row table complete
      if (!waited) { griddep_wait(); waited = true; }  // tmp is final from here on
      for (int e = lt; e < rows * pieces; e += 64) {
        const int row = e / pieces, p = e - row * pieces, tok = rows_s[tb][row];
        float v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = 0.f;
        if (tok >= 0) {
          for (int part = 0; part < a.parts; ++part) {
            const float4* src = reinterpret_cast<const float4*>(a.tmp + (((int64_t)part * a.n + t.s) * a.T + tok) * r + 8 * p);
            const float4 f0 = __ldcg(src), f1 = __ldcg(src + 1);
            v[0] += f0.x; v[1] += f0.y; v[2] += f0.z; v[3] += f0.w;
            v[4] += f1.x; v[5] += f1.y; v[6] += f1.z; v[7] += f1.w;
          }
        }
        uint32_t h[4], l[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint16_t h0 = to_16bit(v[2 * q], a.f16), h1 = to_16bit(v[2 * q + 1], a.f16);
          const uint16_t l0 = to_16bit(v[2 * q] - from_16bit(h0, a.f16), a.f16), l1 = to_16bit(v[2 * q + 1] - from_16bit(h1, a.f16), a.f16);
          h[q] = h0 | ((uint32_t)h1 << 16);
          l[q] = l0 | ((uint32_t)l1 << 16);
        }
        // TMA swizzle of a row of 128 / 64 / 32 bytes: 16-byte piece index XOR address bits 7..9 (8..7, 7)
        const int x = row_bytes == 128 ? (row & 7) : row_bytes == 64 ? ((row >> 1) & 3) : ((row >> 2) & 1);
        const uint32_t at = (uint32_t)(row * row_bytes + ((p ^ x) << 4));
        sts128(hi + at, make_uint4(h[0], h[1], h[2], h[3]));
        if (halves == 2) sts128(lo + at, make_uint4(l[0], l[1], l[2], l[3]));
      }
      fence_proxy_async_smem();
      mbar_arrive(tmp_full(tb));
      ++it;
    }
  } else {
    // epilogue: lane <-> output row of the tile, column <-> token. Two groups of four warps take turns. The eight lanes of
    // a group of rows trade values (three butterfly steps), after which a lane holds eight adjacent outputs of two tokens:
    // y is updated in 16-byte pieces.
    const int quarter = warp & 3, p = lane & 7, group = warp >= 6;
    griddep_wait();
    int job = 0, it = 0;
    B200_FOR_EACH_ITEM(t) {
      const int cnt = t.cnt, tb = it & 1;
      mbar_wait_bounded(tmp_full(tb), (uint32_t)((it >> 1) & 1), &abort_flag);
      for (int j = 0; j < t.tiles; ++j, ++job) {
        if ((job & 1) != group) continue;
        const int buf = job % kGrpAcc;
        const int o = (t.tile0 + j) * kGrpRows + quarter * 32 + (lane & ~7);  // first of the eight outputs
        const bool live = o < t.out;
        uint16_t* const ycol = reinterpret_cast<uint16_t*>(a.y) + t.col + o;
        bool ready = false;
#pragma unroll 1
        for (int c = 0; c < cnt; c += 16) {
          uint16_t* dst[2];
          uint4 old[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int row = rows_s[tb][c + p + 8 * h];
            dst[h] = live && row >= 0 ? ycol + (int64_t)row * a.y_ld : nullptr;
            if (!a.round_delta && dst[h] != nullptr) old[h] = ldg128(dst[h]);
          }
          if (!ready) {
            mbar_wait_bounded(acc_full(buf), (uint32_t)((job / kGrpAcc) & 1), &abort_flag);
            tc_fence_after_sync();
            ready = true;
          }
          uint32_t v[16];
          tmem_ld_32x16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * kGrpTok + c), v);
          tmem_ld_wait();
          // step k: keep the tokens whose bit k equals the lane's, get the same tokens of the row with bit k flipped
          uint32_t w1[8][2], w2[4][4];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint32_t keep = (p & 1) ? v[2 * q + 1] : v[2 * q], give = (p & 1) ? v[2 * q] : v[2 * q + 1];
            const uint32_t got = __shfl_xor_sync(0xffffffffu, give, 1);
            w1[q][0] = (p & 1) ? got : keep;
            w1[q][1] = (p & 1) ? keep : got;
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
              const uint32_t keep = (p & 2) ? w1[2 * q + 1][b] : w1[2 * q][b], give = (p & 2) ? w1[2 * q][b] : w1[2 * q + 1][b];
              const uint32_t got = __shfl_xor_sync(0xffffffffu, give, 2);
              w2[q][b] = (p & 2) ? got : keep;
              w2[q][2 + b] = (p & 2) ? keep : got;
            }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float d[8];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              const uint32_t keep = (p & 4) ? w2[2 * h + 1][b] : w2[2 * h][b], give = (p & 4) ? w2[2 * h][b] : w2[2 * h + 1][b];
              const uint32_t got = __shfl_xor_sync(0xffffffffu, give, 4);
              d[b] = __uint_as_float((p & 4) ? got : keep);
              d[4 + b] = __uint_as_float((p & 4) ? keep : got);
            }
            if (dst[h] == nullptr) continue;
            if (a.round_delta) {
              red_add_bf16x8(dst[h], pack_bf16x2(d[0], d[1]), pack_bf16x2(d[2], d[3]), pack_bf16x2(d[4], d[5]), pack_bf16x2(d[6], d[7]));
            } else {
              uint32_t u[4] = {old[h].x, old[h].y, old[h].z, old[h].w};
#pragma unroll
              for (int b = 0; b < 4; ++b) {
                if (a.f16) {
                  const __half2 y2 = *reinterpret_cast<const __half2*>(&u[b]);
                  const __half2 res = __floats2half2_rn(__low2float(y2) + d[2 * b], __high2float(y2) + d[2 * b + 1]);
                  u[b] = *reinterpret_cast<const uint32_t*>(&res);
                } else {
                  u[b] = add_bf16x2(u[b], d[2 * b], d[2 * b + 1]);
                }
              }
              stg128(dst[h], make_uint4(u[0], u[1], u[2], u[3]));
            }
          }
        }
        tc_fence_before_sync();
        mbar_arrive_relaxed(acc_empty(buf));  // (a releasing arrive would wait for the updates of y: 1 us per tile)
      }
      mbar_arrive_relaxed(tmp_empty(tb));
      ++it;
    }
  }
#undef B200_FOR_EACH_ITEM
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, kGrpAcc * kGrpTok);
  if (tid == 0 && abort_flag != 0) atomicOr(&g_b200_status, kStatusWaitGaveUp);
}

// ============================================================================ host side
struct GroupedProblem {
  void* y; int64_t y_ld; const void* x; int64_t x_ld;
  int T, in_dim, S, r_max;
  SliceTable st;
  const int32_t* rank_per_slot; const float* scale_per_slot;
  const int32_t *sorted_idx, *slot_ids, *counts, *offsets;
  int n_buckets; float scaling;
  int dtype;
};

// K parts of the shrink for `chunks` chunks of `groups` slice groups: about six items per SM, so that the last ones even
// out; or one round of items where that is all there is.
inline int grouped_parts(int chunks, int groups, int in_dim) {
  const int n = chunks * groups, want = 2 * n <= kGrpSMs ? kGrpSMs / n : ceil_div_i(6 * kGrpSMs, n);
  const int parts = std::max(1, std::min(std::min(want, kGrpMaxSplit), ceil_div_i(in_dim, kGrpBK)));
  return ceil_div_i(in_dim, round_up_i(ceil_div_i(in_dim, parts), kGrpBK));
}

// Scratch of the largest split that a batch of T rows can get: it has at least T / 32 chunks in use and any number above
// that. More chunks do not always mean fewer parts (one round of items up to half the SMs, six rounds above), so the bound is
// the larger of the two sides of that line.
inline size_t grouped_workspace_bytes(int T, int n_slices, int r_max) {
  const int chunks = std::max(T / kGrpTok, kGrpSMs / 2 + 1);
  return (size_t)std::min(kGrpMaxSplit, ceil_div_i(6 * kGrpSMs, chunks)) * n_slices * T * r_max * 4 + 256;
}

inline bool grouped_supported(const GroupedProblem& b, const char** why) {
  const char* dummy;
  if (why == nullptr) why = &dummy;
  if (b.dtype != B200_LORA_BF16 && b.dtype != B200_LORA_F16) { *why = "bf16 / fp16 only"; return false; }
  if (b.r_max != 16 && b.r_max != 32 && b.r_max != 64) { *why = "r_max must be 16, 32 or 64"; return false; }
  if (b.sorted_idx == nullptr || b.slot_ids == nullptr || b.counts == nullptr || b.offsets == nullptr || b.n_buckets < 1) {
    *why = "needs the bucket arrays";
    return false;
  }
  if (b.n_buckets > kGrpMaxBuckets || b.n_buckets + b.T / kGrpTok > kGrpMaxChunks || b.T > 65535 * kGrpTok / 2) {
    *why = "too many buckets or rows";
    return false;
  }
  if (b.in_dim % 8 != 0 || b.x_ld % 8 != 0 || !aligned16(b.x)) { *why = "x rows must be 16-byte pieces"; return false; }
  if (b.y_ld % 8 != 0 || !aligned16(b.y)) { *why = "y rows must be 16-byte aligned"; return false; }
  bool any = false;
  for (int s = 0; s < b.st.n; ++s) {
    if (b.st.out[s] == 0) continue;
    any = true;
    if (b.st.out[s] % 8 != 0 || b.st.col[s] % 8 != 0) { *why = "slice widths / offsets must be multiples of 8"; return false; }
    if (!aligned16(b.st.a[s]) || !aligned16(b.st.b[s])) { *why = "slabs must be 16-byte aligned"; return false; }
  }
  if (!any) { *why = "no active slice"; return false; }
  return true;
}

// Chunks expected to be in use: graph buffers carry one bucket per slot, with T rows dealt over nb of them about
// nb * (1 - exp(-T / nb)) hold rows.
inline int grouped_expected_chunks(const GroupedProblem& b) {
  const double nb = (double)b.n_buckets;
  const double in_use = nb * (1.0 - std::exp(-(double)b.T / nb));
  return std::max(1, (int)(in_use + 0.5) + b.T / kGrpTok);
}

// Whether these kernels are the faster ones for a batch that the fused decode kernel takes too: one slice at rank 64 with
// input rows at least as long as its output (o and down) and large adapters, enough of them in use. There the fused kernel has
// only 64 stacked rank rows to deal over a cluster and a long row of each to walk. With several slices its single launch is
// the better choice: it loses up to 20 % where the second wave of its clusters holds few (75 to 110 adapters of even
// popularity), and gains up to 45 % on skewed popularity, which the host does not see. us per projection, fused / these, for even and
// for skewed (Zipf 1.1) popularity, bf16, rank 64, at the expected MB of adapters in use:
//   14336 -> 4096: 95 35 / 30 and 32 / 27, 164 39 / 38 and 35 / 42, 222 70 / 50 and 66 / 47, 393 103 / 73 and 72 / 62, 681 168 /
//   114 and 105 / 78. 7168 -> 4096: 113 42 / 33 and 25 / 34, 120 44 / 34 and 41 / 36, 166 46 / 41 and 44 / 43.
//   6144 -> 2048: 106 30 / 32 and 29 / 27, 134 33 / 40 and 32 / 48, 174 54 / 40 and 31 / 37, 203 57 / 45 and 54 / 45, 303 62 / 60
//   and 55 / 45. 4096 -> 4096: 134 35 / 40 and 33 / 46, 174 56 / 42 and 32 / 39, 303 64 / 61 and 57 / 48.
//   2048 -> 2048 (0.5 MB an adapter): 151 28 / 39 and 24 / 33.
//   Three slices, 4096 -> 6144: 184 50 / 45 and 29 / 53, 222 54 / 49 and 53 / 52, 296 58 / 61 and 56 / 59, 393 81 / 78 and 57 / 78.
//   Two, 4096 -> 28672: 369 88 / 77 and 51 / 82, 445 96 / 90 and 94 / 91, 593 104 / 115 and 99 / 124, 785 147 / 139 and 100 / 121.
//   Rank 32, 14336 -> 4096: 111 33 / 41 and 33 / 35, 229 51 / 67 and 50 / 55, 352 82 / 98 and 73 / 97.
inline bool grouped_preferred(const GroupedProblem& b) {
  int64_t bytes = 0, out = 0;
  int n = 0;
  for (int s = 0; s < b.st.n; ++s)
    if (b.st.out[s] > 0) { bytes += 2 * (int64_t)b.r_max * ((int64_t)b.in_dim + b.st.out[s]); out += b.st.out[s]; ++n; }
  if (n != 1 || b.r_max != 64 || b.in_dim < out || bytes < 1000 * 1000) return false;
  const double nb = (double)b.n_buckets, in_use = nb * (1.0 - std::exp(-(double)b.T / nb));
  return in_use * bytes >= (bytes >= 1400 * 1000 ? 85e6 : 170e6);
}

// Shared memory of one CTA. Small batches: half an SM, so that the CTA of the next launch is resident beside the one that
// runs. Batches that stream many bytes per SM: nearly all of it, which keeps twice the bytes in flight (HBM at 6.5 TB/s is
// 44 GB/s per SM, a round trip under load about 1.5 us).
constexpr int kGrpRingSmall = 84 * 1024, kGrpRingLarge = 196 * 1024;
inline int grouped_ring_bytes(const GroupedProblem& b) {
  int64_t bytes = 0;
  for (int s = 0; s < b.st.n; ++s)
    if (b.st.out[s] > 0) bytes += 2 * (int64_t)b.r_max * std::max(b.in_dim, b.st.out[s]);
  return grouped_expected_chunks(b) * bytes > (int64_t)kGrpSMs * 256 * 1024 ? kGrpRingLarge : kGrpRingSmall;
}

inline GroupedArgs grouped_args(const GroupedProblem& b, SliceTable* active) {
  GroupedArgs a = {};
  a.y = static_cast<uint8_t*>(b.y); a.y_ld = b.y_ld;
  a.T = b.T; a.in_dim = b.in_dim; a.S = b.S; a.r = b.r_max;
  active->n = 0;
  for (int s = 0; s < b.st.n; ++s) {
    if (b.st.out[s] == 0) continue;
    active->a[a.n] = b.st.a[s]; active->b[a.n] = b.st.b[s];
    a.out[a.n] = b.st.out[s]; a.col[a.n] = b.st.col[s];
    ++a.n;
  }
  active->n = a.n;
  a.sorted_idx = b.sorted_idx; a.slot_ids = b.slot_ids; a.counts = b.counts; a.offsets = b.offsets;
  a.rank_per_slot = b.rank_per_slot; a.scale_per_slot = b.scale_per_slot;
  a.n_buckets = b.n_buckets; a.scaling = b.scaling;
  a.f16 = b.dtype == B200_LORA_F16;
  return a;
}

template <typename Kernel>
inline int grouped_launch(Kernel kernel, const char* name, int grid, int threads, size_t smem, const GroupedMaps& maps,
                          const GroupedArgs& a, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid, 1, 1);
  cfg.blockDim = dim3((unsigned)threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = bgmv_options().pdl ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, maps, a);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(B200_LORA_ECUDA, "%s launch: %s", name, cudaGetErrorString(e));
  }
  return B200_LORA_OK;
}

inline int grouped_set_smem(const void* kernel, int bytes) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  return e == cudaSuccess ? B200_LORA_OK : fail(B200_LORA_ECUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
}
inline int grouped_configure() {
  static thread_local int configured_device = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured_device == dev) return B200_LORA_OK;
  if (int rc = grouped_set_smem(reinterpret_cast<const void*>(grouped_shrink_kernel), kGrpRingLarge + 1024)) return rc;
  if (int rc = grouped_set_smem(reinterpret_cast<const void*>(grouped_expand_kernel), kGrpRingLarge + 1024)) return rc;
  configured_device = dev;
  return B200_LORA_OK;
}

// tmp = scaling * x . A^T as up to *parts fp32 partial sums (the number is written back)
inline int grouped_shrink_launch(const GroupedProblem& b, float* tmp, int* parts, cudaStream_t stream) {
  SliceTable st;
  GroupedArgs a = grouped_args(b, &st);
  GroupedMaps maps;
  a.tmp = tmp;
  a.spg = std::min(a.n, kGrpRows / a.r);
  a.m_groups = ceil_div_i(a.n, a.spg);
  a.k_part = round_up_i(ceil_div_i(b.in_dim, *parts), kGrpBK);
  // Stages of up to 32 KB of lora_A (each row piece of 128 .. 512 bytes; wider pieces read DRAM better: 70 us with one panel,
  // 54 with two for 176 MB of rank-64 qkv adapters), but at least four of them.
  const int ring = grouped_ring_bytes(b) - kGrpRows * kGrpBK * 2, panel_w = a.spg * a.r * kGrpBK * 2, panel_x = kGrpTok * kGrpBK * 2;
  a.panels = std::max(1, std::min(std::min(4, 32 * 1024 / panel_w), a.k_part / kGrpBK));
  while (a.panels > 1 && ring / (a.panels * (panel_w + panel_x)) < 4) --a.panels;
  a.k_part = round_up_i(a.k_part, a.panels * kGrpBK);
  *parts = a.parts = ceil_div_i(b.in_dim, a.k_part);
  if (int rc = grouped_configure()) return rc;
  a.whole_stage = a.spg == 1 && b.in_dim % kGrpBK == 0;
  for (int s = 0; s < B200_LORA_MAX_SLICES; ++s) {
    if (s >= a.n) { maps.w[s] = maps.w[0]; continue; }
    if (a.whole_stage) {
      if (int rc = make_tmap_panels(&maps.w[s], st.a[s], (uint64_t)b.S * b.r_max, (uint64_t)b.in_dim, (uint32_t)b.r_max, (uint32_t)a.panels)) return rc;
    } else if (int rc = make_tmap_2d(&maps.w[s], st.a[s], (uint64_t)b.S * b.r_max, (uint64_t)b.in_dim, (uint64_t)b.in_dim, (uint32_t)b.r_max, kGrpBK)) return rc;
  }
  if (int rc = make_tmap_rows(&maps.x, b.x, (uint64_t)b.T, (uint64_t)b.in_dim, (uint64_t)b.x_ld)) return rc;
  // (the last panel's operand tile is 128 rows high whatever the rank: it may reach beyond the ring's lora_A part)
  a.w_bytes = a.panels * panel_w;
  const int stage = a.panels * (panel_w + panel_x);
  a.stages = std::min(kGrpMaxStages, ring / stage);  // (two x warps that take turns: at least two)
  const size_t smem = (size_t)a.stages * stage + kGrpRows * kGrpBK * 2 + 1024;
  return grouped_launch(grouped_shrink_kernel, "grouped_shrink_kernel", kGrpSMs, kGrpShrinkThreads, smem, maps, a, stream);
}

inline int grouped_expand_launch(const GroupedProblem& b, float* tmp, int parts, int round_delta, cudaStream_t stream) {
  SliceTable st;
  GroupedArgs a = grouped_args(b, &st);
  GroupedMaps maps;
  a.tmp = tmp; a.parts = parts; a.round_delta = round_delta;
  if (int rc = grouped_configure()) return rc;
  for (int s = 0; s < B200_LORA_MAX_SLICES; ++s) {
    if (s >= a.n) { maps.w[s] = maps.w[0]; continue; }
    if (int rc = make_tmap_2d(&maps.w[s], st.b[s], (uint64_t)b.S * a.out[s], (uint64_t)b.r_max, (uint64_t)b.r_max, kGrpRows, (uint32_t)b.r_max)) return rc;
  }
  a.tile_cost = a.r == 64 ? 2 : 1;
  const int stage = kGrpRows * a.r * 2, tmp_bytes = 4 * kGrpTok * a.r * 2;
  // an even number: the two MMA warps then always meet the same stages and see every phase of their barriers
  a.stages = std::min(kGrpMaxStages, (grouped_ring_bytes(b) - tmp_bytes) / stage) & ~1;
  const size_t smem = (size_t)a.stages * stage + tmp_bytes + 1024;
  return grouped_launch(grouped_expand_kernel, "grouped_expand_kernel", kGrpSMs, kGrpExpandThreads, smem, maps, a, stream);
}

// K parts of this batch's shrink and the scratch that its partial sums take
inline size_t grouped_need(const GroupedProblem& b, int* parts) {
  int n = 0;
  for (int s = 0; s < b.st.n; ++s) n += b.st.out[s] > 0;
  const int groups = ceil_div_i(n, std::max(1, std::min(n, kGrpRows / b.r_max)));
  *parts = grouped_parts(grouped_expected_chunks(b), groups, b.in_dim);
  return (size_t)*parts * n * b.T * b.r_max * 4 + 256;
}

inline int grouped_add_launch(const GroupedProblem& b, void* workspace, size_t workspace_bytes, int round_delta, cudaStream_t stream) {
  const char* why = nullptr;
  if (!grouped_supported(b, &why)) return fail(B200_LORA_EUNSUPPORTED, "grouped kernels: %s", why);
  int parts;
  const size_t need = grouped_need(b, &parts);  // (256 bytes of it for the alignment)
  if (workspace == nullptr || workspace_bytes < need)
    return fail(B200_LORA_EWORKSPACE, "grouped kernels need %zu bytes of scratch, got %zu", need, workspace_bytes);
  float* const tmp = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(workspace) + 255) & ~(uintptr_t)255);
  if (int rc = grouped_shrink_launch(b, tmp, &parts, stream)) return rc;
  return grouped_expand_launch(b, tmp, parts, round_delta, stream);
}

}  // namespace b200lora
