// Fused linear for large batches: y = x . W^T (+ bias) + LoRA delta with CTA pairs (tcgen05 cta_group::2).
//
// What bounds it: a 128 x 256 tile per CTA (tc_tile_kernel) takes 48 KB from the L2 for 512 cycles of MMA, 94 bytes per cycle
// and SM. Here two CTAs share a 256 x 256 tile: each loads its own 128 rows of x and HALF of the weight tile (32 KB for the
// same 512 cycles), the pair's MMA reads the other half from the peer's shared memory. Everything else is as in
// tc_tile_kernel: persistent CTAs over equal contiguous ranges of tiles, two accumulators of 256 TMEM columns, LoRA steps
// (masked rows of tmp, lora_B tile) behind the K loop of a tile, output through swizzled shared memory and TMA stores.
// 8172 rows, without adapters, us, tile / pair kernel / cuBLAS: 2048 -> 12288 302 / 281 / 264 (all zeros: 262 / 225 / 222, the
// power cap is the difference), 6144 -> 2048 155 / 147 / 127; with rank-32 adapters 316 / 294 and 156 / 153.
//
// The LoRA operands have buffers of their own, filled by a warp of its own while the K loop runs: in the stages of the K loop, 1 us
// ahead of the MMAs, every tile waited for them (2048 -> 12288 of 8172 rows, rank 32: 361 us against 281 without adapters). The MMA
// of a run of equal slots updates the rows of that run only (its lane mask).
//
// Eight epilogue warps in two sets, each with an output buffer: with four, an epilogue was longer than the K loop of the tile behind
// it from 1024 columns of x down (SiLU form, 4001 rows, 1024 -> 2 x 4096, rank 32: 68 us with four, 56 with eight and the steps below).
//
// Who waits for whom: all loads, by both CTAs, count on barriers of the LEADER (rank 0 issues all MMAs); commits arrive at the empty,
// lora_empty and acc_full barriers of both CTAs.
#pragma once

#include "prefill_cluster.cuh"

namespace b200lora {

constexpr int kPairThreads = 352;  // warp 0 TMA, warp 1 MMA (rank 0) + TMEM, warps 2-9 epilogue, warp 10 LoRA loads
constexpr int kPairMaxStages = 5;
constexpr int kPairStageBytes = 2 * kSgmvBM * kSgmvBK * 2;  // 32 KB: 128 rows of x, 128 rows of W
constexpr int kPairOutBufs = 2;                             // one of each epilogue set
constexpr int kPairMaxLoraBufs = 4;
constexpr int kPairMaxSeg = 2;                              // 256-row blocks that a pair's tile range may touch
constexpr int kPairRuns = 2 * kSgmvBM;
constexpr int kPairRunBytes = kPairRuns * 4;                // slot (int16), first and last row of the 256 (uint8 each)
// Dynamic shared memory: ring, LoRA buffers, output buffers, run tables; 1 KB of the 227 is left to static shared memory.
constexpr int kPairFixed = kPairOutBufs * kGemmOutBufBytes + kPairMaxSeg * kPairRunBytes;
__host__ __device__ constexpr int pair_lora_bytes(int r) { return 2 * kSgmvBM * r * 2; }  // tmp tile and half a lora_B tile
__host__ __device__ constexpr int pair_lora_bufs(int r) { return r > 32 ? 2 : 4; }
__host__ __device__ constexpr int pair_stages(int r) {
  const int fit = (kBgmvSmemMax - 1024 - kPairFixed - pair_lora_bufs(r) * pair_lora_bytes(r)) / kPairStageBytes;
  return fit < kPairMaxStages ? fit : kPairMaxStages;  // 5 at rank 16, else 4
}

// ---- cta_group::2 forms
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_pair_elected(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                                  uint32_t accumulate, uint32_t leader) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\t"
      "mov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %4, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accumulate), "r"(leader)
      : "memory");
}
// the same, updating only the rows of D whose bit in `off` is clear (rows 0 - 127 in the leader's tensor memory, 128 - 255 in the peer's)
__device__ __forceinline__ void umma_pair_rows_elected(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                                       uint32_t leader, const uint32_t (&off)[8]) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\t"
      "mov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
      "setp.eq.b32 p, 0, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %4, {%6, %7, %8, %9, %10, %11, %12, %13}, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(leader), "r"(off[0]), "r"(off[1]), "r"(off[2]), "r"(off[3]), "r"(off[4]),
      "r"(off[5]), "r"(off[6]), "r"(off[7])
      : "memory");
}
// one arrival at the barrier of this offset in both CTAs of the pair
__device__ __forceinline__ void umma_commit_pair_elected(uint32_t bar, uint32_t leader) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %2;\n\t}"
      ::"r"(bar), "r"(leader), "h"((uint16_t)3)
      : "memory");
}
// into this CTA's shared memory; the bytes count on `bar`, a barrier of either CTA of the pair (address from mapa_shared)
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst_smem, const CUtensorMap* tmap, int c0, int c1, uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;"
      ::"r"(dst_smem), "l"(tmap), "r"(c0), "r"(c1), "r"(bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ uint64_t l2_policy_evict_normal() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// Runs of equal slot inside the two 128-row blocks blk and blk + 1 (as sgmv_find_runs, by the 128 threads of the epilogue warps)
__device__ __forceinline__ void pair_find_runs(const int32_t* tts, int T, int S, int blk, int i, int16_t* s_slot, int16_t* run_slot, uint8_t* run_lo,
                                               uint8_t* run_hi, int* nruns) {
  __shared__ int warp_starts[4];
  int got[2];  // both halves' loads at once
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int row = (blk + h) * kSgmvBM + i;
    got[h] = row < T ? tts[row] : -1;
    (void)B200_IN_BOUNDS(got[h] >= -1 && got[h] < S);  // ids outside [-1, S) are treated as "no adapter"; the checked build reports them
    if (got[h] >= S || got[h] < -1) got[h] = -1;
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    s_slot[i] = (int16_t)got[h];
    named_bar_sync(2, 128);
    const bool starts = got[h] >= 0 && (i == 0 || s_slot[i - 1] != got[h]), ends = got[h] >= 0 && (i == kSgmvBM - 1 || s_slot[i + 1] != got[h]);
    const unsigned mask = __ballot_sync(0xffffffffu, starts);
    unsigned before = __popc(mask & ((2u << (i & 31)) - 1u));  // runs of this warp that start at or before this row
    if ((i & 31) == 0) warp_starts[i >> 5] = __popc(mask);
    named_bar_sync(2, 128);
    for (int w = 0; w < i >> 5; ++w) before += (unsigned)warp_starts[w];
    if (starts) { run_slot[h * kSgmvBM + before - 1] = (int16_t)got[h]; run_lo[h * kSgmvBM + before - 1] = (uint8_t)i; }
    if (ends) run_hi[h * kSgmvBM + before - 1] = (uint8_t)(i + 1);
    if (i == 0) nruns[h] = warp_starts[0] + warp_starts[1] + warp_starts[2] + warp_starts[3];
    named_bar_sync(2, 128);
  }
}

struct PairMaps {
  CUtensorMap x;                        // [T, in]         box 128 x 64
  CUtensorMap w;                        // [n_total, in]   box 128 x 64
  CUtensorMap t;                        // [n*T(+128), r]  box 128 x r
  CUtensorMap b[B200_LORA_MAX_SLICES];  // [S*out_s, r]    box 128 x r
  CUtensorMap y;                        // [T, n_total]    box 128 x 64 (store)
};

// kSilu: y [T, I] = silu(gate) * up of a projection [gate | up] of 2 I rows of W. The pair's tile is 128 columns of gate (the
// weight rows of rank 0) and the 128 columns of up that go with them (rank 1), so both halves of a product meet in one CTA's
// epilogue, in fp32; neither the projection's output nor a pass over it is left (4001 x 2 x 4096: 130 MB, 21 us of its own).
template <bool kSilu>
__global__ void __launch_bounds__(kPairThreads, 1)
linear_pair_kernel(const __grid_constant__ PairMaps maps, const __grid_constant__ GemmArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ int f_n[2], seg_nruns[kPairMaxSeg];
  __shared__ __align__(8) uint64_t bars[2 * kPairMaxStages + 2 * kPairMaxLoraBufs + 5];
  __shared__ uint4 jobs[kPairMaxLoraBufs][3];  // column of D and instruction descriptor, then the lane mask, of the step in a buffer
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_flag;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = a.r_max, n = a.n, rank = (int)cluster_ctarank();
  constexpr int kCols = kSilu ? kSgmvBN / 2 : kSgmvBN, kHalves = kSilu ? 2 : 1;  // columns of y a tile covers; column ranges of W
  const int ntile_all = (a.n_total + kCols - 1) / kCols, nblk_all = (a.T + 2 * kSgmvBM - 1) / (2 * kSgmvBM);
  const int total_tiles = nblk_all * ntile_all, pairs = (int)gridDim.x >> 1, pair = (int)blockIdx.x >> 1;
  const int per_pair = (total_tiles + pairs - 1) / pairs;
  const int t_begin = min(pair * per_pair, total_tiles), t_end = min(t_begin + per_pair, total_tiles);
  const int blk_first = t_begin / ntile_all;
  const int nseg = t_end > t_begin ? (t_end - 1) / ntile_all - blk_first + 1 : 0;  // <= kPairMaxSeg (host)
  const uint32_t smem_base = smem_u32(smem);  // 1024-byte aligned by the declaration: static shared memory is padded to it
  const int NS = pair_stages(r), LB = pair_lora_bufs(r);
  const uint32_t lora_bytes = (uint32_t)pair_lora_bytes(r), lora_base = smem_base + (uint32_t)(NS * kPairStageBytes);
  const uint32_t out_base = lora_base + (uint32_t)LB * lora_bytes;
  uint8_t* const out_ptr = smem + NS * kPairStageBytes + LB * lora_bytes;
  uint8_t* const tables = out_ptr + kPairOutBufs * kGemmOutBufBytes;
  // (while the tables are made, in the output buffers)
  int16_t* const f_slot = reinterpret_cast<int16_t*>(out_ptr);
  auto f_run = [&](int h) { return f_slot + (1 + h) * kSgmvBM; };
  auto f_lo = [&](int h) { return out_ptr + (6 + h) * kSgmvBM; };
  auto f_hi = [&](int h) { return out_ptr + (8 + h) * kSgmvBM; };
  auto run_slot = [&](int sg) { return reinterpret_cast<int16_t*>(tables + sg * kPairRunBytes); };
  auto run_lo = [&](int sg) { return tables + sg * kPairRunBytes + 2 * kPairRuns; };
  auto run_last = [&](int sg) { return tables + sg * kPairRunBytes + 3 * kPairRuns; };
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * (uint32_t)s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (uint32_t)(kPairMaxStages + s); };
  auto lora_bar = [&](int b) { return bar0 + 8u * (uint32_t)(2 * kPairMaxStages + b); };
  auto lora_empty = [&](int b) { return bar0 + 8u * (uint32_t)(2 * kPairMaxStages + kPairMaxLoraBufs + b); };
  auto acc_full = [&](int b) { return bar0 + 8u * (uint32_t)(2 * kPairMaxStages + 2 * kPairMaxLoraBufs + b); };
  auto acc_empty = [&](int b) { return bar0 + 8u * (uint32_t)(2 * kPairMaxStages + 2 * kPairMaxLoraBufs + 2 + b); };
  constexpr int tmem_cols = 2 * kSgmvBN;
  const uint32_t tables_bar = acc_empty(2);
  const bool aligned = (smem_base & 1023u) == 0;  // (the same in both CTAs)

  if (tid == 0) {
    for (int s = 0; s < kPairMaxStages; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int b = 0; b < kPairMaxLoraBufs; ++b) {
      mbar_init(lora_bar(b), 1);
      mbar_init(lora_empty(b), 1);
    }
    for (int b = 0; b < 2; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 16); }  // eight epilogue warps of each CTA
    mbar_init(tables_bar, 128);
    abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(&tmem_base_s), (uint32_t)tmem_cols);
    tc_fence_before_sync();
  }
  __syncthreads();
  cluster_arrive();
  cluster_wait();  // barriers and tensor memory of both CTAs are ready
  griddep_launch_dependents();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  const int nk = a.in_dim / kSgmvBK;
  auto seg_range = [&](int sg, int& blk, int& ja, int& jb) {
    blk = blk_first + sg;
    ja = max(t_begin - blk * ntile_all, 0);
    jb = min(t_end - blk * ntile_all, ntile_all);
  };
  // Piece q of tile j: the columns [lo, hi) of W that slice s = q / kHalves covers in range q % kHalves, and where D has them
  const int n_pieces = n * kHalves;
  auto piece = [&](int q, int j, int& s, int& lo, int& hi, int& d) {
    s = q / kHalves;
    const int h = q % kHalves, base = h * a.n_total + j * kCols;
    lo = max(a.col[s], base);
    hi = min(a.col[s] + a.out[s], base + kCols);
    d = h * kCols + lo - base;
    return lo < hi;
  };
  const int row_bytes = r * 2;
  const uint32_t t_tile_bytes = (uint32_t)kSgmvBM * r * 2;

  if (!aligned) {
    if (tid == 0) atomicOr(&g_b200_status, kStatusBadSmemBase);
  } else if (warp == 0) {
    // ---- loads: this CTA's rows of x and tmp, this CTA's half of the W and lora_B tiles
    const uint32_t leader = elect_one();
    if (leader) { tma_prefetch_desc(&maps.x); tma_prefetch_desc(&maps.w); tma_prefetch_desc(&maps.t); tma_prefetch_desc(&maps.y); }
    const uint64_t w_policy = l2_policy_evict_last(), x_policy = l2_policy_evict_normal();
    const uint32_t full0 = mapa_shared(full_bar(0), 0);  // the leader's
    int st = 0, round = 0;
    if (!a.after_shrink) griddep_wait();
    for (int sg = 0; sg < nseg; ++sg) {
      int blk, ja, jb;
      seg_range(sg, blk, ja, jb);
      ja = uniform(ja); jb = uniform(jb);
      const int row0 = (2 * blk + rank) * kSgmvBM;
      for (int j = ja; j < jb; ++j) {
        for (int kc = 0; kc < nk; ++kc) {
          if (round > 0) mbar_wait_bounded(empty_bar(st), (uint32_t)((round & 1) ^ 1), &abort_flag);
          if (leader) {
            const uint32_t base = smem_base + (uint32_t)st * kPairStageBytes, bar = full0 + 8u * (uint32_t)st;
            if (rank == 0) mbar_arrive_expect_tx(full_bar(st), 2 * kPairStageBytes);  // both CTAs' loads
            tma_load_2d_pair(base, &maps.x, kc * kSgmvBK, row0, bar, x_policy);
            tma_load_2d_pair(base + kPairStageBytes / 2, &maps.w, kc * kSgmvBK, j * kCols + rank * (kSilu ? a.n_total : kSgmvBM), bar, w_policy);
          }
          __syncwarp();
          if (++st == NS) { st = 0; ++round; }
        }
      }
    }
  } else if (warp == 10) {
    // ---- LoRA loads: this CTA's rows of tmp and half of the lora_B tile
    const uint32_t leader = elect_one(), lora0 = mapa_shared(lora_bar(0), 0);
    const uint64_t policy = l2_policy_evict_normal();
    if (a.lora) {
      mbar_wait_bounded(tables_bar, 0u, &abort_flag);
      griddep_wait();  // tmp is final from here on
    }
    int b = 0, round = 0;
    for (int sg = 0; sg < nseg; ++sg) {
      int blk, ja, jb;
      seg_range(sg, blk, ja, jb);
      const int row0 = (2 * blk + rank) * kSgmvBM, nruns = a.lora ? seg_nruns[sg] : 0;
      for (int j = ja; j < jb; ++j)
        for (int u = 0; u < nruns; ++u) {
          const int slot = uniform(run_slot(sg)[u]);
          // What the MMA warp needs is put beside the operands here, well ahead: between two K loops 30 instructions of one warp
          // for each run and piece were 0.5 us of an idle tensor pipe.
          const int lo_row = run_lo(sg)[u], hi_row = run_last(sg)[u] + 1;
          uint32_t off[8];
#pragma unroll
          for (int w = 0; w < 8; ++w) off[w] = rows_outside(lo_row, hi_row, w);
          for (int q = 0; q < n_pieces; ++q) {
            int s, lo, hi, d;
            if (!piece(q, j, s, lo, hi, d)) continue;
            if (round > 0) mbar_wait_bounded(lora_empty(b), (uint32_t)((round & 1) ^ 1), &abort_flag);
            if (leader) {
              const uint32_t base = lora_base + (uint32_t)b * lora_bytes, bar = lora0 + 8u * (uint32_t)b;
              if (rank == 0) {
                jobs[b][0] = make_uint4((uint32_t)d, umma_idesc_bf16(2 * kSgmvBM, hi - lo), 0u, 0u);  // (a multiple of 32: see the launch)
                jobs[b][1] = make_uint4(off[0], off[1], off[2], off[3]);
                jobs[b][2] = make_uint4(off[4], off[5], off[6], off[7]);
                mbar_arrive_expect_tx(lora_bar(b), 2 * lora_bytes);  // both CTAs' loads
              }
              tma_load_2d_pair(base, &maps.t, 0, s * a.T + row0, bar, policy);
              tma_load_2d_pair(base + t_tile_bytes, &maps.b[s], 0, slot * a.out[s] + (lo - a.col[s]) + rank * ((hi - lo) >> 1), bar, policy);
            }
            __syncwarp();
            if (++b == LB) { b = 0; ++round; }
          }
        }
    }
  } else if (warp == 1 && rank == 0) {
    // ---- MMA for both CTAs
    const uint32_t leader = elect_one();
    const uint64_t desc_x = umma_smem_desc(smem_base, 128), desc_t = umma_smem_desc(lora_base, row_bytes);
    const uint32_t hi_x = (uint32_t)(desc_x >> 32), hi_t = (uint32_t)(desc_t >> 32), lo0 = (uint32_t)desc_x, lt0 = (uint32_t)desc_t;
    const uint32_t idesc_base = umma_idesc_bf16(2 * kSgmvBM, kSgmvBN);
    int st = 0, round = 0, lb = 0, lround = 0, job = 0;
    for (int sg = 0; sg < nseg; ++sg) {
      int blk, ja, jb;
      seg_range(sg, blk, ja, jb);
      ja = uniform(ja); jb = uniform(jb);
      int nruns = 0, steps = 0;  // LoRA steps of a tile
      for (int j = ja; j < jb; ++j, ++job) {
        const int buf = job & 1;
        const uint32_t d_tmem = tmem_base + (uint32_t)(buf * kSgmvBN);
        if (job >= 2) mbar_wait_bounded_acquire_cluster(acc_empty(buf), (uint32_t)(((job >> 1) - 1) & 1), &abort_flag);
        tc_fence_after_sync();
        for (int kc = 0; kc < nk; ++kc) {
          mbar_wait_bounded_acquire_cluster(full_bar(st), (uint32_t)(round & 1), &abort_flag);
          tc_fence_after_sync();
          const uint32_t xl = lo0 + ((uint32_t)st * kPairStageBytes >> 4), wl = xl + (kPairStageBytes / 2 >> 4);
#pragma unroll
          for (int k4 = 0; k4 < kSgmvBK / 16; ++k4)
            umma_pair_elected(d_tmem, xl + 2u * k4, wl + 2u * k4, hi_x, idesc_base, (kc > 0 || k4 > 0) ? 1u : 0u, leader);
          umma_commit_pair_elected(empty_bar(st), leader);
          if (++st == NS) { st = 0; ++round; }
          if (a.lora && kc == min(1, nk - 1)) {  // (while the MMAs of the first steps run)
            if (j == ja) {
              mbar_wait_bounded(tables_bar, 0u, &abort_flag);
              nruns = uniform(seg_nruns[sg]);
            }
            steps = 0;
            for (int q = 0; q < n_pieces; ++q) {
              int s, lo, hi, d;
              steps += piece(q, j, s, lo, hi, d) ? nruns : 0;
            }
          }
        }
        for (int k = 0; k < steps; ++k) {
          mbar_wait_bounded_acquire_cluster(lora_bar(lb), (uint32_t)(lround & 1), &abort_flag);
          tc_fence_after_sync();
          const uint32_t tl = lt0 + ((uint32_t)lb * lora_bytes >> 4), bl = tl + (t_tile_bytes >> 4);
          const uint4 what = jobs[lb][0], m0 = jobs[lb][1], m1 = jobs[lb][2];
          const uint32_t off[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
          for (int k4 = 0; k4 < 4; ++k4)
            if (16 * k4 < r) umma_pair_rows_elected(d_tmem + what.x, tl + 2u * k4, bl + 2u * k4, hi_t, what.y, leader, off);
          umma_commit_pair_elected(lora_empty(lb), leader);
          if (++lb == LB) { lb = 0; ++lround; }
        }
        umma_commit_pair_elected(acc_full(buf), leader);
      }
    }
  } else if (warp >= 2 && warp <= 9) {
    // ---- epilogue: thread <-> row of this CTA's half; the two sets take the 64-column chunks of a tile in turn
    const int quarter = warp & 3, row_in_blk = quarter * 32 + lane, set = (warp - 2) >> 2, etid = tid - 64 - 128 * set;
    const uint32_t acc_empty0 = mapa_shared(acc_empty(0), 0);
    int job = 0;
    if (a.lora && set == 0) {
      // Runs of equal slot of every block, first half then second, a run over the middle once. Made while the first K loop runs.
      for (int sg = 0; sg < nseg; ++sg) {
        pair_find_runs(a.token_to_slot, a.T, a.S, 2 * (blk_first + sg), etid, f_slot, f_run(0), f_lo(0), f_hi(0), f_n);
        const int n0 = f_n[0], n1 = f_n[1];
        const int joint = n0 > 0 && n1 > 0 && f_hi(0)[n0 - 1] == kSgmvBM && f_lo(1)[0] == 0 && f_run(0)[n0 - 1] == f_run(1)[0] ? 1 : 0;
        const int total = n0 + n1 - joint;
        for (int i = etid; i < total; i += 128) {
          const int k0 = i < n0 ? i : -1, k1 = i >= n0 - joint ? i - n0 + joint : -1;  // entry of the first / second half's list
          run_slot(sg)[i] = k0 >= 0 ? f_run(0)[k0] : f_run(1)[k1];
          run_lo(sg)[i] = (uint8_t)(k0 >= 0 ? f_lo(0)[k0] : kSgmvBM + f_lo(1)[k1]);
          run_last(sg)[i] = (uint8_t)((k1 >= 0 ? kSgmvBM + f_hi(1)[k1] : f_hi(0)[k0]) - 1);
        }
        if (etid == 0) seg_nruns[sg] = total;
        named_bar_sync(2, 128);
      }
      mbar_arrive(tables_bar);
    }
    for (int sg = 0; sg < nseg; ++sg) {
      int blk, ja, jb;
      seg_range(sg, blk, ja, jb);
      const int row0 = (2 * blk + rank) * kSgmvBM;
      for (int j = ja; j < jb; ++j, ++job) {
        const int buf = job & 1;
        mbar_wait_bounded_acquire_cluster(acc_full(buf), (uint32_t)((job >> 1) & 1), &abort_flag);
        tc_fence_after_sync();
        for (int c = kGemmOutChunk * set; c < kCols; c += 2 * kGemmOutChunk) {
          const int col0 = j * kCols + c;
          if (col0 >= a.n_total || row0 >= a.T) break;  // uniform over the set
          const uint32_t obuf = out_base + (uint32_t)set * kGemmOutBufBytes;
          if (etid == 0) bulk_wait_group_read<0>();  // the store that last used this buffer has read it
          named_bar_sync(3 + (uint32_t)set, 128);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t v[32];
            const uint32_t at = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * kSgmvBN + c + 32 * h);
            tmem_ld_32x32(at, v);
            if constexpr (kSilu) {
              uint32_t up[32];
              tmem_ld_32x32(at + (uint32_t)kCols, up);
              tmem_ld_wait();
#pragma unroll
              for (int q = 0; q < 32; ++q) {
                const float g = __uint_as_float(v[q]);
                // (__fdividef, good to 2 ulp: with the correctly rounded division and its branch the elements of a thread took
                // turns, 390 cycles each, and the kernel 189 us instead of the projection's 64)
                v[q] = __float_as_uint(__fdividef(g, 1.f + expf(-g)) * __uint_as_float(up[q]));
              }
            } else {
              tmem_ld_wait();
              if (a.bias != nullptr) {
#pragma unroll
                for (int q = 0; q < 32; ++q) {
                  const int cc = col0 + 32 * h + q;
                  const float bv = cc < a.n_total ? __bfloat162float(a.bias[cc]) : 0.f;
                  v[q] = __float_as_uint(__uint_as_float(v[q]) + bv);
                }
              }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint4 o;
              o.x = pack_bf16x2(__uint_as_float(v[8 * q + 0]), __uint_as_float(v[8 * q + 1]));
              o.y = pack_bf16x2(__uint_as_float(v[8 * q + 2]), __uint_as_float(v[8 * q + 3]));
              o.z = pack_bf16x2(__uint_as_float(v[8 * q + 4]), __uint_as_float(v[8 * q + 5]));
              o.w = pack_bf16x2(__uint_as_float(v[8 * q + 6]), __uint_as_float(v[8 * q + 7]));
              const uint32_t chunk16 = (uint32_t)(4 * h + q) ^ (uint32_t)(row_in_blk & 7);  // the store box's 128-byte swizzle
              asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(obuf + (uint32_t)row_in_blk * 128u + chunk16 * 16u),
                           "r"(o.x), "r"(o.y), "r"(o.z), "r"(o.w)
                           : "memory");
            }
          }
          fence_proxy_async_smem();
          named_bar_sync(3 + (uint32_t)set, 128);
          if (etid == 0) {
            tma_store_2d_hint(&maps.y, obuf, col0, row0, l2_policy_evict_first());
            bulk_commit_group();
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote_release(acc_empty0 + 8u * (uint32_t)buf);
      }
    }
    if (etid == 0) bulk_wait_group_read<0>();
  }
  __syncthreads();
  cluster_arrive();
  cluster_wait();  // no CTA leaves while the pair's MMA, commits or arrivals may still reach its memory
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, (uint32_t)tmem_cols);
  }
  if (tid == 0 && abort_flag != 0) atomicOr(&g_b200_status, kStatusWaitGaveUp);
}

// ------------------------------------------------------------------ host side
// LoRA stages are MMAs over a column range of which each CTA holds one half: a multiple of 32 columns.
inline bool linear_pair_lora_ok(const SliceTable& st) {
  for (int s = 0; s < st.n; ++s)
    if (st.out[s] > 0 && (st.col[s] % 32 != 0 || st.out[s] % 32 != 0)) return false;
  return true;
}

// n_total: columns of y. silu: W has 2 n_total rows.
inline int linear_pair_launch(const SgmvMaps& sm, const SgmvArgs& sa, const void* const* slab_b, const void* weight, int64_t w_ld, int n_total,
                              const void* bias, bool lora, bool silu, cudaStream_t stream) {
  PairMaps maps;
  GemmArgs a = {};
  a.T = sa.T; a.in_dim = sa.in_dim; a.n_total = n_total; a.bias = static_cast<const __nv_bfloat16*>(bias);
  a.S = sa.S; a.r_max = sa.r_max; a.n = sa.n;
  for (int s = 0; s < B200_LORA_MAX_SLICES; ++s) { a.out[s] = sa.out[s]; a.col[s] = sa.col[s]; }
  a.token_to_slot = sa.token_to_slot;
  a.lora = a.after_shrink = lora ? 1 : 0;
  if (a.S > 32767) return fail(B200_LORA_EUNSUPPORTED, "fused linear: more than 32767 adapter slots");
  maps.x = sm.x;
  maps.t = sm.t;
  if (int rc = make_tmap_2d(&maps.w, weight, (uint64_t)n_total * (silu ? 2 : 1), (uint64_t)sa.in_dim, (uint64_t)w_ld, kSgmvBM, kSgmvBK)) return rc;
  if (int rc = make_tmap_2d(&maps.y, sa.y, (uint64_t)sa.T, (uint64_t)n_total, (uint64_t)sa.y_ld, kSgmvBM, kGemmOutChunk)) return rc;
  for (int s = 0; s < B200_LORA_MAX_SLICES; ++s) maps.b[s] = maps.w;
  for (int s = 0; lora && s < sa.n; ++s)
    if (int rc = make_tmap_2d(&maps.b[s], slab_b[s], (uint64_t)sa.S * sa.out[s], (uint64_t)sa.r_max, (uint64_t)sa.r_max, kSgmvBM, (uint32_t)sa.r_max)) return rc;
  const int cols = silu ? kSgmvBN / 2 : kSgmvBN;
  const int ntile = (n_total + cols - 1) / cols, total = (sa.T + 2 * kSgmvBM - 1) / (2 * kSgmvBM) * ntile;
  int pairs = std::min(kTileSMs / 2, total);
  const int max_per = (kPairMaxSeg - 1) * ntile;  // a range of that many tiles touches at most kPairMaxSeg blocks
  if ((total + pairs - 1) / pairs > max_per) pairs = (total + max_per - 1) / max_per;
  const int smem = pair_stages(sa.r_max) * kPairStageBytes + pair_lora_bufs(sa.r_max) * pair_lora_bytes(sa.r_max) + kPairFixed;
  if (int rc = sgmv_set_smem(reinterpret_cast<const void*>(silu ? linear_pair_kernel<true> : linear_pair_kernel<false>), smem)) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * pairs), 1, 1);
  cfg.blockDim = dim3(kPairThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = bgmv_options().pdl ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, silu ? linear_pair_kernel<true> : linear_pair_kernel<false>, maps, a);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(B200_LORA_ECUDA, "linear_pair_kernel launch: %s", cudaGetErrorString(e));
  }
  return B200_LORA_OK;
}

// Pair tiles (256 x 256) from which the pair kernel takes a projection; with fewer, the 74 pairs are filled unevenly and
// tc_tile_kernel's 128 x 256 tiles are as fast. us, pair / tile kernel, rank 32: 2048 -> 2048, 3000 rows (96 tiles) 32.7 / 35.3;
// 2048 -> 2560, 2000 rows (80) 38.9 / 38.4; 1024 -> 1024, 4001 rows (64) 20.4 / 18.9; 1024 -> 8192, 4001 rows (512) 53.9 / 60.9.
constexpr int64_t kPairMinTiles = 96;
struct LinearProblem {
  SgmvProblem lora;          // y, x, slabs, token_to_slot (null token_to_slot or no slice: plain linear)
  const void* weight; int64_t w_ld; int n_total; const void* bias;
  bool silu = false;         // y = silu(gate) * up of the projection's halves, [T, n_total / 2]
};

// Whether prefill_cluster_kernel takes a fused linear (and its plan): where its expected time is less than that of the shrink launch and
// the kernel behind it, the latter a regression over 149 measured points that it meets within 9 %: launches and tile rounds, K steps of
// the pair or the tile kernel with few and with all SMs busy, of the shrink. Over 156 points (12 projections, 64 to 4500 rows of up to eight
// prompts) the choice of kernel and split loses 2.1 % to the best, the tiles alone, without groups of columns, 12. us, the others / this: 2048 ->
// 2560, rank 64, 64, 300 rows 18.7 / 12.9, 19.6 / 17.7; 6144 -> 2048 64, 300 and 600 rows 40 / 27, 40 / 32, 40 / 36; 1024 -> 8192, rank 32, 64, 300,
// 1000 rows 13.3 / 10.0, 15.5 / 13.2, 24.8 / 21.9. The others keep 2048 -> 12288, rank 64 (of 2000 rows 89 / 117) and 6144 -> 2048 from 1000 rows on.
// And, as the sums put the two too close to each other (this kernel up to 20 % too high), for up to 128 rank rows where a CTA of a cluster
// without groups has one tile or, over up to 2048 columns of x, no more tiles than the CTAs of the other two (over 1024 one more). 150 points that
// the sums alone leave to the others, all ranks, the others / this: one tile 4096 -> 1024, 2200 to 3700 rows 34.3 / 31.4, 4096 -> 512, 3200 to 9000
// rows 39.6 / 36.6, 1024 -> 1280, 3200 rows 18.8 / 16.7; two 2048 -> 2048, 2200 to 4200 rows 33.2 / 30.0, 2048 -> 1024, 5000 to 9000 rows 36.1 / 32.6. Two
// tiles over more columns: 4096 -> 4096, 1700 rows 52.7 / 60.7, 4096 -> 2048, 3200 rows 53.8 / 61.4, 4096 -> 1024, 5000 rows 57.7 / 60.6. (A second tile
// has all K steps again, and x with them.) The rule loses 0.2 % to the best of these points; with two tiles over 4096 columns 3.1.
inline bool prefill_cluster_linear_ok(const LinearProblem& p, PcArgs* plan) {
  const SgmvProblem& b = p.lora;
  int n = 0;
  for (int s = 0; s < b.st.n; ++s) {
    if (b.st.out[s] == 0) continue;
    if (b.st.col[s] % 16 != 0 || b.st.out[s] % 16 != 0) return false;  // (the MMAs of a slice would reach into the next one)
    ++n;
  }
  double here;
  if (ceil_div_i(b.T, kSgmvBM) > kTileSMs || !sgmv_supported(b, nullptr) || !prefill_cluster_plan(b, n, p.n_total, true, plan, &here)) return false;
  const int nk = b.in_dim / kSgmvBK, blocks = ceil_div_i(b.T, kSgmvBM), tiles = blocks * ceil_div_i(p.n_total, kSgmvBN);
  const int pair_tiles = ceil_div_i(b.T, 2 * kSgmvBM) * ceil_div_i(p.n_total, kSgmvBN);
  const bool pairs = pair_tiles >= kPairMinTiles;
  const int rounds = pairs ? ceil_div_i(pair_tiles, kTileSMs / 2) : ceil_div_i(tiles, kTileSMs);
  int parts = 1;  // K parts of the shrink
  while (parts < 8 && blocks * parts * 2 <= kTileSMs && ceil_div_i(nk, 2 * parts) * (2 * parts - 1) < nk) parts *= 2;
  const double busy = pairs ? ceil_div_i(pair_tiles, rounds) / (kTileSMs / 2.0) : ceil_div_i(tiles, rounds) / (double)kTileSMs;
  const double others = 7.4 + rounds * (1.25 + nk * (pairs ? 0.243 + 0.146 * busy : 0.223 + 0.262 * busy)) + 0.2 * ceil_div_i(nk, parts) + 0.02 * n * b.r_max;
  int ck = 1;  // the cluster without groups: tiles of its CTAs
  while (ck < 8 && blocks <= clusters_resident(2 * ck) && ceil_div_i(nk, 2 * ck) * (2 * ck - 1) < nk) ck *= 2;
  const int own = ceil_div_i(ceil_div_i(p.n_total, 64 * ck), kSgmvBN / 64);
  return here < 0.95 * others || (n * b.r_max <= 128 && b.in_dim <= (own > 1 ? 2048 : 4096) && ((own <= rounds && own <= 3) || (own <= 2 && (own - rounds) * nk <= 16)));
}

// What a fused linear runs: prefill_cluster_kernel (`plan`), or, behind the shrink if it has a delta, CTA pairs or 128 x 256 tiles.
enum LinearKernel { kLinearCluster = 1, kLinearPairs = 2, kLinearTiles = 3 };
inline LinearKernel linear_kernel(const LinearProblem& p, bool with_lora, PcArgs* plan) {
  if (with_lora && !p.silu && prefill_cluster_linear_ok(p, plan)) return kLinearCluster;
  const int64_t pair_tiles = (int64_t)ceil_div_i(p.lora.T, 2 * kSgmvBM) * ceil_div_i(p.n_total, kSgmvBN);
  return (p.silu || pair_tiles >= kPairMinTiles) && (!with_lora || linear_pair_lora_ok(p.lora.st)) ? kLinearPairs : kLinearTiles;
}

// y = x . W^T (+ bias) + LoRA delta, the delta accumulated into the GEMM's TMEM accumulator.
inline int linear_lora_launch(const LinearProblem& p, void* workspace, size_t workspace_bytes, cudaStream_t stream) {
  const SgmvProblem& b = p.lora;
  if (b.in_dim % kSgmvBK != 0) return fail(B200_LORA_EUNSUPPORTED, "fused linear: in_dim must be a multiple of 64");
  if (p.n_total % 8 != 0 || p.w_ld % 8 != 0 || b.x_ld % 8 != 0 || b.y_ld % 8 != 0)
    return fail(B200_LORA_EUNSUPPORTED, "fused linear: widths and row strides must be multiples of 8");
  if (p.silu && (p.n_total % 64 != 0 || p.bias != nullptr)) return fail(B200_LORA_EUNSUPPORTED, "fused linear with SiLU: width a multiple of 64, no bias");
  if ((reinterpret_cast<uintptr_t>(p.weight) & 15u) || (reinterpret_cast<uintptr_t>(b.x) & 15u) ||
      (reinterpret_cast<uintptr_t>(b.y) & 15u) || (reinterpret_cast<uintptr_t>(p.bias) & 1u))
    return fail(B200_LORA_EUNSUPPORTED, "fused linear: pointers must be 16-byte aligned");
  int slices = 0;
  for (int s = 0; s < b.st.n; ++s) slices += b.st.out[s] > 0;
  const bool with_lora = slices > 0 && b.token_to_slot != nullptr;
  SgmvMaps sm;
  SgmvArgs sa = {};
  PcArgs plan = {};
  const LinearKernel kernel = linear_kernel(p, with_lora, &plan);
  if (kernel == kLinearCluster) {
    // (uses none; the entry point's contract is the same for every shape)
    if (int rc = sgmv_workspace_check(b, slices, workspace, workspace_bytes)) return rc;
    return prefill_cluster_launch(b, plan, p.weight, p.w_ld, p.n_total, p.bias, false, stream);
  }
  if (with_lora) {
    if (int rc = sgmv_prepare(b, workspace, workspace_bytes, &sm, &sa)) return rc;
    if (int rc = sgmv_launch_shrink(sm, sa, stream)) return rc;
  } else {
    // no adapter work: only the x and y views are needed
    sa.y = static_cast<__nv_bfloat16*>(b.y); sa.y_ld = b.y_ld; sa.T = b.T; sa.in_dim = b.in_dim; sa.S = 1; sa.r_max = 16;
    sa.n = 0; sa.token_to_slot = nullptr;
    if (int rc = make_tmap_2d(&sm.x, b.x, (uint64_t)b.T, (uint64_t)b.in_dim, (uint64_t)b.x_ld, kSgmvBM, kSgmvBK)) return rc;
    sm.t = sm.x;
    for (int s = 0; s < B200_LORA_MAX_SLICES; ++s) { sm.a[s] = sm.x; sm.b[s] = sm.x; }
  }
  if (kernel == kLinearPairs) {
    const void* slab_b[B200_LORA_MAX_SLICES];
    int n = 0;
    for (int s = 0; s < b.st.n; ++s)
      if (b.st.out[s] > 0) slab_b[n++] = b.st.b[s];
    return linear_pair_launch(sm, sa, slab_b, p.weight, p.w_ld, p.silu ? p.n_total / 2 : p.n_total, p.bias, with_lora, p.silu, stream);
  }
  if (p.silu) return fail(B200_LORA_EUNSUPPORTED, "fused linear with SiLU: slices and columns must be multiples of 32");
  const bool fuse = with_lora && tc_lora_stage_ok(sa);
  GemmMaps gm;
  GemmArgs ga;
  if (int rc = tc_tile_prepare(sm, sa, p.weight, p.w_ld, p.n_total, p.bias, false, fuse, &gm, &ga)) return rc;
  if (int rc = tc_tile_launch(gm, ga, stream)) return rc;
  if (!with_lora || fuse) return B200_LORA_OK;
  return sgmv_launch_expand(sm, sa, stream);  // slices not 16-column aligned: delta in a second pass
}

}  // namespace b200lora
