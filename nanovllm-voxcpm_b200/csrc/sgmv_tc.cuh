// Prefill multi-LoRA kernels (bf16) on the Blackwell tensor cores: tcgen05.mma with TMEM
// accumulators, operands staged in shared memory by tiled TMA loads (no multicast), mbarrier
// pipelines between a TMA warp, an MMA-issuing thread and four epilogue warps.
//
// Tiling follows the token order, not the bucket arrays: block k owns rows [128k, 128k+128)
// of x / y. Inside a block, maximal runs of consecutive rows with the same slot (>= 0) are
// found from token_to_slot; in a prefill batch a block is one run, two at a request boundary.
// Each run is one M=128 MMA tile whose rows outside the run are computed and thrown away
// (masked in the epilogue), so rows with slot -1 are never written.
//
//   sgmv_shrink_kernel : tmp[s, rows, :] = sc * x[rows, :] . A_s[slot]^T        (K = in)
//   sgmv_expand_kernel : y[rows, cols]  += tmp[s, rows, :] . B_s[slot][cols]^T   (K = r)
// tmp [n, T, r_max] (bf16) lives in caller-provided scratch memory.
#pragma once

#include "tc_common.cuh"
#include "bgmv_fused.cuh"  // launch options shared by all kernels (programmatic dependent launch on / off)

namespace b200lora {

constexpr int kSgmvThreads = 192;   // warp 0: TMA, warp 1: MMA + TMEM owner, warps 2-5: epilogue
constexpr int kSgmvBM = 128;        // rows per block / MMA M
constexpr int kSgmvBK = 64;         // K columns per shrink stage (one 128-byte swizzle row)
constexpr int kSgmvBN = 256;        // output columns per expand tile
constexpr int kSgmvShrinkMaxStages = 12; // the launch picks as many 64-column stages as fit into shared memory
constexpr int kSgmvExpandStages = 3;
constexpr int kSgmvAutoMinTokens = 512;  // IMPL_AUTO uses these kernels from this batch size on

struct SgmvArgs {
  __nv_bfloat16* y; int64_t y_ld;
  __nv_bfloat16* tmp;                       // [n, T, r_max]
  int T, in_dim, S, r_max, n;
  int out[B200_LORA_MAX_SLICES], col[B200_LORA_MAX_SLICES];
  const int32_t* token_to_slot;
  const float* scale_per_slot; float scaling;
  int zero_fill;                            // shrink: write zero rows for tokens without adapter
  int skip_clean;                           // expand: leave blocks in which every row has an adapter to tc_tile_kernel
  int gate;                                 // leave batches of scattered rows to another kernel (rows_scattered)
  int shrink_gmax;                          // shrink: runs of a block whose K loops share one pass over x (set by the launch)
  int shrink_ring_bytes;                    // shrink: bytes of the TMA ring (set by the launch)
  int shrink_ck;                            // shrink: CTAs of a cluster = parts of K (set by the launch)
};

struct SgmvMaps {
  CUtensorMap x;                            // [T, in]            box 128 x 64
  CUtensorMap a[B200_LORA_MAX_SLICES];      // [S*r_max, in]      box r_max x 64
  CUtensorMap t;                            // [n*T, r_max]       box 128 x r_max
  CUtensorMap b[B200_LORA_MAX_SLICES];      // [S*out_s, r_max]   box 256 x r_max
};

// Runs of equal slot inside the 128-row block `blk`, found by the CTA's first four warps (a scan of the block by one thread
// took 2 us per block). (table element types are the caller's: slot ids fit int16 for S <= 32767, row bounds 0..128 fit uint8)
template <typename TS, typename TR>
__device__ __forceinline__ void sgmv_find_runs(const int32_t* tts, int T, int S, int blk, TS* s_slot, TS* run_slot,
                                               TR* run_lo, TR* run_hi, int* nruns) {
  __shared__ int warp_starts[4];
  const int i = threadIdx.x, row = blk * kSgmvBM + i;
  if (i < kSgmvBM) {
    int sl = -1;
    if (row < T) sl = tts[row];
    (void)B200_IN_BOUNDS(sl >= -1 && sl < S);  // ids outside [-1, S) are treated as "no adapter"; the checked build reports them
    if (sl >= S || sl < -1) sl = -1;
    s_slot[i] = (TS)sl;
  }
  __syncthreads();
  bool starts = false, ends = false;
  unsigned before = 0;
  if (i < kSgmvBM) {
    const int sl = s_slot[i];
    starts = sl >= 0 && (i == 0 || s_slot[i - 1] != sl);
    ends = sl >= 0 && (i == kSgmvBM - 1 || s_slot[i + 1] != sl);
    const unsigned mask = __ballot_sync(0xffffffffu, starts);
    before = __popc(mask & ((2u << (i & 31)) - 1u));  // runs of this warp that start at or before this row
    if ((i & 31) == 0) warp_starts[i >> 5] = __popc(mask);
  }
  __syncthreads();
  if (i < kSgmvBM) {
    for (int w = 0; w < i >> 5; ++w) before += (unsigned)warp_starts[w];
    if (starts) { run_slot[before - 1] = s_slot[i]; run_lo[before - 1] = (TR)i; }
    if (ends) run_hi[before - 1] = (TR)(i + 1);
  }
  if (i == 0) *nruns = warp_starts[0] + warp_starts[1] + warp_starts[2] + warp_starts[3];
  __syncthreads();
}

__device__ __forceinline__ void store_bf16x32(__nv_bfloat16* dst, const uint32_t (&v)[32], float sc, int ncols) {
  // v holds fp32 bit patterns of 32 consecutive columns; write the first `ncols` (multiple of 8)
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (q * 8 < ncols) {
      uint4 o;
      o.x = pack_bf16x2(__uint_as_float(v[8 * q + 0]) * sc, __uint_as_float(v[8 * q + 1]) * sc);
      o.y = pack_bf16x2(__uint_as_float(v[8 * q + 2]) * sc, __uint_as_float(v[8 * q + 3]) * sc);
      o.z = pack_bf16x2(__uint_as_float(v[8 * q + 4]) * sc, __uint_as_float(v[8 * q + 5]) * sc);
      o.w = pack_bf16x2(__uint_as_float(v[8 * q + 6]) * sc, __uint_as_float(v[8 * q + 7]) * sc);
      stg128(dst + 8 * q, o);
    }
  }
}

// Optional timeline of tuning builds: wall clock (ns) at entry / exit of every shrink CTA, SM clock at the
// k-steps of CTA 0's MMA thread.
#ifdef B200_TRACE
#define B200_SHRINK_TRACE_CTA(which)                                                        \
  if (threadIdx.x == 0 && blockIdx.x < 512) {                                               \
    unsigned long long t_;                                                                  \
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));                                  \
    g_b200_trace[4096 + 2 * blockIdx.x + (which)] = (long long)t_;                          \
  }
#define B200_SHRINK_TRACE_K(i) \
  if (blockIdx.x == 0 && (i) < 256) g_b200_trace[6144 + (i)] = clock64();
#else
#define B200_SHRINK_TRACE_CTA(which)
#define B200_SHRINK_TRACE_K(i)
#endif

// ============================================================================ shrink
// One cluster per 128-row block. Its CTAs split K: a CTA's K loop is a chain of latencies (0.5 us per 64 columns, 31 us for
// 1000 rows of 2048-wide layers on 16 CTAs), so the loop is made short and the GPU filled; the partial sums meet in
// distributed shared memory. The lora_A tiles of a run's slices lie side by side and are one MMA operand of n * r columns.
__global__ void __launch_bounds__(kSgmvThreads, 1)
sgmv_shrink_kernel(const __grid_constant__ SgmvMaps maps, const SgmvArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ int s_slot[kSgmvBM], run_slot[kSgmvBM], run_lo[kSgmvBM], run_hi[kSgmvBM];
  __shared__ int nruns_s;
  __shared__ __align__(8) uint64_t bars[2 * kSgmvShrinkMaxStages + 4];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_flag;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int CK = a.shrink_ck, ck = CK > 1 ? (int)cluster_ctarank() : 0;
  const int blk = (int)blockIdx.x / CK;
  const int r = a.r_max, n = a.n, width = n * r;
  B200_SHRINK_TRACE_CTA(0)
  if (a.gate && rows_scattered(a.token_to_slot, a.T)) {
    griddep_wait();
    return;
  }
  const uint32_t a_tile_bytes = (uint32_t)r * kSgmvBK * 2;
  const uint32_t x_tile_bytes = kSgmvBM * kSgmvBK * 2;
  const uint32_t smem_base = (smem_u32(smem) + 1023u) & ~1023u;  // swizzled tiles need 1024-byte alignment
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * (uint32_t)s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (uint32_t)(kSgmvShrinkMaxStages + s); };
  const uint32_t acc_full = bar0 + 8u * (2 * kSgmvShrinkMaxStages);
  const uint32_t acc_empty = acc_full + 8u, part_ready = acc_full + 16u, part_done = acc_full + 24u;
  int tmem_cols = 32;  // the last slice is read in 32-column chunks
  while (tmem_cols < (a.shrink_gmax * n - 1) * r + ((r + 31) & ~31)) tmem_cols *= 2;

  if (tid == 0) {
    for (int s = 0; s < kSgmvShrinkMaxStages; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, kSgmvBM);
    mbar_init(part_ready, (uint32_t)CK);  // every CTA of the cluster has written / read the partial sums of an exchange
    mbar_init(part_done, (uint32_t)CK);
    abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_s), (uint32_t)tmem_cols);
    tc_fence_before_sync();
  }
  sgmv_find_runs(a.token_to_slot, a.T, a.S, blk, s_slot, run_slot, run_lo, run_hi, &nruns_s);  // has __syncthreads
  if (CK > 1) { cluster_arrive(); cluster_wait(); }  // the barriers of every CTA of the cluster are initialised
  // Launched under programmatic dependent launch: everything above (barriers, TMEM, the run table from the index
  // metadata) may overlap the previous kernel of the stream; x is read and tmp written only from here on.
  griddep_wait();
  // Only now may the tile kernel that follows start: it reads x (and W) without waiting for anything, so it must
  // not run before the kernels ahead of this one are complete; it waits for this kernel before it reads tmp.
  griddep_launch_dependents();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  const int nruns = nruns_s;
  const int nk_all = a.in_dim / kSgmvBK, nk_per = (nk_all + CK - 1) / CK;
  const int kc0 = min(ck * nk_per, nk_all), nk = min(nk_per, nk_all - kc0);  // this CTA's K steps (at least one: see the launch)
  // The runs of a block (two at a request boundary) share ONE pass over x: every K step loads the x tile once
  // and one lora_A tile per run and slice, and the MMAs of run i accumulate into their own TMEM columns
  // [i * n * r, +n * r). Up to G runs per pass; the ring depth follows from the stage size of this block.
  const int G = min(a.shrink_gmax, max(nruns, 1));
  const uint32_t stage_bytes = x_tile_bytes + (uint32_t)(G * n) * a_tile_bytes;
  const int NS = min(kSgmvShrinkMaxStages, (int)((uint32_t)a.shrink_ring_bytes / stage_bytes));
  const int npass = (nruns + G - 1) / G;

  if (warp == 0) {
    const uint32_t leader = elect_one();
    if (leader) {
      tma_prefetch_desc(&maps.x);
      for (int s = 0; s < n; ++s) tma_prefetch_desc(&maps.a[s]);
    }
    int st = 0, round = 0;
    for (int pi = 0; pi < npass; ++pi) {
      // the partial sums of a pass lie where the ring is
      if (CK > 1 && pi > 0) mbar_wait_bounded(acc_empty, (uint32_t)((pi - 1) & 1), &abort_flag);
      const int u0 = pi * G, g = min(G, nruns - u0);
      int row[4];  // first lora_A row of each run of the pass (G <= 4)
#pragma unroll
      for (int ui = 0; ui < 4; ++ui) row[ui] = uniform(ui < g ? run_slot[u0 + ui] * r : 0);
      for (int kc = 0; kc < nk; ++kc) {
        if (round > 0) mbar_wait_bounded(empty_bar(st), (uint32_t)((round & 1) ^ 1), &abort_flag);
        if (leader) {
          const uint32_t base = smem_base + (uint32_t)st * stage_bytes, bar = full_bar(st);
          mbar_arrive_expect_tx(bar, x_tile_bytes + (uint32_t)(g * n) * a_tile_bytes);
          tma_load_2d(base, &maps.x, (kc0 + kc) * kSgmvBK, blk * kSgmvBM, bar);
          uint32_t dst = base + x_tile_bytes;
#pragma unroll
          for (int ui = 0; ui < 4; ++ui)
            if (ui < g)
              for (int s = 0; s < n; ++s, dst += a_tile_bytes) tma_load_2d(dst, &maps.a[s], (kc0 + kc) * kSgmvBK, row[ui], bar);
        }
        __syncwarp();
        if (++st == NS) { st = 0; ++round; }
      }
    }
  } else if (warp == 1) {
    const uint32_t leader = elect_one();
    const uint64_t desc0 = umma_smem_desc(smem_base, 128);
    const uint32_t hi = (uint32_t)(desc0 >> 32), lo0 = (uint32_t)desc0;
    const uint32_t idesc = umma_idesc_bf16(kSgmvBM, width);
    int st = 0, round = 0;
    for (int pi = 0; pi < npass; ++pi) {
      const int jobs = uniform(min(G, nruns - pi * G));
      if (pi > 0) mbar_wait_bounded(acc_empty, (uint32_t)((pi - 1) & 1), &abort_flag);
      tc_fence_after_sync();
      for (int kc = 0; kc < nk; ++kc) {
        mbar_wait_bounded(full_bar(st), (uint32_t)(round & 1), &abort_flag);
        B200_SHRINK_TRACE_K(kc)
        tc_fence_after_sync();
        const uint32_t xl = lo0 + ((uint32_t)st * stage_bytes >> 4);
        uint32_t al = xl + (x_tile_bytes >> 4), d = tmem_base;
        for (int q = 0; q < jobs; ++q, al += (uint32_t)n * a_tile_bytes >> 4, d += (uint32_t)width) {  // runs of the pass
#pragma unroll
          for (int k4 = 0; k4 < kSgmvBK / 16; ++k4) umma_elected(d, xl + 2u * k4, al + 2u * k4, hi, idesc, (kc > 0 || k4 > 0) ? 1u : 0u, leader);
        }
        umma_commit_elected(empty_bar(st), leader);  // stage reusable once these MMAs have read it
        if (++st == NS) { st = 0; ++round; }
      }
      umma_commit_elected(acc_full, leader);
    }
  } else {
    // epilogue: thread <-> row; a warp may only touch its own quarter of the 128 TMEM lanes
    const int quarter = warp & 3, row_in_blk = quarter * 32 + lane, etid = tid - 64;
    const int row = blk * kSgmvBM + row_in_blk;
    if (a.zero_fill && ck == 0 && row < a.T && s_slot[row_in_blk] < 0) {
      for (int s = 0; s < n; ++s) {
        __nv_bfloat16* dst = a.tmp + ((int64_t)s * a.T + row) * r;
        for (int c = 0; c < r; c += 8) stg128(dst + c, make_uint4(0, 0, 0, 0));
      }
    }
    int exchange = 0;
    for (int pi = 0; pi < npass; ++pi) {
      const int u0 = pi * G, g = min(G, nruns - u0);
      mbar_wait_bounded(acc_full, (uint32_t)(pi & 1), &abort_flag);
      tc_fence_after_sync();
      for (int ui = 0; ui < g; ++ui) {
        const int u = u0 + ui;
        // (a TMEM load is a warp-wide operation on one column range: a warp whose 32 rows straddle two runs
        //  reads both runs' columns and every lane keeps the ones of its own run)
        const int lo_row = run_lo[u], hi_row = run_hi[u];
        const bool touched = hi_row > quarter * 32 && lo_row < quarter * 32 + 32;  // warp-uniform
        const int slot = run_slot[u];
        const float sc = a.scaling * (a.scale_per_slot != nullptr ? a.scale_per_slot[slot] : 1.0f);
        if (CK == 1) {
          if (!touched) continue;
          const bool mine = row_in_blk >= lo_row && row_in_blk < hi_row && row < a.T;
          for (int s = 0; s < n; ++s) {
            for (int c = 0; c < r; c += 32) {
              uint32_t v[32];
              tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((ui * n + s) * r + c), v);
              tmem_ld_wait();
              if (mine) store_bf16x32(a.tmp + ((int64_t)s * a.T + row) * r + c, v, sc, min(32, r - c));
            }
          }
          continue;
        }
        // this CTA's partial sums into its own shared memory, as [4 columns][row] pieces of 16 bytes: the lanes of a remote read
        // then cover consecutive bytes (row-major sums, 16 bytes a lane at a pitch, came at 8 bytes per clock) ...
        if (exchange > 0) mbar_wait_bounded_acquire_cluster(part_done, (uint32_t)((exchange - 1) & 1), &abort_flag);
        if (touched) {
          for (int c = 0; c < width; c += 16) {
            uint32_t v[16];
            tmem_ld_32x16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ui * width + c), v);
            tmem_ld_wait();
            const uint32_t dst = smem_base + (uint32_t)((c >> 2) * kSgmvBM + row_in_blk) * 16u;
#pragma unroll
            for (int q = 0; q < 4; ++q) sts128(dst + 16u * kSgmvBM * q, make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]));
          }
        }
        named_bar_sync(2, kSgmvBM);
        if (etid < CK) mbar_arrive_remote_release(mapa_shared(part_ready, (uint32_t)etid));
        mbar_wait_bounded_acquire_cluster(part_ready, (uint32_t)(exchange & 1), &abort_flag);
        // ... then every CTA adds its share of (8 columns x row) pieces over the cluster
        const int pieces = (width >> 3) * kSgmvBM, per = (pieces + CK - 1) / CK;
        const int first = ck * per + etid, last = min((ck + 1) * per, pieces);
        auto add_pieces = [&](auto parts) {
          // eight remote reads of 32 bytes in flight per thread: one at a time each costs a round trip of 500 cycles
          constexpr int kParts = decltype(parts)::value, kBatch = 8 / kParts;
          for (int e0 = first; e0 < last; e0 += kBatch * kSgmvBM) {
            float4 v[8][2];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const int e = e0 + (q / kParts) * kSgmvBM, er = e & (kSgmvBM - 1);
              v[q][0] = v[q][1] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (e < last && er >= lo_row && er < hi_row) {
                const uint32_t src = mapa_shared(smem_base + (uint32_t)(2 * (e >> 7) * kSgmvBM + er) * 16u, (uint32_t)(q % kParts));
                v[q][0] = ld_cluster_f32x4(src);
                v[q][1] = ld_cluster_f32x4(src + 16u * kSgmvBM);
              }
            }
#pragma unroll
            for (int h = 0; h < kBatch; ++h) {
              const int e = e0 + h * kSgmvBM, er = e & (kSgmvBM - 1), grow = blk * kSgmvBM + er;
              if (e >= last || er < lo_row || er >= hi_row || grow >= a.T) continue;
              float4 s0 = v[h * kParts][0], s1 = v[h * kParts][1];
#pragma unroll
              for (int q = 1; q < kParts; ++q) {
                const float4 w0 = v[h * kParts + q][0], w1 = v[h * kParts + q][1];
                s0.x += w0.x; s0.y += w0.y; s0.z += w0.z; s0.w += w0.w;
                s1.x += w1.x; s1.y += w1.y; s1.z += w1.z; s1.w += w1.w;
              }
              const int col = 8 * (e >> 7), s = col / r, c = col - s * r;
              stg128(a.tmp + ((int64_t)s * a.T + grow) * r + c,
                     make_uint4(pack_bf16x2(s0.x * sc, s0.y * sc), pack_bf16x2(s0.z * sc, s0.w * sc), pack_bf16x2(s1.x * sc, s1.y * sc),
                                pack_bf16x2(s1.z * sc, s1.w * sc)));
            }
          }
        };
        if (CK == 8) add_pieces(std::integral_constant<int, 8>{});
        else if (CK == 4) add_pieces(std::integral_constant<int, 4>{});
        else add_pieces(std::integral_constant<int, 2>{});
        if (++exchange < nruns) {  // (after the last one the cluster barrier at the end keeps the sums in place)
          named_bar_sync(2, kSgmvBM);
          if (etid < CK) mbar_arrive_remote_release(mapa_shared(part_done, (uint32_t)etid));
        }
      }
      // (the partial sums lie where the ring is: no refill before every CTA has read them)
      if (CK > 1 && pi + 1 < npass) mbar_wait_bounded_acquire_cluster(part_done, (uint32_t)((exchange - 1) & 1), &abort_flag);
      if (CK > 1) fence_proxy_async_smem();
      tc_fence_before_sync();
      mbar_arrive(acc_empty);
    }
  }
  __syncthreads();
  B200_SHRINK_TRACE_CTA(1)
  if (warp == 1) tmem_dealloc(tmem_base, (uint32_t)tmem_cols);
  if (tid == 0 && abort_flag != 0) atomicOr(&g_b200_status, kStatusWaitGaveUp);
  if (CK > 1) { cluster_arrive(); cluster_wait(); }  // the peers have read this CTA's partial sums
}

// ============================================================================ expand
__global__ void __launch_bounds__(kSgmvThreads, 1)
sgmv_expand_kernel(const __grid_constant__ SgmvMaps maps, const SgmvArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ int s_slot[kSgmvBM], run_slot[kSgmvBM], run_lo[kSgmvBM], run_hi[kSgmvBM];
  __shared__ int nruns_s;
  __shared__ __align__(8) uint64_t bars[2 * kSgmvExpandStages + 4];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_flag;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int blk = blockIdx.x, z = blockIdx.y, Z = gridDim.y;
  if (a.gate && rows_scattered(a.token_to_slot, a.T)) return;
  const int r = a.r_max, n = a.n;
  const uint32_t t_tile_bytes = (uint32_t)kSgmvBM * r * 2;
  const uint32_t b_tile_bytes = (uint32_t)kSgmvBN * r * 2;
  const uint32_t stage_bytes = t_tile_bytes + b_tile_bytes;
  const uint32_t smem_base = (smem_u32(smem) + 1023u) & ~1023u;  // swizzled tiles need 1024-byte alignment
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * (uint32_t)s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (uint32_t)(kSgmvExpandStages + s); };
  auto acc_full = [&](int b) { return bar0 + 8u * (uint32_t)(2 * kSgmvExpandStages + b); };
  auto acc_empty = [&](int b) { return bar0 + 8u * (uint32_t)(2 * kSgmvExpandStages + 2 + b); };
  constexpr int tmem_cols = 2 * kSgmvBN;  // two accumulator buffers

  if (tid == 0) {
    for (int s = 0; s < kSgmvExpandStages; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 128); }
    abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_s), (uint32_t)tmem_cols);
    tc_fence_before_sync();
  }
  sgmv_find_runs(a.token_to_slot, a.T, a.S, blk, s_slot, run_slot, run_lo, run_hi, &nruns_s);
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  int nruns = nruns_s;
  {
    // blocks in which every in-range row has an adapter are done by tc_tile_kernel when asked to
    const int nvalid = min(kSgmvBM, a.T - blk * kSgmvBM);
    int covered = 0;
    for (int u = 0; u < nruns; ++u) covered += run_hi[u] - run_lo[u];
    if (a.skip_clean && covered == nvalid) nruns = 0;
  }
  const int row_bytes = r * 2;  // 32 / 64 / 128: the swizzle span of both operand tiles

  // Jobs of this CTA, in the same order for all three roles:
  //   for run u, for slice s, for column tile j = z, z+Z, ... of the slice
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&maps.t);
      for (int s = 0; s < n; ++s) tma_prefetch_desc(&maps.b[s]);
      int st = 0, round = 0;
      for (int u = 0; u < nruns; ++u) {
        const int slot = run_slot[u];
        for (int s = 0; s < n; ++s) {
          const int ntile = (a.out[s] + kSgmvBN - 1) / kSgmvBN;
          for (int j = z; j < ntile; j += Z) {
            if (round > 0) mbar_wait_bounded(empty_bar(st), (uint32_t)((round & 1) ^ 1), &abort_flag);
            const uint32_t base = smem_base + (uint32_t)st * stage_bytes;
            mbar_arrive_expect_tx(full_bar(st), stage_bytes);
            tma_load_2d(base, &maps.t, 0, s * a.T + blk * kSgmvBM, full_bar(st));
            tma_load_2d(base + t_tile_bytes, &maps.b[s], 0, slot * a.out[s] + j * kSgmvBN, full_bar(st));
            if (++st == kSgmvExpandStages) { st = 0; ++round; }
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = umma_idesc_bf16(kSgmvBM, kSgmvBN);
      int st = 0, round = 0, job = 0;
      for (int u = 0; u < nruns; ++u) {
        for (int s = 0; s < n; ++s) {
          const int ntile = (a.out[s] + kSgmvBN - 1) / kSgmvBN;
          for (int j = z; j < ntile; j += Z, ++job) {
            const int buf = job & 1;
            if (job >= 2) mbar_wait_bounded(acc_empty(buf), (uint32_t)(((job >> 1) - 1) & 1), &abort_flag);
            mbar_wait_bounded(full_bar(st), (uint32_t)(round & 1), &abort_flag);
            tc_fence_after_sync();
            const uint32_t base = smem_base + (uint32_t)st * stage_bytes;
            const uint64_t tdesc = umma_smem_desc(base, row_bytes);
            const uint64_t bdesc = umma_smem_desc(base + t_tile_bytes, row_bytes);
            for (int k4 = 0; k4 < r / 16; ++k4)
              umma_bf16(tmem_base + (uint32_t)(buf * kSgmvBN), tdesc + 2u * k4, bdesc + 2u * k4, idesc, k4 > 0 ? 1u : 0u);
            umma_commit(empty_bar(st));
            umma_commit(acc_full(buf));
            if (++st == kSgmvExpandStages) { st = 0; ++round; }
          }
        }
      }
    }
  } else {
    const int quarter = warp & 3;
    const int row_in_blk = quarter * 32 + lane;
    const int row = blk * kSgmvBM + row_in_blk;
    int job = 0;
    for (int u = 0; u < nruns; ++u) {
      const bool mine = row_in_blk >= run_lo[u] && row_in_blk < run_hi[u] && row < a.T;
      for (int s = 0; s < n; ++s) {
        const int ntile = (a.out[s] + kSgmvBN - 1) / kSgmvBN;
        for (int j = z; j < ntile; j += Z, ++job) {
          const int buf = job & 1;
          mbar_wait_bounded(acc_full(buf), (uint32_t)((job >> 1) & 1), &abort_flag);
          tc_fence_after_sync();
          const int c0 = j * kSgmvBN;
          __nv_bfloat16* yrow = a.y + (int64_t)row * a.y_ld + a.col[s] + c0;
          for (int c = 0; c < kSgmvBN; c += 32) {
            uint32_t v[32];
            tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * kSgmvBN + c), v);
            tmem_ld_wait();
            if (mine) {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                if (c0 + c + 8 * q < a.out[s]) {
                  uint4 yv = ldg128(yrow + c + 8 * q);
                  yv.x = add_bf16x2(yv.x, __uint_as_float(v[8 * q + 0]), __uint_as_float(v[8 * q + 1]));
                  yv.y = add_bf16x2(yv.y, __uint_as_float(v[8 * q + 2]), __uint_as_float(v[8 * q + 3]));
                  yv.z = add_bf16x2(yv.z, __uint_as_float(v[8 * q + 4]), __uint_as_float(v[8 * q + 5]));
                  yv.w = add_bf16x2(yv.w, __uint_as_float(v[8 * q + 6]), __uint_as_float(v[8 * q + 7]));
                  stg128(yrow + c + 8 * q, yv);
                }
              }
            }
          }
          tc_fence_before_sync();
          mbar_arrive(acc_empty(buf));
        }
      }
    }
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, (uint32_t)tmem_cols);
  if (tid == 0 && abort_flag != 0) atomicOr(&g_b200_status, kStatusWaitGaveUp);
}

// ============================================================================ host side
struct SgmvProblem {
  void* y; int64_t y_ld; const void* x; int64_t x_ld;
  int T, in_dim, S, r_max;
  SliceTable st;
  const float* scale_per_slot; const int32_t* token_to_slot; float scaling;
};

inline size_t sgmv_workspace_bytes(int T, int n_slices, int r_max) {
  // tmp [n, T, r_max] bf16, plus one 128-row tile of slack so the last TMA box stays inside the allocation
  return ((size_t)n_slices * (size_t)T + kSgmvBM) * (size_t)r_max * 2 + 1024;
}

// `with_x` / `with_b`: which of the two halves the caller runs (shrink reads x and lora_A, expand reads tmp and lora_B)
inline bool sgmv_supported(const SgmvProblem& b, const char** why, bool with_x = true, bool with_b = true) {
  const char* dummy;
  if (why == nullptr) why = &dummy;
  int n = 0;
  for (int s = 0; s < b.st.n; ++s) n += b.st.out[s] > 0;
  if (n == 0) { *why = "no active slice"; return false; }
  if (b.r_max != 16 && b.r_max != 32 && b.r_max != 64) { *why = "r_max must be 16, 32 or 64"; return false; }
  if (n * b.r_max > 512) { *why = "n_slices * r_max exceeds the 512 TMEM columns"; return false; }
  if (with_x) {
    if (b.in_dim % kSgmvBK != 0) { *why = "in_dim must be a multiple of 64"; return false; }
    if (b.x_ld % 8 != 0 || (reinterpret_cast<uintptr_t>(b.x) & 15u)) { *why = "x must be 16-byte aligned with a row stride that is a multiple of 8"; return false; }
  }
  if (with_b && (b.y_ld % 8 != 0 || (reinterpret_cast<uintptr_t>(b.y) & 15u))) { *why = "y must be 16-byte aligned with a row stride that is a multiple of 8"; return false; }
  for (int s = 0; s < b.st.n; ++s) {
    if (b.st.out[s] == 0) continue;
    if (with_b && (b.st.out[s] % 8 != 0 || b.st.col[s] % 8 != 0)) { *why = "slice widths / offsets must be multiples of 8"; return false; }
    if ((with_x && (reinterpret_cast<uintptr_t>(b.st.a[s]) & 15u)) || (with_b && (reinterpret_cast<uintptr_t>(b.st.b[s]) & 15u))) {
      *why = "slabs must be 16-byte aligned";
      return false;
    }
  }
  return true;
}

// Launch arguments and tensor maps over an intermediate `tmp` [n, T, r_max] (bf16, 16-byte aligned) that holds
// `tmp_rows` rows: rows beyond that are neither written nor read (the maps clip).
inline int sgmv_prepare_tmp(const SgmvProblem& b, void* tmp, uint64_t tmp_rows, bool with_x, bool with_b, SgmvMaps* maps,
                            SgmvArgs* args) {
  const char* why = nullptr;
  if (!sgmv_supported(b, &why, with_x, with_b)) return fail(B200_LORA_EUNSUPPORTED, "prefill kernels: %s", why);
  if (tmp == nullptr || (reinterpret_cast<uintptr_t>(tmp) & 15u)) return fail(B200_LORA_EINVAL, "prefill kernels: the intermediate must be 16-byte aligned");
  SgmvArgs a = {};
  a.n = 0;
  const void* slab_a[B200_LORA_MAX_SLICES];
  const void* slab_b[B200_LORA_MAX_SLICES];
  for (int s = 0; s < b.st.n; ++s) {
    if (b.st.out[s] == 0) continue;
    slab_a[a.n] = b.st.a[s]; slab_b[a.n] = b.st.b[s];
    a.out[a.n] = b.st.out[s]; a.col[a.n] = b.st.col[s];
    ++a.n;
  }
  a.y = static_cast<__nv_bfloat16*>(b.y); a.y_ld = b.y_ld;
  a.tmp = static_cast<__nv_bfloat16*>(tmp);
  a.T = b.T; a.in_dim = b.in_dim; a.S = b.S; a.r_max = b.r_max;
  a.token_to_slot = b.token_to_slot; a.scale_per_slot = b.scale_per_slot; a.scaling = b.scaling;
  a.zero_fill = a.gate = 0;
  if (int rc = make_tmap_2d(&maps->t, a.tmp, tmp_rows, (uint64_t)b.r_max, (uint64_t)b.r_max, kSgmvBM, (uint32_t)b.r_max)) return rc;
  if (with_x) {
    if (int rc = make_tmap_2d(&maps->x, b.x, (uint64_t)b.T, (uint64_t)b.in_dim, (uint64_t)b.x_ld, kSgmvBM, kSgmvBK)) return rc;
  } else {
    maps->x = maps->t;  // never dereferenced by the expand half
  }
  for (int s = 0; s < a.n; ++s) {
    if (with_x) {
      if (int rc = make_tmap_2d(&maps->a[s], slab_a[s], (uint64_t)b.S * b.r_max, (uint64_t)b.in_dim, (uint64_t)b.in_dim, (uint32_t)b.r_max, kSgmvBK)) return rc;
    } else {
      maps->a[s] = maps->t;
    }
    if (with_b) {
      if (int rc = make_tmap_2d(&maps->b[s], slab_b[s], (uint64_t)b.S * a.out[s], (uint64_t)b.r_max, (uint64_t)b.r_max, kSgmvBN, (uint32_t)b.r_max)) return rc;
    } else {
      maps->b[s] = maps->t;
    }
  }
  for (int s = a.n; s < B200_LORA_MAX_SLICES; ++s) { maps->a[s] = maps->a[0]; maps->b[s] = maps->b[0]; }
  *args = a;
  return B200_LORA_OK;
}

inline int sgmv_workspace_check(const SgmvProblem& b, int n, const void* workspace, size_t workspace_bytes) {
  const size_t need = sgmv_workspace_bytes(b.T, std::max(n, 1), b.r_max);
  if (workspace == nullptr || workspace_bytes < need)
    return fail(B200_LORA_EWORKSPACE, "prefill kernels need %zu bytes of scratch, got %zu", need, workspace_bytes);
  return B200_LORA_OK;
}

// Builds the launch arguments and tensor maps shared by the two kernels, the intermediate in caller-provided scratch.
inline int sgmv_prepare(const SgmvProblem& b, void* workspace, size_t workspace_bytes, SgmvMaps* maps, SgmvArgs* args) {
  int n = 0;
  for (int s = 0; s < b.st.n; ++s) n += b.st.out[s] > 0;
  if (int rc = sgmv_workspace_check(b, n, workspace, workspace_bytes)) return rc;
  uintptr_t ws = (reinterpret_cast<uintptr_t>(workspace) + 1023) & ~(uintptr_t)1023;
  return sgmv_prepare_tmp(b, reinterpret_cast<void*>(ws), (uint64_t)n * b.T + kSgmvBM, true, true, maps, args);
}

inline int sgmv_set_smem(const void* kernel, size_t bytes) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return fail(B200_LORA_ECUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  return B200_LORA_OK;
}

inline int sgmv_launch_shrink(const SgmvMaps& maps, const SgmvArgs& a_in, cudaStream_t stream) {
  SgmvArgs a = a_in;
  // A CTA streams its 128 rows of x through a ring that fills the shared memory of the SM: the more bytes in flight, the
  // better. Up to 4 runs of a block share a pass, as long as their accumulators fit into the 512 TMEM columns and three
  // stages of that size fit into the ring.
  const size_t ring = 216 * 1024;
  const size_t x_tile = kSgmvBM * kSgmvBK * 2, a_tiles = (size_t)a.n * a.r_max * kSgmvBK * 2;
  int gmax = 1;
  for (int g = 2; g <= 4; ++g) {
    const int cols = (g * a.n - 1) * a.r_max + ((a.r_max + 31) & ~31);
    if (cols <= 512 && ring / (x_tile + g * a_tiles) >= 3) gmax = g;
  }
  a.shrink_gmax = gmax;
  a.shrink_ring_bytes = (int)ring;
  const size_t smem = ring + 1024;
  if (int rc = sgmv_set_smem(reinterpret_cast<const void*>(sgmv_shrink_kernel), smem)) return rc;
  const int nblk = (a.T + kSgmvBM - 1) / kSgmvBM, nk = a.in_dim / kSgmvBK;
  // K parts: as many as fill the SMs once, every part at least one K step
  a.shrink_ck = 1;
  while (a.shrink_ck < 8 && nblk * a.shrink_ck * 2 <= 148 && ((nk + 2 * a.shrink_ck - 1) / (2 * a.shrink_ck)) * (2 * a.shrink_ck - 1) < nk) a.shrink_ck *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(nblk * a.shrink_ck), 1, 1);
  cfg.blockDim = dim3(kSgmvThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)a.shrink_ck;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = bgmv_options().pdl ? 2 : 1;  // B200_LORA_OPT_PDL = 0: strict stream order (the waits in the kernel are then no-ops)
  cudaError_t e = cudaLaunchKernelEx(&cfg, sgmv_shrink_kernel, maps, a);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(B200_LORA_ECUDA, "sgmv_shrink_kernel launch: %s", cudaGetErrorString(e));
  }
  return B200_LORA_OK;
}

inline int sgmv_launch_expand(const SgmvMaps& maps, const SgmvArgs& a, cudaStream_t stream) {
  const size_t smem = (size_t)kSgmvExpandStages * ((size_t)kSgmvBM * a.r_max * 2 + (size_t)kSgmvBN * a.r_max * 2) + 1024;
  if (int rc = sgmv_set_smem(reinterpret_cast<const void*>(sgmv_expand_kernel), smem)) return rc;
  const int nblk = (a.T + kSgmvBM - 1) / kSgmvBM;
  int max_tiles = 1;
  for (int s = 0; s < a.n; ++s) max_tiles = std::max(max_tiles, (a.out[s] + kSgmvBN - 1) / kSgmvBN);
  int Z = std::max(1, std::min(max_tiles, (2 * 148 + nblk - 1) / nblk));
  sgmv_expand_kernel<<<dim3(nblk, Z), kSgmvThreads, smem, stream>>>(maps, a);
  return check_launch("sgmv_expand_kernel");
}

}  // namespace b200lora
