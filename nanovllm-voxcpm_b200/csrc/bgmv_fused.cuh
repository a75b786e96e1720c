// Fused decode multi-LoRA kernel (bf16, fp16): shrink + expand in ONE launch.
//
// Work decomposition
//   grid = (C, clusters), thread-block cluster = (C, 1, 1). Bucket g of the batch is the tokens
//   sorted_idx[offsets[g] .. +counts[g]), which all use adapter slot slot_ids[g]; it is cut into
//   windows of 16 tokens (one MMA M tile), and a cluster takes one window. There is a cluster per
//   bucket, for its first window, and extra ones for the further windows of popular buckets (256
//   rows over 32 adapters of skewed popularity, four layers of 1024: 92 us; with 32 rows per cluster
//   in two passes 133, with a whole bucket in one cluster 315). With fewer rows than buckets there is
//   one per window that the rows can make.
//   Clusters without rows exit at once.
//   Inside a cluster the adapter's weights are split so that every byte of
//   lora_A[slot] and lora_B[slot] is pulled from HBM by exactly one CTA:
//     shrink : the n*r stacked rank rows are split across the C CTAs (full K each)
//     expand : each slice's output rows are split across the C CTAs
//   and the rank-r intermediate tmp[16 tokens, n*r] (bf16) is all-gathered through
//   distributed shared memory between the two phases (st.async: the data and their byte
//   count on the receiver's mbarrier in one operation).
//
// Roles
//   warp 8      producer: walks the CTA's tile list and issues 1-D bulk async copies
//               (cp.async.bulk, the TMA unit) into a ring of stages guarded by full/empty
//               mbarriers. A shrink tile is 8 rank rows x up to 1024 columns (one 16 KB
//               copy when the rows are contiguous, else 8 row copies), an expand tile is
//               one contiguous copy of up to 16 KB of lora_B rows. The weights do not
//               depend on the previous kernel of the stream, so under programmatic
//               dependent launch they are requested before griddepcontrol.wait.
//   warps 0-7   consumers: mma.sync m16n8k16 bf16 -> fp32 with tokens as the 16-row
//               operand and weight rows as the
//               8-column operand. Activations are read straight into MMA fragments
//               (16-byte global loads, once per 1024-column part); y is read one tile
//               ahead and written back with 16-byte stores.
//   Fragments are read as 16-byte vectors: thread (g,t) of a warp takes columns
//   [8t, 8t+8) of a 32-column block for both operands, which is a fixed permutation of the
//   k index shared by A and B and therefore leaves the dot products unchanged.
//
// Rows whose slot is -1 are in no bucket and are never read or written.
#pragma once

#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"

namespace b200lora {

constexpr int kBgmvWarps = 8;                       // consumer warps
constexpr int kBgmvConsumers = kBgmvWarps * 32;
constexpr int kBgmvThreads = kBgmvConsumers + 32;   // + producer warp
constexpr int kBgmvTok = 16;           // tokens per cluster: a window of a bucket (one MMA M tile)
constexpr int kBgmvMaxRc = 64;         // stacked rank rows per CTA
constexpr int kBgmvKP = 1024;          // columns per shrink tile
constexpr int kBgmvXBlocks = kBgmvKP / 32 / kBgmvWarps;  // 32-column blocks per warp and tile
constexpr int kBgmvSmemMax = 232448;   // 227 KB opt-in maximum per CTA
constexpr int kBgmvMaxStages = 12;
constexpr int kBgmvMaxExpandTiles = 256;  // expand tiles of one CTA (its table has up to eight blocks of each)


// Optional phase timeline (SM clock) of rank-0 CTAs, compiled in only for tuning builds.
#ifdef B200_TRACE
__device__ long long g_b200_trace[1024 * 32];
#define B200_TRACE_AT(i, who) \
  if (tid == (who) && c == 0 && blockIdx.y < 1024) g_b200_trace[blockIdx.y * 32 + (i)] = clock64();
#else
#define B200_TRACE_AT(i, who)
#endif
#define B200_TRACE_POINT(i) B200_TRACE_AT(i, 0)
#define B200_TRACE_PRODUCER(i) B200_TRACE_AT(i, kBgmvConsumers)

struct BgmvProblem {
  void* y; int64_t y_ld; const void* x; int64_t x_ld;
  int T, in_dim, S, r_max;
  SliceTable st;
  const int32_t* rank_per_slot; const float* scale_per_slot;
  const int32_t *sorted_idx, *slot_ids, *counts, *offsets;
  int n_buckets; float scaling;
  // 0 = fused add; 1 = shrink only: tmp_io[s, t, 0:r] = scaling * x[t] . A_s[slot_t]^T (fp32, rows with an
  // adapter only); 2 = expand only: y += tmp_io . B^T. The pair serves the tensor-parallel exchange of tmp.
  // 3 = overwrite: y[t, cols] = delta for rows with an adapter and -0.0 for every other row (y is not
  // read); a base GEMM that then accumulates into y (beta = 1) gives base + delta, and x + (-0.0) == x
  // keeps rows without adapter bit-identical to the base result.
  // 4 = y = delta in fp32 [T, y_ld], rows with an adapter only: one of the planes that decode_step.cuh adds up.
  int mode = 0;
  // Precision of the rank-r intermediate and of the update. 0 (bf16, r_max % 32 == 0): tmp rounded to bf16, the delta
  // rounded to bf16 and added at the L2. 1 (bf16) / 2 (fp16): tmp kept as the sum of two 16-bit numbers, y read, added to
  // in fp32 and rounded once; modes 0, 1 and 2, r_max % 16 == 0. What the per-token kernel computes, which these sizes and
  // types used to take (a 37-row batch of rank-16 adapters: 45 us per projection there, 3 us here).
  int kind = 0;
  int beside = 0;          // CTAs of another kind in the launch
  void* tmp_io = nullptr;  // [n_slices, T, r_max], fp32 or (io16) values of the activations' type
  int io16 = 0;
  int zero_rows = 0;       // mode 1: rows without adapter are written as zeros (token_to_slot tells which)
  int no_add = 0;          // mode 2, kinds 1 and 2: y = delta in rows with an adapter instead of y += delta
  int gate = 0;            // modes 1, 2: leave batches of contiguous rows to another kernel (rows_scattered)
  const int32_t* token_to_slot = nullptr;  // modes 1 and 3: which rows have no adapter; gate
};

struct BgmvParams {
  __nv_bfloat16* y; int64_t y_ld; const __nv_bfloat16* x; int64_t x_ld;
  int T, in_dim, S, r_max;
  SliceTable st;  // active slices only
  const int32_t* rank_per_slot; const float* scale_per_slot;
  const int32_t *sorted_idx, *slot_ids, *counts, *offsets;
  int n_buckets; float scaling;
  int clusters, by_window;  // clusters of the launch; by_window: cluster i takes the i-th window of the batch
  int c_shift;      // cluster size C = 1 << c_shift
  int KP, nkp;      // columns per shrink tile (min(in, 1024)) and number of K parts
  int pitchA;       // bytes between rows of a shrink tile (KP*2, +64 when rows are copied one by one)
  int ER, er_shift; // out rows per expand tile (power of two, 32..256)
  int oc[B200_LORA_MAX_SLICES];  // out rows of each slice owned by one CTA (multiple of 32)
  int stage_bytes, NS;
  int red_pitch;    // floats per token row of the cross-warp reduction buffer
  int pitchT;       // bytes per token row of tmp
  int kind;
  int off_red, off_tmp, off_tab, off_bar;
  int full_k;       // every K part has all 1024 columns
  int y_cols;       // columns of y that the slices may touch (largest column end)
  int ksplit;       // 1: the K parts (not the rank rows) are dealt over the CTAs of a cluster
  int pitchR, off_recv;  // K split: floats per token row of the received partial sums
  int use_pdl;
  int mode;         // 0 fused, 1 shrink only (tmp_io written), 2 expand only (tmp_io read), 3 overwrite y
  void* tmp_io;
  int io16, zero_rows, no_add, gate;
  const int32_t* token_to_slot;
};

__host__ __device__ __forceinline__ int ceil_div_i(int a, int b) { return (a + b - 1) / b; }
__host__ __device__ __forceinline__ int round_up_i(int a, int b) { return ceil_div_i(a, b) * b; }

// mode 3: rows that get no delta (no adapter, unknown slot, adapter of rank 0) are set to -0.0 over the
// columns of all slices; the rows are dealt over the CTAs of the grid, `nthreads` threads of each taking part.
__device__ __forceinline__ void bgmv_fill_rows_without_delta(const BgmvParams& p, int cta, int n_ctas, int thread, int nthreads) {
  const uint4 negz = make_uint4(0x80008000u, 0x80008000u, 0x80008000u, 0x80008000u);
  for (int row = cta; row < p.T; row += n_ctas) {
    const int sl = p.token_to_slot[row];
    bool dead = sl < 0 || sl >= p.S;
    if (!dead && p.rank_per_slot != nullptr) dead = p.rank_per_slot[sl] <= 0;
    if (!dead) continue;
#pragma unroll
    for (int s = 0; s < B200_LORA_MAX_SLICES; ++s) {
      if (s < p.st.n) {
        __nv_bfloat16* dst = p.y + (int64_t)row * p.y_ld + p.st.col[s];
        for (int i = thread; i < (p.st.out[s] >> 3); i += nthreads) stg128(dst + 8 * i, negz);
      }
    }
  }
}

// mode 1 with zero_rows: rows without adapter of the intermediate [n, T, r_max], dealt as above
__device__ __forceinline__ void bgmv_zero_rows_without_adapter(const BgmvParams& p, int cta, int n_ctas, int thread, int nthreads) {
  const int vecs = (p.r_max * (p.io16 ? 2 : 4)) >> 4;  // 16-byte pieces of a row
  for (int row = cta; row < p.T; row += n_ctas) {
    const int sl = p.token_to_slot[row];
    if (sl >= 0 && sl < p.S) continue;
    for (int i = thread; i < p.st.n * vecs; i += nthreads) {
      const int s = i / vecs;
      stg128(static_cast<uint8_t*>(p.tmp_io) + (((int64_t)s * p.T + row) * vecs + (i - s * vecs)) * 16, make_uint4(0, 0, 0, 0));
    }
  }
}

// Two CTAs per SM: the CTAs of the next launch of the stream become resident while this launch still
// runs, so their weight copies overlap this launch's dependent chain.
#ifndef BGMV_MINBLOCKS
#define BGMV_MINBLOCKS 2
#endif
// kMode = BgmvParams::mode, compiled separately so that no path carries the branches of another;
// kFullK = every K part has all 1024 columns (in_dim a multiple of 1024): no column checks in the shrink
// kKind = BgmvProblem::kind; kWide = r_max > 32: output tiles are less than 256 rows high (in kind 0 the intermediate of a slice
// has more than one block of 32 columns)
// block_y / blocks_y: this CTA's bucket index and their number (a launch may carry other work beside the buckets)
template <int kMode, bool kFullK, int kKind, bool kWide>
__device__ __forceinline__ void bgmv_body(const BgmvParams& p, uint8_t* smem, const int block_y, const int blocks_y) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  int bucket = block_y;
  const int C = 1 << p.c_shift;
  const int c = (int)cluster_ctarank();
  const int NS = p.NS;
  constexpr bool kF32Out = kMode == 4, kOverwrite = kMode == 3;
  constexpr bool kPrecise = kKind != 0, kF16 = kKind == 2;
  constexpr bool kBlocks = kPrecise && !kF32Out;  // adds that read y
  constexpr int mode = kMode;

  B200_TRACE_POINT(0)
  // Let the next launch of the stream start at once: before its own griddepcontrol.wait it only
  // reads index metadata and lora slabs, which no kernel of this library writes, so its weight
  // traffic overlaps this kernel's compute and keeps HBM busy across launch boundaries.
  if (p.use_pdl) griddep_launch_dependents();
  if ((kMode == 1 || kMode == 2) && p.gate && !rows_scattered(p.token_to_slot, p.T)) {
    if (p.use_pdl && block_y == 0 && c == 0) griddep_wait();
    return;
  }
  // ---- bucket metadata (uniform across the cluster); barrier set-up overlaps the loads
  // Extra cluster e looks after multiple m = (e + 1) * 16 inside the sorted rows: if m lies behind the
  // first row of a bucket [start, start + cnt), it is the i-th such multiple there, and the cluster takes the bucket's i-th
  // window. (A bucket of cnt rows has ceil(cnt / 16) - 1 windows beyond its first and at least that many multiples.)
  int window_no = 0;
  if (p.by_window) {
    // Fewer rows than buckets (graph buffers carry a bucket for every slot): the launch has a cluster for every window that T
    // rows can make, and cluster i takes the i-th one. (A cluster per bucket cost 64 rows over 128 adapters two waves of CTAs
    // that only found no rows.)
    int seen = 0;
    bucket = -1;
    for (int b0 = 0; b0 < p.n_buckets && bucket < 0; b0 += 128) {
      int held[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) held[i] = b0 + 32 * i + lane < p.n_buckets ? p.counts[b0 + 32 * i + lane] : 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int windows = held[i] > 0 && held[i] <= p.T ? (held[i] + kBgmvTok - 1) / kBgmvTok : 0;
        int upto = windows;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
          const int v = __shfl_up_sync(0xffffffffu, upto, d);
          if (lane >= d) upto += v;
        }
        const int first = seen + upto - windows;
        const unsigned mine = __ballot_sync(0xffffffffu, block_y >= first && block_y < first + windows);
        if (mine != 0) {
          bucket = b0 + 32 * i + __ffs((int)mine) - 1;
          window_no = block_y - __shfl_sync(0xffffffffu, first, __ffs((int)mine) - 1);
        }
        seen = __shfl_sync(0xffffffffu, seen + upto, 31);
      }
    }
  } else if (bucket >= p.n_buckets) {
    // (every warp looks for itself: most of these clusters find nothing, and the sooner they leave, the sooner the next launch
    // has their place)
    const int m = (bucket - p.n_buckets + 1) * kBgmvTok;
    bucket = -1;
    for (int b0 = 0; b0 < p.n_buckets && bucket < 0; b0 += 128) {
      int lo[4], cnt4[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int b = b0 + 32 * i + lane;
        lo[i] = b < p.n_buckets ? p.offsets[b] : m;
        cnt4[i] = b < p.n_buckets ? p.counts[b] : 0;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const unsigned mine = __ballot_sync(0xffffffffu, lo[i] < m && m - lo[i] < cnt4[i]);
        if (mine != 0) {
          const int owner = __ffs((int)mine) - 1;
          bucket = b0 + 32 * i + owner;
          window_no = m / kBgmvTok - __shfl_sync(0xffffffffu, lo[i], owner) / kBgmvTok;
        }
      }
    }
    if (bucket < 0) {
      if (p.use_pdl && (kOverwrite || (kMode == 1 && p.zero_rows))) griddep_wait();
      if (kMode == 1 && p.zero_rows) bgmv_zero_rows_without_adapter(p, block_y * C + c, blocks_y * C, tid, kBgmvThreads);
      if (kOverwrite) bgmv_fill_rows_without_delta(p, block_y * C + c, blocks_y * C, tid, kBgmvThreads);
      return;
    }
  }
  const int slot = bucket >= 0 ? p.slot_ids[bucket] : -1;
  const int rows_all = bucket >= 0 ? p.counts[bucket] : 0, start_all = bucket >= 0 ? p.offsets[bucket] : 0;
  const int cnt = min(kBgmvTok, rows_all - window_no * kBgmvTok);
  const int start = start_all + window_no * kBgmvTok;

  float* red = reinterpret_cast<float*>(smem + p.off_red);
  uint8_t* tmp_base = smem + p.off_tmp;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + p.off_bar);  // full[], empty[], tmp_ready
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * kBgmvMaxStages + 1);
  const uint32_t bar_base = smem_u32(bars);
  const uint32_t ring_base = smem_u32(smem);
  const uint32_t tmp_ready_bar = bar_base + 8u * (uint32_t)(2 * kBgmvMaxStages);
  auto full_bar = [&](int s) { return bar_base + 8u * (uint32_t)s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (uint32_t)(kBgmvMaxStages + s); };

  int rank = p.r_max;
  if (p.rank_per_slot != nullptr && slot >= 0 && slot < p.S) rank = min(max(p.rank_per_slot[slot], 0), p.r_max);
  const int r_eff = min(p.r_max, kPrecise ? (rank + 15) & ~15 : (rank + 31) & ~31);
  // (a bucket whose row range leaves the batch is ignored; the bounds-checked build reports it)
  if (cnt > 0 && slot >= 0) (void)B200_IN_BOUNDS(slot < p.S && start_all >= 0 && start_all <= p.T - rows_all);
  if (slot < 0 || slot >= p.S || cnt <= 0 || start_all < 0 || start_all > p.T - rows_all || r_eff == 0) {
    // An idle cluster holds nothing, but one CTA of every launch must outlive the previous launch
    // of the stream: a launch that ended before its predecessor would let the launch behind it
    // pass its own wait too early.
    if (p.use_pdl && (kOverwrite || (kMode == 1 && p.zero_rows) || (block_y == 0 && c == 0))) griddep_wait();
    if (kMode == 1 && p.zero_rows) bgmv_zero_rows_without_adapter(p, block_y * C + c, blocks_y * C, tid, kBgmvThreads);
    if (kOverwrite)  // an idle cluster still does its share of the -0.0 rows
      bgmv_fill_rows_without_delta(p, block_y * C + c, blocks_y * C, tid, kBgmvThreads);
    return;
  }
  if (tid < NS) {
    mbar_init(full_bar(tid), 1);
    mbar_init(empty_bar(tid), kBgmvWarps);
    if (tid == 0) {
      mbar_init(tmp_ready_bar, 1u);  // completed by byte count (st.async from every CTA of the cluster)
      *abort_flag = 0;
    }
    mbar_fence_init();
  }
  const float sc = p.scaling * (p.scale_per_slot != nullptr ? p.scale_per_slot[slot] : 1.0f);
  B200_TRACE_POINT(1)

  const int n = p.st.n;
  const int in_dim = p.in_dim;
  const int Q = n * r_eff;                                       // stacked rank rows
  // Shrink work of the cluster: either the rank rows are split over the CTAs (each takes all K parts of
  // its rows, the bf16 results are all-gathered), or - long input rows - the K parts are dealt over the
  // CTAs (each takes all rank rows of its K parts, the fp32 partial sums are exchanged and added).
  const bool ksplit = (kMode == 0 || kMode >= 3) && p.ksplit != 0;
  const int Rc = ksplit ? Q : ((((Q + C - 1) >> p.c_shift) + 7) & ~7);  // rows owned per CTA
  const int q_lo = ksplit ? 0 : min(c * Rc, Q);
  const int rows_c = mode == 2 ? 0 : min(q_lo + Rc, Q) - q_lo;   // multiple of 8, may be 0 (expand only: no shrink rows)
  const int nt_c = rows_c >> 3;                                  // 8-row tiles of this CTA
  const int KP = p.KP, pitchA = p.pitchA, ER = p.ER, nkp = p.nkp;
  const int kp0 = ksplit ? c : 0, kstep = ksplit ? C : 1;        // K parts of this CTA: kp0, kp0 + kstep, ...
  const int nkp_c = ksplit ? (nkp > c ? (nkp - c + C - 1) >> p.c_shift : 0) : nkp;
  const int shrink_tiles = nt_c * nkp_c;
  int e_lo[B200_LORA_MAX_SLICES], e_n[B200_LORA_MAX_SLICES], e_tiles[B200_LORA_MAX_SLICES];
  int tiles_exp = 0;
#pragma unroll
  for (int s = 0; s < B200_LORA_MAX_SLICES; ++s) {
    e_lo[s] = e_n[s] = e_tiles[s] = 0;
    if (s < n && mode != 1) {  // (shrink only: no expand tiles)
      const int out = p.st.out[s];
      e_lo[s] = min(c * p.oc[s], out);
      e_n[s] = min(e_lo[s] + p.oc[s], out) - e_lo[s];
      e_tiles[s] = (e_n[s] + ER - 1) >> p.er_shift;
      tiles_exp += e_tiles[s];
    }
  }
  const int total = shrink_tiles + tiles_exp;
  // bytes delivered into this CTA: 16 token rows of all Q stacked rank rows, as bf16 once
  // (all-gather) or as fp32 from every CTA of the cluster (K split)
  if (tid == 0 && (mode == 0 || mode >= 3))
    mbar_arrive_expect_tx(tmp_ready_bar, ksplit ? (uint32_t)(C * kBgmvTok * Q * 4) : (uint32_t)(kBgmvTok * Q * (kPrecise ? 4 : 2)));

  __syncthreads();  // barriers initialised
  B200_TRACE_POINT(2)
  // Start-up cluster barrier: every CTA of the cluster has initialised its barriers once it
  // completes. Consumers wait on it before their first remote store, the producer before it exits.
  cluster_arrive();

  if (warp == kBgmvWarps) {
    // =========================== producer warp ===========================
    int i_shrink = shrink_tiles > 0 ? 1 : 0, i_kp = 0, i_j = 0;  // cursor: phase, K part, 8-row tile
    int i_s = 0, i_et = 0;                                       // cursor: slice / tile in slice
    int i_qs = 0, i_qr = q_lo;                                   // slice / row of the cursor's first rank row
    while (i_qr >= r_eff) { i_qr -= r_eff; ++i_qs; }
    const int q0_s = i_qs, q0_r = i_qr;
    int p_stage = 0, p_round = 0;
    const int npro = min(NS, total);
#pragma unroll 1
    for (int it = 0; it < total; ++it) {
      if (p_round > 0) mbar_wait_bounded(empty_bar(p_stage), (uint32_t)((p_round & 1) ^ 1), abort_flag);
      const uint32_t sbase = ring_base + (uint32_t)p_stage * (uint32_t)p.stage_bytes;
      const uint32_t fb = full_bar(p_stage);
      if (i_shrink) {
        const int k0 = (kp0 + i_kp * kstep) * KP;
        const uint32_t row_bytes = (uint32_t)min(KP, in_dim - k0) * 2u;
        const void* aptr = nullptr;
#pragma unroll
        for (int s = 0; s < B200_LORA_MAX_SLICES; ++s)
          if (s == i_qs) aptr = p.st.a[s];
        const __nv_bfloat16* src =
            static_cast<const __nv_bfloat16*>(aptr) + ((int64_t)slot * p.r_max + i_qr) * in_dim + k0;
        // 8 rank rows of slice i_qs, columns [k0, k0 + row_bytes / 2), into stage p_stage
        if (!B200_IN_BOUNDS(aptr != nullptr && i_qs < n && i_qr + 8 <= p.r_max && k0 < in_dim && p_stage < NS &&
                            8 * pitchA <= p.stage_bytes)) {
          if (lane == 0) mbar_arrive(fb);  // the tile is skipped; its consumers see stale bytes, never a stuck barrier
        } else
        if (nkp == 1) {
          // the 8 rows are contiguous in the slab: one copy (each copy costs the TMA unit ~100 cycles)
          if (lane == 0) {
            mbar_arrive_expect_tx(fb, 8u * row_bytes);
            bulk_g2s(sbase, src, 8u * row_bytes, fb);
          }
        } else {
          if (lane == 0) mbar_arrive_expect_tx(fb, 8u * row_bytes);
          __syncwarp();
          if (lane < 8) bulk_g2s(sbase + (uint32_t)(lane * pitchA), src + (int64_t)lane * in_dim, row_bytes, fb);
        }
        // advance: 8-row tiles inner, K parts outer
        ++i_j;
        i_qr += 8;
        if (i_qr >= r_eff) { i_qr = 0; ++i_qs; }
        if (i_j == nt_c) {
          i_j = 0; i_qs = q0_s; i_qr = q0_r;
          if (++i_kp == nkp_c) i_shrink = 0;
        }
      } else {
#pragma unroll
        for (int s = 0; s < B200_LORA_MAX_SLICES - 1; ++s)  // skip slices this CTA has no tiles of
          if (i_s == s && i_et >= e_tiles[s]) { i_s = s + 1; i_et = 0; }
        int lo = 0, en = 0, out = 0;
        const void* bptr = nullptr;
#pragma unroll
        for (int s = 0; s < B200_LORA_MAX_SLICES; ++s)
          if (s == i_s) { lo = e_lo[s]; en = e_n[s]; out = p.st.out[s]; bptr = p.st.b[s]; }
        const int r0 = i_et << p.er_shift;
        const int nrows = min(ER, en - r0);
        if (!B200_IN_BOUNDS(bptr != nullptr && nrows > 0 && lo + r0 + nrows <= out && p_stage < NS &&
                            nrows * p.r_max * 2 <= p.stage_bytes)) {
          if (lane == 0) mbar_arrive(fb);
        } else
        if (lane == 0) {
          const uint32_t bytes = (uint32_t)nrows * (uint32_t)p.r_max * 2u;
          mbar_arrive_expect_tx(fb, bytes);
          const __nv_bfloat16* src =
              static_cast<const __nv_bfloat16*>(bptr) + ((int64_t)slot * out + lo + r0) * p.r_max;
          bulk_g2s(sbase, src, bytes, fb);
        }
        ++i_et;
      }
      __syncwarp();
      if (++p_stage == NS) { p_stage = 0; ++p_round; }
      if (it + 1 == npro) { B200_TRACE_PRODUCER(3) }
      // (What the ring cannot hold is not prefetched to the L2 either: on top of a full ring on every SM it only queued in
      // front of the copies that are waited for. Without it 200 rows over 128 adapters, 2048-wide: 17.1 -> 14.2 us, 256 rows
      // over 32: 4.91 -> 4.79.)
    }
    cluster_wait();
    return;
  }

  // ============================= consumer warps =============================
  // Everything that does not depend on the previous launch of the stream is done before the wait:
  // token rows, the table of this CTA's expand tiles, thread-constant address pieces and L2 prefetches of x
  // (a prefetch never creates stale data: L2 is the point of coherence). What runs after the wait is
  // the dependent chain activations -> shrink -> all-gather -> expand, kept as short as possible.
  int tok_lo = -1, tok_hi = -1;
  if (g < cnt) tok_lo = p.sorted_idx[start + g];
  if (g + 8 < cnt) tok_hi = p.sorted_idx[start + g + 8];
  (void)B200_IN_BOUNDS(tok_lo < p.T && tok_hi < p.T && tok_lo >= -1 && tok_hi >= -1);
  if (tok_lo >= p.T) tok_lo = -1;
  if (tok_hi >= p.T) tok_hi = -1;

  // Expand rows of this CTA in blocks of 32 (ring order), dealt to the warps in turn: warp w multiplies blocks w, w + 8, ..., so that
  // tiles of fewer than 256 rows are multiplied side by side. (With every tile from warp 0 on, k and v cost a step each while seven
  // warps waited; us a launch, before / now: 1024-wide, rank 32, qkv of 256 rows over 32 adapters 4.58 / 4.24, of 4 rows 2.96 / 2.57;
  // rank 64, a step of two tiles with every warp waiting for both: 2048-wide, 48 over 64, gate_up 12.4 / 11.7; 4096-wide, 512 over
  // 88, o 29.5 / 25.2.)
  // Kind 0, and mode 4: a table of the tiles, x = first y column, y = rows | slice << 16 | warp of the first block << 20. Kinds 1 and 2 ask for a
  // block's y while they multiply the block before, which may lie several tiles back: a table of the blocks, x = first y column, y =
  // rows | slice << 8 | block of its tile << 12 | tile << 16. (Asked for a tile ahead, the y of narrow slices, at ranks above 32 all
  // of it, came late: us a layer, by tile / by block: fp16, rank 64, 128 rows over 32 adapters, 1024-wide 36.8 / 34.5, 4096-wide 90.5
  // / 83.7; bf16, rank 48, 256 rows 34.6 / 30.5; rank 16, 37 rows 13.3 / 12.8. Kind 0 with the longer table loses up to 1 %, and
  // so do projections beside a GEMM of kind 1, which read no y: a step of four layers at rank 16, 128 rows over 100 adapters, by block / by
  // tile, 1024-wide 241.3 / 237.2, 2048-wide 359.7 / 353.9.)
  int2* etab = reinterpret_cast<int2*>(smem + p.off_tab);
  int entries = tiles_exp;
  if (kBlocks) {
    entries = 0;
#pragma unroll
    for (int s = 0; s < B200_LORA_MAX_SLICES; ++s) entries += (e_n[s] + 31) >> 5;
  }
#pragma unroll 1
  for (int i = tid; i < entries; i += kBgmvConsumers) {
    int s_e = 0, r0 = kBlocks ? i << 5 : i << p.er_shift, tile = 0, blocks = 0;  // slice, first row in it; tiles and blocks of those before
#pragma unroll
    for (int s = 0; s < B200_LORA_MAX_SLICES - 1; ++s)
      if (s_e == s && r0 >= e_n[s]) {
        r0 -= kBlocks ? (e_n[s] + 31) & ~31 : e_tiles[s] << p.er_shift;
        tile += e_tiles[s];
        blocks += (e_n[s] + 31) >> 5;
        s_e = s + 1;
      }
    int lo = 0, en = 0, cb = 0;
#pragma unroll
    for (int s = 0; s < B200_LORA_MAX_SLICES; ++s)
      if (s == s_e) { lo = e_lo[s]; en = e_n[s]; cb = p.st.col[s]; }
    if (kBlocks)
      etab[i] = make_int2(cb + lo + r0, min(32, en - r0) | (s_e << 8) | (((r0 & (ER - 1)) >> 5) << 12) | ((tile + (r0 >> p.er_shift)) << 16));
    else
      etab[i] = make_int2(cb + lo + r0, min(ER, en - r0) | (s_e << 16) | (((blocks + (r0 >> 5)) & (kBgmvWarps - 1)) << 20));
  }
  if (kBlocks && tid < kBgmvWarps) etab[entries + tid] = make_int2(0, -65536);  // (no rows, of no tile: behind the last block of a warp)
  named_bar_sync(1, kBgmvConsumers);  // table complete

  const int x_col = warp * 32 + t * 8;  // shrink: first column of the thread inside a K part (block i adds 256)
  if (p.use_pdl) {
#pragma unroll 1
    for (int ikp = 0; ikp < (rows_c > 0 ? nkp_c : 0); ++ikp) {
      const int k0 = (kp0 + ikp * kstep) * KP;
#pragma unroll 1
      for (int kc = k0 + x_col; kc < min(k0 + KP, in_dim); kc += kBgmvWarps * 32) {
        if (tok_lo >= 0) prefetch_l2(p.x + (int64_t)tok_lo * p.x_ld + kc);
        if (tok_hi >= 0) prefetch_l2(p.x + (int64_t)tok_hi * p.x_ld + kc);
      }
    }
  }

  // thread-constant pieces of the shared-memory addresses
  const uint32_t pitchB = (uint32_t)p.r_max * 2u;
  const uint32_t a_off = (uint32_t)(g * pitchA + x_col * 2);                            // shrink tile: row g
  const uint32_t w_off = (uint32_t)(8 * (g >> 1) + (g & 1)) * pitchB + (uint32_t)t * (kPrecise ? 8u : 16u);  // expand tile
  // MMA column n of n-tile j reads slab row 8*(n/2) + 2j + (n%2) of the warp's 32 rows: thread (g,t)
  // then owns 8 consecutive output columns 8t..8t+7 of the block.
  const uint32_t t_off = (uint32_t)(g * p.pitchT + t * 16);                             // tmp: token row g
  float* const red_wr = red + ((size_t)warp * kBgmvTok + g) * p.red_pitch + 2 * t;      // + 8 * pitch: token g + 8
  // expand: 32-column blocks of the intermediate; kinds 1 and 2 keep it as groups [four high halves | four low halves], 16 columns
  // a block, so that a 16-byte fragment is both halves of four columns and the weights are read once
  const int kblocks = kPrecise ? r_eff >> 4 : r_eff >> 5;
  // all-gather item of this thread: one token row x four consecutive rank rows of this CTA
  const int groups = rows_c >> 2;
  const bool has_item = tid < kBgmvTok * groups;
  const int it_tok = has_item ? tid / max(groups, 1) : 0;
  const int it_q = q_lo + 4 * (has_item ? tid - it_tok * groups : 0);
  const float* const red_rd = red + (size_t)it_tok * p.red_pitch + (it_q - q_lo);
  const uint32_t it_off = (uint32_t)(it_tok * p.pitchT + it_q * (kPrecise ? 4 : 2));
  const uint32_t tmp_u32 = smem_u32(tmp_base);
  // row of the intermediate that this thread writes / reads (looked up here, not on the chain behind the wait: 0.4 us)
  int io_row = -1;
  if (kMode == 1 && has_item && it_tok < cnt) io_row = p.sorted_idx[start + it_tok];
  if (kMode == 2 && (tid >> 4) < cnt) io_row = p.sorted_idx[start + (tid >> 4)];
  if (io_row >= p.T) io_row = -1;

  if (p.use_pdl) griddep_wait();  // x and y of this launch are final from here on
  if (kOverwrite) bgmv_fill_rows_without_delta(p, block_y * C + c, blocks_y * C, tid, kBgmvConsumers);
  if (kMode == 1 && p.zero_rows) bgmv_zero_rows_without_adapter(p, block_y * C + c, blocks_y * C, tid, kBgmvConsumers);
  B200_TRACE_POINT(4)

  int c_stage = 0;
  uint32_t c_parity = 0, stage_addr = ring_base;  // stage being consumed: index, phase, address
  auto advance = [&]() {
    stage_addr += (uint32_t)p.stage_bytes;
    if (++c_stage == NS) { c_stage = 0; c_parity ^= 1u; stage_addr = ring_base; }
  };

  __nv_bfloat16* const ylo_p = p.y + (int64_t)max(tok_lo, 0) * p.y_ld + 8 * t;  // + first column of the warp's block
  __nv_bfloat16* const yhi_p = p.y + (int64_t)max(tok_hi, 0) * p.y_ld + 8 * t;
  // kinds 1 and 2: y of a warp's next block is requested while it multiplies the one before, the first one behind the shrink
  // (its 0.5 us of latency then lie beside the exchange: 37 rows, rank 16 74.1 -> 70.9 us a layer stack, 64 rows fp16 43.5 -> 40.7; before the
  // shrink it delays the x loads: 76.0 and 45.0)
  uint4 y_next[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
  auto load_y = [&](int2 block) {
    if (kF32Out || (kMode == 2 && p.no_add)) return;
    if (8 * t >= (block.y & 0xff) || !B200_IN_BOUNDS(block.x >= 0 && block.x + 8 * t + 8 <= p.y_cols)) return;
    if (tok_lo >= 0) y_next[0] = ldg128(ylo_p + block.x);
    if (tok_hi >= 0) y_next[1] = ldg128(yhi_p + block.x);
  };
  const int2* block_at = etab + warp;
  int2 block_next = make_int2(0, 0);  // of this warp
  if (kBlocks) block_next = *block_at;
  const __nv_bfloat16* const xlo_p = p.x + (int64_t)max(tok_lo, 0) * p.x_ld + x_col;
  const __nv_bfloat16* const xhi_p = p.x + (int64_t)max(tok_hi, 0) * p.x_ld + x_col;

  // ===== shrink: red[warp][tok][row] = x[16 tok, K blocks of this warp] . A_rows^T =====
#pragma unroll 1
  for (int kp = 0; kp < (rows_c > 0 ? nkp_c : 0); ++kp) {
    const int k0 = (kp0 + kp * kstep) * KP;
    // activation fragments of this warp's 32-column blocks, kept for all row tiles
    uint4 xlo[kBgmvXBlocks], xhi[kBgmvXBlocks];
#pragma unroll
    for (int i = 0; i < kBgmvXBlocks; ++i) {
      xlo[i] = xhi[i] = make_uint4(0, 0, 0, 0);
      if (kFullK || (x_col + 256 * i < KP && k0 + x_col + 256 * i < in_dim)) {
        if (tok_lo >= 0) xlo[i] = ldg128_nc(xlo_p + k0 + 256 * i);
        if (tok_hi >= 0) xhi[i] = ldg128_nc(xhi_p + k0 + 256 * i);
      }
    }
    // kTiles (1 or 2) 8-row tiles of the ring against the warp's activation fragments: all loads
    // first, then the independent MMA chains of both tiles, then the stores; sums of the K blocks go
    // to the warp's rows of the reduction buffer (added to what earlier K parts left there)
    auto shrink_tiles_fn = [&](auto n_tiles, int j, uint32_t addr0, uint32_t addr1) {
      constexpr int kTiles = decltype(n_tiles)::value;
      float acc[kTiles][2][4];
#pragma unroll
      for (int u = 0; u < kTiles; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) acc[u][h][0] = acc[u][h][1] = acc[u][h][2] = acc[u][h][3] = 0.f;
#pragma unroll
      for (int i = 0; i < kBgmvXBlocks; ++i) {
        uint4 w[kTiles];
#pragma unroll
        for (int u = 0; u < kTiles; ++u) {
          w[u] = make_uint4(0, 0, 0, 0);
          if (kFullK || (x_col + 256 * i < KP && k0 + x_col + 256 * i < in_dim))
            w[u] = lds128((u == 0 ? addr0 : addr1) + a_off + 512u * i);
        }
#pragma unroll
        for (int u = 0; u < kTiles; ++u) {
          mma_16816<kF16>(acc[u][0], xlo[i].x, xhi[i].x, xlo[i].y, xhi[i].y, w[u].x, w[u].y);
          mma_16816<kF16>(acc[u][1], xlo[i].z, xhi[i].z, xlo[i].w, xhi[i].w, w[u].z, w[u].w);
        }
      }
#pragma unroll
      for (int u = 0; u < kTiles; ++u) {
        // acc holds (tok g | g+8, rank rows 8(j+u)+2t, 8(j+u)+2t+1)
        float2* r0 = reinterpret_cast<float2*>(red_wr + 8 * (j + u));
        float2* r1 = reinterpret_cast<float2*>(red_wr + 8 * p.red_pitch + 8 * (j + u));
        float2 a = make_float2(0.f, 0.f), b = a;
        if (kp != 0) { a = *r0; b = *r1; }
        *r0 = make_float2(a.x + acc[u][0][0] + acc[u][1][0], a.y + acc[u][0][1] + acc[u][1][1]);
        *r1 = make_float2(b.x + acc[u][0][2] + acc[u][1][2], b.y + acc[u][0][3] + acc[u][1][3]);
      }
    };
    int j = 0;
#pragma unroll 1
    for (; j + 1 < nt_c; j += 2) {
      const int s0 = c_stage;
      const uint32_t a0 = stage_addr;
      mbar_wait_bounded(full_bar(s0), c_parity, abort_flag);
      if (kp == 0 && j == 0) { B200_TRACE_POINT(5) }
      advance();
      const int s1 = c_stage;
      const uint32_t a1 = stage_addr;
      mbar_wait_bounded(full_bar(s1), c_parity, abort_flag);
      advance();
      shrink_tiles_fn(std::integral_constant<int, 2>{}, j, a0, a1);
      __syncwarp();
      if (lane == 0) {
        mbar_arrive_relaxed(empty_bar(s0));
        mbar_arrive_relaxed(empty_bar(s1));
      }
    }
#pragma unroll 1
    for (; j < nt_c; ++j) {
      mbar_wait_bounded(full_bar(c_stage), c_parity, abort_flag);
      if (kp == 0 && j == 0) { B200_TRACE_POINT(5) }
      shrink_tiles_fn(std::integral_constant<int, 1>{}, j, stage_addr, stage_addr);
      __syncwarp();
      if (lane == 0) mbar_arrive_relaxed(empty_bar(c_stage));
      advance();
    }
  }
  B200_TRACE_POINT(6)
  if (kBlocks) load_y(block_next);

  // ===== cross-warp reduction of the K slices, scale, bf16, all-gather =====
  named_bar_sync(1, kBgmvConsumers);
  B200_TRACE_POINT(7)
  cluster_wait();  // start-up barrier: peers run and their barriers are initialised
  if (mode == 2) {
    // expand only: tmp comes from global memory (fp32 [n, T, r_max], summed over the
    // tensor-parallel ranks) and is rounded to bf16 into this CTA's own buffer
    const int tok = tid >> 4, trow = io_row;
#pragma unroll 1
    for (int pr = tid & 15; pr < (Q >> 1); pr += 16) {
      const int q = 2 * pr, s = q / r_eff, rr = q - s * r_eff;
      const int64_t at = ((int64_t)s * p.T + trow) * p.r_max + rr;
      uint32_t* const dst = reinterpret_cast<uint32_t*>(tmp_base + (size_t)tok * p.pitchT + (size_t)(kPrecise ? (q >> 2) * 16 + (q & 3) * 2 : q * 2));
      if (p.io16) {
        *dst = trow >= 0 ? *reinterpret_cast<const uint32_t*>(static_cast<const uint16_t*>(p.tmp_io) + at) : 0u;
        if (kPrecise) dst[2] = 0u;
      } else {
        float2 v = make_float2(0.f, 0.f);
        if (trow >= 0) v = *reinterpret_cast<const float2*>(static_cast<const float*>(p.tmp_io) + at);
        const uint32_t h = pack_16x2<kF16>(v.x, v.y);
        *dst = h;
        if (kPrecise) dst[2] = pack_rest<kF16>(v.x, v.y, h);
      }
    }
    named_bar_sync(1, kBgmvConsumers);
  } else {
    if (has_item) {
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < kBgmvWarps; ++w) {
        const float4 v = *reinterpret_cast<const float4*>(red_rd + (size_t)w * kBgmvTok * p.red_pitch);
        a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
      }
      if (mode == 1) {
        // shrink only: fp32 result of this CTA's rank rows straight to global memory
        const int trow = io_row;
        if (trow >= 0) {
          const int s = it_q / r_eff, rr = it_q - s * r_eff;
          const int64_t at = ((int64_t)s * p.T + trow) * p.r_max + rr;
          if (p.io16) {
            *reinterpret_cast<uint2*>(static_cast<uint16_t*>(p.tmp_io) + at) =
                make_uint2(pack_16x2<kF16>(a.x * sc, a.y * sc), pack_16x2<kF16>(a.z * sc, a.w * sc));
          } else {
            float2* dst = reinterpret_cast<float2*>(static_cast<float*>(p.tmp_io) + at);
            dst[0] = make_float2(a.x * sc, a.y * sc);
            dst[1] = make_float2(a.z * sc, a.w * sc);
          }
        }
      } else if (ksplit) {
        // to every CTA of the cluster (this one included): this CTA's fp32 partial sums over its K parts,
        // into the block the receiver keeps for this sender
        const uint32_t dst = smem_u32(smem + p.off_recv) + (uint32_t)((c * kBgmvTok + it_tok) * p.pitchR + it_q) * 4u;
#pragma unroll 1
        for (int rc = 0; rc < C; ++rc)
          st_async_f32x4(mapa_shared(dst, (uint32_t)rc), a, mapa_shared(tmp_ready_bar, (uint32_t)rc));
      } else {
        // to every CTA of the cluster (this one included): 8 bytes of tmp + their count on the
        // receiver's barrier in one operation
        const uint32_t v0 = pack_16x2<kF16>(a.x * sc, a.y * sc), v1 = pack_16x2<kF16>(a.z * sc, a.w * sc);
        const uint32_t l0 = kPrecise ? pack_rest<kF16>(a.x * sc, a.y * sc, v0) : 0u, l1 = kPrecise ? pack_rest<kF16>(a.z * sc, a.w * sc, v1) : 0u;
#pragma unroll 1
        for (int rc = 0; rc < C; ++rc) {
          if (kPrecise) st_async_b32x4(mapa_shared(tmp_u32 + it_off, (uint32_t)rc), make_uint4(v0, v1, l0, l1), mapa_shared(tmp_ready_bar, (uint32_t)rc));
          else st_async_b32x2(mapa_shared(tmp_u32 + it_off, (uint32_t)rc), v0, v1, mapa_shared(tmp_ready_bar, (uint32_t)rc));
        }
      }
    }
    if (mode != 1) {
      B200_TRACE_POINT(8)
      mbar_wait_bounded_acquire_cluster(tmp_ready_bar, 0u, abort_flag);
      if (ksplit) {
        // add the C partial sums of this thread's item, scale, round: tmp, kept locally
        if (has_item) {
          float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
          const float* src = reinterpret_cast<const float*>(smem + p.off_recv) + (size_t)it_tok * p.pitchR + it_q;
#pragma unroll 1
          for (int rc = 0; rc < C; ++rc) {
            const float4 v = *reinterpret_cast<const float4*>(src + (size_t)rc * kBgmvTok * p.pitchR);
            a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
          }
          const uint32_t v0 = pack_16x2<kF16>(a.x * sc, a.y * sc), v1 = pack_16x2<kF16>(a.z * sc, a.w * sc);
          uint8_t* dst = tmp_base + it_off;
          if (kPrecise)
            *reinterpret_cast<uint4*>(dst) = make_uint4(v0, v1, pack_rest<kF16>(a.x * sc, a.y * sc, v0), pack_rest<kF16>(a.z * sc, a.w * sc, v1));
          else
            *reinterpret_cast<uint2*>(dst) = make_uint2(v0, v1);
        }
        named_bar_sync(1, kBgmvConsumers);
      }
      B200_TRACE_POINT(9)
    }
  }

  // ===== expand: y[tok, cols] += tmp[16 tok, r] . B_rows^T ======================
  // Rows of a block beyond the tile's rows hold stale bytes; their products land in columns that are not written.
  uint4 a_lo = make_uint4(0, 0, 0, 0), a_hi = a_lo;  // kind 0, ranks up to 32: the intermediate's fragments of the slice at hand
  int a_slice = -1;
  // this warp's `rows` rows of slice `slice`, from row `row` of the tile on, into y from column c0 on
  auto expand_fn = [&](const int c0, const int rows, const int slice, const int row, const uint4 y_lo, const uint4 y_hi) {
    float d[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) d[j][0] = d[j][1] = d[j][2] = d[j][3] = 0.f;
    const uint32_t a_addr = tmp_u32 + t_off + (uint32_t)(slice * r_eff * (kPrecise ? 4 : 2));
    const uint32_t w_addr = stage_addr + w_off + (uint32_t)row * pitchB;
    if constexpr (!kWide && !kPrecise) {
      uint4 w[4];  // (r_eff = r_max = 32: one block)
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = lds128(w_addr + 2u * j * pitchB);
      if (slice != a_slice) {
        a_slice = slice;
        a_lo = lds128(a_addr);
        a_hi = lds128(a_addr + 8u * (uint32_t)p.pitchT);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) mma_16816<kF16>(d[j], a_lo.x, a_hi.x, a_lo.y, a_hi.y, w[j].x, w[j].y);
#pragma unroll
      for (int j = 0; j < 4; ++j) mma_16816<kF16>(d[j], a_lo.z, a_hi.z, a_lo.w, a_hi.w, w[j].z, w[j].w);
    } else {
#pragma unroll 1
      for (int kb = 0; kb < kblocks; ++kb) {
        const uint32_t a_kb = a_addr + 64u * kb, w_kb = w_addr + (kPrecise ? 32u : 64u) * kb;
        const uint4 alo = lds128(a_kb);
        const uint4 ahi = lds128(a_kb + 8u * (uint32_t)p.pitchT);
        uint4 w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (kPrecise) {
            const uint2 four = lds64(w_kb + 2u * j * pitchB);
            w[j] = make_uint4(four.x, four.y, four.x, four.y);
          } else {
            w[j] = lds128(w_kb + 2u * j * pitchB);
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_16816<kF16>(d[j], alo.x, ahi.x, alo.y, ahi.y, w[j].x, w[j].y);
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_16816<kF16>(d[j], alo.z, ahi.z, alo.w, ahi.w, w[j].z, w[j].w);
      }
    }
    if (8 * t >= rows || !B200_IN_BOUNDS(c0 >= 0 && c0 + 8 * t + 8 <= p.y_cols)) return;
    if (kF32Out) {
      float* const yf = reinterpret_cast<float*>(p.y) + c0 + 8 * t;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int tok = h ? tok_hi : tok_lo;
        if (tok < 0) continue;
        float4* const dst = reinterpret_cast<float4*>(yf + (int64_t)tok * p.y_ld);
        dst[0] = make_float4(d[0][2 * h], d[0][2 * h + 1], d[1][2 * h], d[1][2 * h + 1]);
        dst[1] = make_float4(d[2][2 * h], d[2][2 * h + 1], d[3][2 * h], d[3][2 * h + 1]);
      }
      return;
    }
    if (kPrecise) {
      if (tok_lo >= 0)
        stg128(ylo_p + c0, make_uint4(add_16x2<kF16>(y_lo.x, d[0][0], d[0][1]), add_16x2<kF16>(y_lo.y, d[1][0], d[1][1]),
                                      add_16x2<kF16>(y_lo.z, d[2][0], d[2][1]), add_16x2<kF16>(y_lo.w, d[3][0], d[3][1])));
      if (tok_hi >= 0)
        stg128(yhi_p + c0, make_uint4(add_16x2<kF16>(y_hi.x, d[0][2], d[0][3]), add_16x2<kF16>(y_hi.y, d[1][2], d[1][3]),
                                      add_16x2<kF16>(y_hi.z, d[2][2], d[2][3]), add_16x2<kF16>(y_hi.w, d[3][2], d[3][3])));
      return;
    }
    const uint4 lo4 = make_uint4(pack_bf16x2(d[0][0], d[0][1]), pack_bf16x2(d[1][0], d[1][1]),
                                 pack_bf16x2(d[2][0], d[2][1]), pack_bf16x2(d[3][0], d[3][1]));
    const uint4 hi4 = make_uint4(pack_bf16x2(d[0][2], d[0][3]), pack_bf16x2(d[1][2], d[1][3]),
                                 pack_bf16x2(d[2][2], d[2][3]), pack_bf16x2(d[3][2], d[3][3]));
    if (kOverwrite) {
      if (tok_lo >= 0) stg128(ylo_p + c0, lo4);
      if (tok_hi >= 0) stg128(yhi_p + c0, hi4);
    } else {
      // The delta is rounded to bf16 and added to y by one 16-byte reduction at the L2: y never
      // travels to the SM and nothing waits for it. Each element of y receives exactly one
      // reduction per launch, so the result does not depend on their order.
      if (tok_lo >= 0) red_add_bf16x8(ylo_p + c0, lo4.x, lo4.y, lo4.z, lo4.w);
      if (tok_hi >= 0) red_add_bf16x8(yhi_p + c0, hi4.x, hi4.y, hi4.z, hi4.w);
    }
  };
#pragma unroll 1
  for (int e = 0; e < tiles_exp; ++e) {
    // (every warp waits for every tile: a wait that skipped phases of a stage could no longer tell them apart)
    const int2 te = kBlocks ? block_next : etab[e];
    const int row = kBlocks ? ((te.y >> 12) & 7) * 32 : ((warp - (te.y >> 20)) & (kBgmvWarps - 1)) * 32;
    const bool mine = kBlocks ? te.y >> 16 == e : row < (te.y & 0xffff);
    const uint4 y_lo = y_next[0], y_hi = y_next[1];
    if (kBlocks && mine) block_next = *(block_at += kBgmvWarps);
    mbar_wait_bounded(full_bar(c_stage), c_parity, abort_flag);
    if (e < 10) { B200_TRACE_POINT(12 + 2 * e) }
    if (mine) {
      if (kBlocks) load_y(block_next);
      if (kBlocks) expand_fn(te.x, te.y & 0xff, (te.y >> 8) & 15, row, y_lo, y_hi);
      else expand_fn(te.x + row, (te.y & 0xffff) - row, (te.y >> 16) & 15, row, y_lo, y_hi);
    }
    if (e < 10) { B200_TRACE_POINT(13 + 2 * e) }
    __syncwarp();
    if (lane == 0) mbar_arrive_relaxed(empty_bar(c_stage));
    advance();
  }
  B200_TRACE_POINT(10)
  B200_TRACE_POINT(11)
  if (tid == 0 && *abort_flag != 0) atomicOr(&g_b200_status, kStatusWaitGaveUp);
}

template <int kMode, bool kFullK, int kKind, bool kWide>
__global__ void __launch_bounds__(kBgmvThreads, BGMV_MINBLOCKS) bgmv_fused_kernel(const __grid_constant__ BgmvParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  bgmv_body<kMode, kFullK, kKind, kWide>(p, smem, (int)blockIdx.y, (int)gridDim.y);
}

// ------------------------------------------------------------------ host side
struct BgmvOptions {
  int cluster = 0;   // 0 = auto
  int pdl = 1;
  int ring_kb = 0;   // cap of the stage ring in KB (0 = default)
  int ksplit = 1;    // 1 = deal K parts over the cluster when the input rows are long enough (default)
};
inline BgmvOptions& bgmv_options() {
  static BgmvOptions o;
  return o;
}
// Default budget of one CTA: half of an SM's shared memory (228 KB minus 1 KB that the system keeps per
// resident CTA), so that a CTA of the next launch fits beside one of this launch.
constexpr int kBgmvSmemCoResident = (228 * 1024 - 2 * 1024) / 2;

inline bool aligned16(const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15u) == 0; }
inline int floor_pow2(int v) { int r = 1; while (r * 2 <= v) r *= 2; return r; }
inline int log2_exact(int v) { int s = 0; while ((1 << s) < v) ++s; return s; }

// How the CTAs of a cluster share the shrink: the rank rows (rc each, all K), or with input rows of at least one K part (1024
// columns) per CTA and all rank rows in one CTA the K parts, up to 20 KB of received partial sums (64 rank rows over 8 CTAs, 35
// KB: one layer of 4096, rank 64, 1 / 16 rows 45 / 60 us, with the row split 40 / 53). The shrink-only / expand-only pair keeps
// the row split. rc = 0: the rank rows are too many for C CTAs.
struct BgmvSplit { bool by_k; int rc; };
inline BgmvSplit bgmv_split(const BgmvProblem& b, int Q, int C) {
  const bool by_k = bgmv_options().ksplit && C > 1 && (b.mode == 0 || b.mode >= 3) && ceil_div_i(b.in_dim, kBgmvKP) >= C && Q <= kBgmvMaxRc &&
                    C * kBgmvTok * (Q + 4) * 4 <= 20 * 1024;
  const int rc = by_k ? Q : round_up_i(ceil_div_i(Q, C), 8);
  return {by_k, rc <= kBgmvMaxRc ? rc : 0};
}

// Cluster size for the active slices `st` of a problem.
inline int bgmv_cluster(const BgmvProblem& b, const SliceTable& st) {
  int C = 1;
  const int Q = st.n * b.r_max;
  // Buckets expected to hold rows: graph buffers carry one bucket per slot, most of them empty. With T rows dealt over nb buckets
  // about nb * (1 - exp(-T / nb)) are in use; a skewed popularity uses fewer and gives them more windows, which the host does not
  // see.
  const double nb = (double)b.n_buckets, rows = (double)std::max(b.T, 1);
  const double in_use = nb * (1.0 - std::exp(-rows / nb));
  if (b.mode == 1 || b.mode == 2) {
    int64_t bucket_bytes = 0;
    for (int s = 0; s < st.n; ++s) bucket_bytes += 2 * (int64_t)b.r_max * ((int64_t)b.in_dim + st.out[s]);
    const double kb = (double)bucket_bytes / 1024.0 * std::max(1.0, 32.0 / b.r_max);  // (16 rank rows take as long as 32)
    // A shrink or an expand alone, which take turns: 4 CTAs per bucket while two launches fit side by side (296 CTAs are resident
    // at two per SM), then 2, then 1; more for large adapters, as far as those are resident together or their streams are long.
    // 1024-wide, rank 16, 8 rows, gate_up's expand with 4 / 8: 5.7 / 4.2 us; rank 32, 200 rows over 32 (bf16 intermediate, from a graph),
    // the eight launches of a layer with 1 / 2 / 4 / 8 everywhere 60 / 43 / 30 / 40, gate_up's expand by itself 21 / 12.9 / 8.8 / 7.2.
    const double resident = 2.0 * 148, half = 0.38 * resident, clusters = in_use + (b.T - 1) / kBgmvTok;
    C = in_use * 2 <= half ? 4 : (in_use <= half ? 2 : 1);
    while (C < 4 && (kb / C > 512 || (kb / C > 256 && in_use * C * 2 <= resident))) C *= 2;
    if (C == 4 && ((kb / 4 > 128 && clusters * 8 <= resident) || (kb / 4 >= 256 && in_use * 8 <= resident))) C = 8;
    return C;
  }
  // The least of a sum in KB of lora_B that a CTA could take meanwhile: what it takes of lora_B (rows of 16 ranks count as 32;
  // kinds 1 and 2, which multiply two halves of the intermediate and read y, 1.6 times), of lora_A and of x; the CTAs of the
  // launch that share an SM, and those that wait for a place (the GEMM's CTAs hold theirs longer); the exchange. The factors are
  // a fit, made for the least loss against the best size of each point, over 6688 measured points: adds (4512) of 1 to 4000 rows
  // over 6 to 900 adapters, even and skewed, graph and eager index arrays, widths 1024 to 4096, ranks 16 to 128, down of 4 to 7
  // and 14 K parts, and projections beside their GEMM (2176) of 1 to 128 rows. Mean loss 1.0 % (adds) and 1.3 %, of which 0.4 and
  // 0.6 is popularity, which the host does not see: the same rows over the same buckets, 2048-wide, rank 64, 48 over 100, take
  // 55.6 us a layer with clusters of four and 60.2 with the sizes taken (eight, o four) if even, 49.1 and 35.9 if skewed. Sums of
  // shares unrounded by rank rows and K parts, with a line at 290 CTAs, lost 2.3 and 1.6 %. us a launch with clusters of 1 / 2 /
  // 4 / 8, the size taken in brackets:
  //   adds: 1024-wide, rank 16, 8 rows over 32 adapters, gate_up 16.2 / 9.0 / 5.4 / [3.8]; rank 32, 64 over 32, o 3.7 / 2.9 /
  //   [2.5] / 3.6, 128 over 128, gate_up 19.7 / [12.6] / 14.9 / 19.7 (of skewed popularity 20.3 / 11.0 / 9.5 / 15.5), 384 over
  //   128, o 5.1 / [5.0] / 8.1 / 16.8; 4 rows, down of 4 K parts 9.3 / 4.8 / [3.0] / 3.2, of 5 11.9 / 7.3 / 5.5 / [3.7], of 6
  //   14.9 / 7.7 / 5.5 / [4.1], of 7 16.7 / 9.6 / 5.4 / [4.4], of 6 and 16 rows a bucket 15.3 / 8.0 / [6.0] / 7.4; 2048-wide, 384
  //   over 32 of skewed popularity, gate_up 28.3 / 21.6 / [12.2] / 16.3; rank 64, 256 over 32, down 33.8 / 22.8 / 15.9 / [12.5],
  //   of skewed popularity 32.8 / 23.0 / 16.3 / [19.1], 64 over 64, gate_up 32 / 32 / 18.3 / [21.5]; 4096-wide, 4 over 8, gate_up 55 / 28 /
  //   15.2 / [7.6]. (The fit, the points, and here the down of 5 to 7 K parts and what lies beside a GEMM are of the kernel before
  //   output tiles were dealt over the warps; the others, measured since, moved by 0 to 8 %, none to another order but near ties.)
  //   beside a GEMM (with the launch of the consumer): 1024-wide, rank 32, 64 rows over 64 adapters, qkv 11.4 / [11.4] / 15.9 /
  //   26, o 6.7 / [6.1] / 9.9 / 17.6, gate_up 22 / [15.0] / 17.9 / 24, down 13.4 / [9.5] / 13.9 / 25; 24 over 128, gate_up 18.7 /
  //   11.7 / [10.6] / 13.9; 8 over 32, qkv 8.8 / 8.6 / 7.9 / [7.1], gate_up 17.6 / 10.2 / [7.6] / 7.2; 128 over 128, o [8.2] /
  //   11.4 / 17.9 / 36; 2048-wide, 64 over 128, gate_up 35 / 27.4 / [27.2] / 35.
  double least = 0.0;
  const double windows = in_use + 0.9 * std::max(0.0, rows - 1.0 - 2.0 * in_use) / kBgmvTok, rows_each = std::min((double)kBgmvTok, rows / in_use);
  const int kparts = ceil_div_i(b.in_dim, kBgmvKP);
  for (int c = 1, any = 0; c <= 8; c *= 2) {
    const BgmvSplit split = bgmv_split(b, Q, c);
    if (split.rc == 0) continue;
    const double columns = split.by_k ? std::min(ceil_div_i(kparts, c) * kBgmvKP, b.in_dim) : b.in_dim;
    double b_rows = 0.0;
    for (int s = 0; s < st.n; ++s) b_rows += round_up_i(ceil_div_i(st.out[s], c), 32);
    const double share_b = b_rows * 2.0 * std::max(b.r_max, 32) / 1024.0 * (b.kind != 0 ? 1.6 : 1.0);
    const double share = share_b + (1.9 * split.rc + 0.8 * rows_each) * columns * 2.0 / 1024.0;
    const double ctas = 2.8 * b.beside + c * windows;
    const double cost = share + 0.75 * std::max(0.0, ctas - 148.0) + 2.25 * std::max(0.0, ctas - 296.0) + 3.8 * c;
    if (!any || cost < least) { least = cost; C = c; any = 1; }
  }
  return C;
}

// Tiling of a problem with the active slices `st` for clusters of C CTAs (more where the rank rows need them); false (and a
// reason) when it does not fit a CTA.
inline bool bgmv_plan_cluster(const BgmvProblem& b, const SliceTable& st, int C, BgmvParams* pp, const char** why) {
  const int Q = st.n * b.r_max;
  BgmvSplit split = bgmv_split(b, Q, C);
  while (split.rc == 0 && C < 8) split = bgmv_split(b, Q, C *= 2);
  if (split.rc == 0) { *why = "n_slices * r_max too large for one cluster"; return false; }
  const bool ksplit = split.by_k;
  const int Rc = split.rc;

  BgmvParams p;
  // (a bucket of n rows has 1 + (n - 1) / 16 windows, the most with as many buckets in use as there are rows)
  const int in_use_max = std::min(b.n_buckets, std::max(b.T, 1));
  p.clusters = b.n_buckets + (b.T - 1) / kBgmvTok;
  p.by_window = in_use_max + (b.T - in_use_max) / kBgmvTok < p.clusters && in_use_max < b.n_buckets ? 1 : 0;
  if (p.by_window) p.clusters = in_use_max + (b.T - in_use_max) / kBgmvTok;
  p.y = static_cast<__nv_bfloat16*>(b.y); p.y_ld = b.y_ld;
  p.x = static_cast<const __nv_bfloat16*>(b.x); p.x_ld = b.x_ld;
  p.T = b.T; p.in_dim = b.in_dim; p.S = b.S; p.r_max = b.r_max; p.st = st;
  p.rank_per_slot = b.rank_per_slot; p.scale_per_slot = b.scale_per_slot;
  p.sorted_idx = b.sorted_idx; p.slot_ids = b.slot_ids; p.counts = b.counts; p.offsets = b.offsets;
  p.n_buckets = b.n_buckets; p.scaling = b.scaling;
  p.c_shift = log2_exact(C);
  p.KP = std::min(b.in_dim, kBgmvKP);
  p.nkp = ceil_div_i(b.in_dim, p.KP);
  p.pitchA = p.KP * 2 + (p.nkp > 1 ? 64 : 0);  // dense when a tile is one contiguous copy
  const int stageA = 8 * p.pitchA;
  p.ER = std::max(32, std::min(256, floor_pow2(16384 / (b.r_max * 2))));
  p.er_shift = log2_exact(p.ER);
  int tiles = (Rc / 8) * (ksplit ? ceil_div_i(p.nkp, C) : p.nkp);
  for (int s = 0; s < B200_LORA_MAX_SLICES; ++s) p.oc[s] = 0;
  for (int s = 0; s < st.n; ++s) {
    p.oc[s] = round_up_i(ceil_div_i(st.out[s], C), 32);
    tiles += ceil_div_i(p.oc[s], p.ER);
  }
  const int stageB = p.ER * b.r_max * 2;
  p.stage_bytes = round_up_i(std::max(stageA, stageB), 128);
  // floats per token row: a multiple of 4 (16-byte reads) that is 8 modulo 16, so that the eight token
  // rows of a half warp start in different banks
  p.red_pitch = (Rc % 16 == 8) ? Rc : Rc + 8;
  const int red_bytes = round_up_i(kBgmvWarps * kBgmvTok * p.red_pitch * 4, 128);
  p.kind = b.kind;
  p.pitchT = round_up_i(Q * (b.kind != 0 ? 4 : 2), 128) + 64;
  const int tmp_bytes = round_up_i(kBgmvTok * p.pitchT, 128);
  const int bar_bytes = 256;
  int exp_tiles = 0, exp_blocks = 0;
  for (int s = 0; s < st.n; ++s) {
    exp_tiles += ceil_div_i(p.oc[s], p.ER);
    exp_blocks += p.oc[s] / 32;
  }
  if (exp_tiles > kBgmvMaxExpandTiles) { *why = "too many expand tiles per CTA"; return false; }
  const int tab_bytes = round_up_i((b.kind != 0 && b.mode != 4 ? exp_blocks + kBgmvWarps : exp_tiles) * 8, 128);
  p.ksplit = ksplit ? 1 : 0;
  p.pitchR = Q + 4;
  const int recv_bytes = ksplit ? round_up_i(C * kBgmvTok * p.pitchR * 4, 128) : 0;
  const int fixed = red_bytes + tmp_bytes + recv_bytes + tab_bytes + bar_bytes;
  // ring: what fits beside a second CTA on the SM, unless the caller set a size (up to the whole SM), and as many stages as hold 256
  // rows of lora_B (two of 128 up to eight of 32; fewer in flight not measured)
  const int ring_bytes = bgmv_options().ring_kb > 0 ? bgmv_options().ring_kb * 1024
                                                    : std::max(kBgmvSmemCoResident - fixed - 256, std::max(2, 256 / p.ER) * p.stage_bytes);
  int NS = std::min(std::max(tiles, std::max(2, 256 / p.ER)), (kBgmvSmemMax - fixed - 256) / p.stage_bytes);
  NS = std::min(NS, kBgmvMaxStages);
  NS = std::min(NS, std::max(std::max(2, 256 / p.ER), ring_bytes / p.stage_bytes));
  if (NS < std::max(2, 256 / p.ER)) { *why = "shared memory too small for the stages of 256 rows"; return false; }
  p.NS = NS;
  p.off_red = NS * p.stage_bytes;
  p.off_tmp = p.off_red + red_bytes;
  p.off_recv = p.off_tmp + tmp_bytes;
  p.off_tab = p.off_recv + recv_bytes;
  p.off_bar = p.off_tab + tab_bytes;
  p.full_k = (p.KP == kBgmvKP && b.in_dim % kBgmvKP == 0) ? 1 : 0;
  p.y_cols = 0;
  for (int s = 0; s < st.n; ++s) p.y_cols = std::max(p.y_cols, st.col[s] + st.out[s]);
  p.use_pdl = bgmv_options().pdl ? 1 : 0;
  p.mode = b.mode;
  p.tmp_io = b.tmp_io; p.io16 = b.io16; p.zero_rows = b.zero_rows; p.no_add = b.no_add; p.gate = b.gate;
  p.token_to_slot = b.token_to_slot;
  if ((b.mode == 1 || b.mode == 2) && b.tmp_io == nullptr) { *why = "shrink-only / expand-only need the tmp array"; return false; }
  if (b.mode == 3 && b.token_to_slot == nullptr) { *why = "overwrite mode needs token_to_slot"; return false; }
  *pp = p;
  return true;
}

// Fills `pp` with the tiling for this problem; returns false (and a reason) when
// the fused kernel cannot run it.
inline bool bgmv_plan(const BgmvProblem& b, BgmvParams* pp, const char** why) {
  const char* dummy;
  if (why == nullptr) why = &dummy;
  SliceTable st;
  st.n = 0;
  for (int s = 0; s < B200_LORA_MAX_SLICES; ++s) { st.a[s] = st.b[s] = nullptr; st.out[s] = st.col[s] = 0; }
  for (int s = 0; s < b.st.n; ++s) {
    if (b.st.out[s] == 0) continue;
    st.a[st.n] = b.st.a[s]; st.b[st.n] = b.st.b[s]; st.out[st.n] = b.st.out[s]; st.col[st.n] = b.st.col[s];
    ++st.n;
  }
  if (st.n == 0) { *why = "no active slice"; return false; }
  if (b.r_max % (b.kind != 0 ? 16 : 32) != 0 || b.r_max > 256) {
    *why = b.kind != 0 ? "r_max must be a multiple of 16, <= 256" : "r_max must be a multiple of 32, <= 256";
    return false;
  }
  if (b.kind != 0 && b.mode == 3) { *why = "overwrite mode is for bf16 with r_max a multiple of 32"; return false; }
  if (b.kind == 2 && b.mode == 4) { *why = "the fp32 form is for bf16"; return false; }
  if (b.in_dim % 32 != 0) { *why = "in_dim must be a multiple of 32"; return false; }
  if (b.x_ld % 8 != 0 || b.y_ld % 8 != 0) { *why = "row strides must be multiples of 8 elements"; return false; }
  if (!aligned16(b.x) || !aligned16(b.y)) { *why = "x / y must be 16-byte aligned"; return false; }
  for (int s = 0; s < st.n; ++s) {
    if (st.out[s] % 8 != 0 || st.col[s] % 8 != 0) { *why = "slice widths / offsets must be multiples of 8"; return false; }
    if (!aligned16(st.a[s]) || !aligned16(st.b[s])) { *why = "slabs must be 16-byte aligned"; return false; }
  }
  if (b.n_buckets < 1 || b.n_buckets + b.T / kBgmvTok > 65535) { *why = "n_buckets outside [1, 65535]"; return false; }

  const int asked = bgmv_options().cluster;
  if (asked == 1 || asked == 2 || asked == 4 || asked == 8) return bgmv_plan_cluster(b, st, asked, pp, why);
  // the cheapest cluster whose CTAs can hold their share; a larger one where that one cannot (outputs of more than 256 tiles a CTA:
  // 65536 columns at rank 96 in clusters of two)
  for (int C = bgmv_cluster(b, st);; C *= 2) {
    if (bgmv_plan_cluster(b, st, C, pp, why)) return true;
    if (C >= 8) return false;
  }
}

// (the caller has planned it)
inline int bgmv_launch(const BgmvParams& p, cudaStream_t stream) {
  const size_t smem = (size_t)p.off_bar + 256;
  static thread_local int configured_device = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured_device != dev) {
#define B200_BGMV_ALL(M, K)                                                                                                  \
  (const void*)bgmv_fused_kernel<M, false, K, false>, (const void*)bgmv_fused_kernel<M, true, K, false>,                     \
      (const void*)bgmv_fused_kernel<M, false, K, true>, (const void*)bgmv_fused_kernel<M, true, K, true>
    const void* kernels[] = {B200_BGMV_ALL(0, 0), B200_BGMV_ALL(1, 0), B200_BGMV_ALL(2, 0), B200_BGMV_ALL(3, 0), B200_BGMV_ALL(0, 1), B200_BGMV_ALL(0, 2), B200_BGMV_ALL(1, 1),
                             B200_BGMV_ALL(1, 2), B200_BGMV_ALL(2, 1), B200_BGMV_ALL(2, 2)};
#undef B200_BGMV_ALL
    for (const void* k : kernels) {
      cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kBgmvSmemMax);
      if (e != cudaSuccess) return fail(B200_LORA_ECUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    }
    configured_device = dev;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1u << p.c_shift, (unsigned)p.clusters, 1);
  cfg.blockDim = dim3(kBgmvThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  int na = 0;
  attrs[na].id = cudaLaunchAttributeClusterDimension;
  attrs[na].val.clusterDim.x = 1u << p.c_shift;
  attrs[na].val.clusterDim.y = 1;
  attrs[na].val.clusterDim.z = 1;
  ++na;
  if (p.use_pdl) {
    attrs[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = (unsigned)na;
  cudaError_t e;
#define B200_BGMV_LAUNCH(M, K)                                                               \
  (p.ER == 256 ? (p.full_k ? cudaLaunchKernelEx(&cfg, bgmv_fused_kernel<M, true, K, false>, p)   \
                           : cudaLaunchKernelEx(&cfg, bgmv_fused_kernel<M, false, K, false>, p)) \
               : (p.full_k ? cudaLaunchKernelEx(&cfg, bgmv_fused_kernel<M, true, K, true>, p)    \
                           : cudaLaunchKernelEx(&cfg, bgmv_fused_kernel<M, false, K, true>, p)))
  switch (8 * p.kind + p.mode) {  // (mode 4: decode_step.cuh)
    case 1: e = B200_BGMV_LAUNCH(1, 0); break;
    case 2: e = B200_BGMV_LAUNCH(2, 0); break;
    case 3: e = B200_BGMV_LAUNCH(3, 0); break;
    case 8: e = B200_BGMV_LAUNCH(0, 1); break;
    case 9: e = B200_BGMV_LAUNCH(1, 1); break;
    case 10: e = B200_BGMV_LAUNCH(2, 1); break;
    case 16: e = B200_BGMV_LAUNCH(0, 2); break;
    case 17: e = B200_BGMV_LAUNCH(1, 2); break;
    case 18: e = B200_BGMV_LAUNCH(2, 2); break;
    default: e = B200_BGMV_LAUNCH(0, 0); break;
  }
#undef B200_BGMV_LAUNCH
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(B200_LORA_ECUDA, "bgmv_fused_kernel launch: %s", cudaGetErrorString(e));
  }
  return B200_LORA_OK;
}

// A kernel that waits for the launch ahead itself (griddepcontrol.wait in every CTA): it may become resident while that one runs.
template <typename... Params, typename... Args>
inline int launch_dependent(void (*kernel)(Params...), const char* name, dim3 grid, int threads, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = bgmv_options().pdl ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(B200_LORA_ECUDA, "%s launch: %s", name, cudaGetErrorString(e));
  }
  return B200_LORA_OK;
}

}  // namespace b200lora
