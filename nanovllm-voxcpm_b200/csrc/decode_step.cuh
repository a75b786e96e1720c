// Kernels of a decode step's layer chain for small batches (up to 128 rows): base GEMM, attention and the glue between them,
// built so that the chain is short.
//
// A decode step of a small model is a chain of dependent launches, each bound by latency: with library GEMMs, the LoRA add
// behind each of them, split-KV attention and separate glue kernels a layer of a 1024-wide decoder took 94 us (64 rows),
// against 12 us of HBM time for its weights. Here
//   * the base product and the LoRA delta of a projection are one launch: clusters of the fused decode kernel write their delta
//     (fp32) into one plane of a buffer [planes, T, out], GEMM CTAs beside them the K parts into the others;
//   * the consumer of a projection (add + norm, RoPE + attention, SiLU * up) adds the planes in fp32: no rounding of the base
//     output, no pass of its own;
//   * RoPE, the cache store and attention are one kernel per (request, kv head).
// All are launched as programmatic dependents; weights are requested before the wait.
#pragma once

#include "bgmv_fused.cuh"
#include "glue.cuh"
#include "tc_common.cuh"

namespace b200lora {

constexpr int kDecMaxRows = 128;
constexpr int kDecMaxPlanes = 9;      // 8 K parts + the LoRA delta

// ============================================================================ projection
// part[p][t][o] = sum over K part p of x[t][k] W[o][k], as D^T = W . x^T on tcgen05: 128 weight rows are the M operand, the
// tokens the N operand. CTA = (weight row tile, K part).
constexpr int kDecGemmMaxStages = 4;
constexpr int kDecBK = 64;
constexpr int kDecGemmBars = 128;  // bytes of the barriers and flags in front of the ring

struct DecGemmArgs {
  float* part;
  int T, in_dim, out, n_pad;  // n_pad: T rounded up to 16
  int tiles, parts, k_part;   // weight row tiles, K parts and their columns (multiple of 64)
  int stages;
  // the plane of the delta: rows without one are zeroed here (a cluster of the delta kernel that has no rows exits at once)
  float* delta;
  const int32_t *token_to_slot, *rank_per_slot;
  int S;
};
struct DecGemmMaps {
  CUtensorMap w;  // [out, in], box 128 x 64
  CUtensorMap x;  // [T, in], box n_pad x 64
};

// One GEMM CTA of kBgmvThreads threads: warp 8 TMA, warp 0 MMA, warps 4-7 epilogue.
__device__ __forceinline__ void decode_gemm_body(const DecGemmMaps& maps, const DecGemmArgs& a, uint8_t* smem, int unit) {
  // barriers, TMEM base and abort flag in the first bytes, the ring behind them (no static shared memory: with it two CTAs of
  // the delta kernel would no longer fit on an SM)
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
  volatile uint32_t& tmem_base_s = *reinterpret_cast<volatile uint32_t*>(smem + 8 * (2 * kDecGemmMaxStages + 1));
  volatile int& abort_flag = *reinterpret_cast<volatile int*>(smem + 8 * (2 * kDecGemmMaxStages + 1) + 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (unit >= a.tiles * a.parts) {
    griddep_launch_dependents();
    griddep_wait();
    return;
  }
  const uint32_t smem_base = (smem_u32(smem) + kDecGemmBars + 1023u) & ~1023u;
  constexpr uint32_t kW = 128 * kDecBK * 2;
  const uint32_t x_bytes = (uint32_t)a.n_pad * kDecBK * 2, stage = kW + ((x_bytes + 1023u) & ~1023u);
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * (uint32_t)s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (uint32_t)(kDecGemmMaxStages + s); };
  const uint32_t acc_full = bar0 + 8u * (2 * kDecGemmMaxStages);
  const int NS = a.stages;
  int tmem_cols = 32;
  while (tmem_cols < a.n_pad) tmem_cols *= 2;
  if (tid == 0) {
    for (int s = 0; s < NS; ++s) { mbar_init(full_bar(s), 2); mbar_init(empty_bar(s), 1); }  // full: W and x
    mbar_init(acc_full, 1);
    abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(&tmem_base_s)), (uint32_t)tmem_cols);
    tc_fence_before_sync();
  }
  __syncthreads();
  griddep_launch_dependents();  // (after this CTA holds its tensor memory)
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  const int tile = unit / a.parts, part = unit - tile * a.parts;
  const int row0 = tile * 128, k0 = part * a.k_part;
  const int nk = (min(a.k_part, a.in_dim - k0) + kDecBK - 1) / kDecBK;
  if (warp == kBgmvWarps) {
    const uint32_t leader = elect_one();
    if (leader) { tma_prefetch_desc(&maps.w); tma_prefetch_desc(&maps.x); }
    auto load_w = [&](int kc, int st) {
      if (leader) {
        mbar_arrive_expect_tx(full_bar(st), kW);
        tma_load_2d(smem_base + (uint32_t)st * stage, &maps.w, k0 + kc * kDecBK, row0, full_bar(st));
      }
      __syncwarp();
    };
    for (int kc = 0; kc < min(nk, NS); ++kc) load_w(kc, kc);  // weights depend on nothing
    griddep_wait();
    int st = 0, round = 0;
    for (int kc = 0; kc < nk; ++kc) {
      if (round > 0) {
        mbar_wait_bounded(empty_bar(st), (uint32_t)((round & 1) ^ 1), &abort_flag);
        load_w(kc, st);
      }
      if (leader) {
        mbar_arrive_expect_tx(full_bar(st), x_bytes);
        tma_load_2d(smem_base + (uint32_t)st * stage + kW, &maps.x, k0 + kc * kDecBK, 0, full_bar(st));
      }
      __syncwarp();
      if (++st == NS) { st = 0; ++round; }
    }
  } else if (warp == 0) {
    const uint32_t leader = elect_one();
    const uint64_t desc0 = umma_smem_desc(smem_base, 128);
    const uint32_t hi = (uint32_t)(desc0 >> 32), lo0 = (uint32_t)desc0, idesc = umma_idesc_bf16(128, a.n_pad);
    int st = 0, round = 0;
    for (int kc = 0; kc < nk; ++kc) {
      mbar_wait_bounded(full_bar(st), (uint32_t)(round & 1), &abort_flag);
      tc_fence_after_sync();
      const uint32_t w = lo0 + ((uint32_t)st * stage >> 4), xr = w + (kW >> 4);
#pragma unroll
      for (int k4 = 0; k4 < kDecBK / 16; ++k4) umma_elected(tmem_base, w + 2u * k4, xr + 2u * k4, hi, idesc, (kc > 0 || k4 > 0) ? 1u : 0u, leader);
      umma_commit_elected(empty_bar(st), leader);
      if (++st == NS) { st = 0; ++round; }
    }
    umma_commit_elected(acc_full, leader);
  } else if (warp >= 4 && warp < 8) {
    const int quarter = warp & 3, o = row0 + quarter * 32 + lane;
    griddep_wait();  // the previous launch may still read the planes
    if (a.delta != nullptr && part == 0) {  // (32 rows at a time: one by one the lookups took 12 us)
      for (int t0 = 0; t0 < a.T; t0 += 32) {
        bool dead = false;
        if (t0 + lane < a.T) {
          const int sl = a.token_to_slot[t0 + lane];
          dead = sl < 0 || sl >= a.S || (a.rank_per_slot != nullptr && a.rank_per_slot[sl] <= 0);
        }
        for (unsigned rows = __ballot_sync(0xffffffffu, dead); rows != 0; rows &= rows - 1)
          if (o < a.out) a.delta[(int64_t)(t0 + __ffs((int)rows) - 1) * a.out + o] = 0.f;
      }
    }
    mbar_wait_bounded(acc_full, 0u, &abort_flag);
    tc_fence_after_sync();
    // Through shared memory (the ring is free: every MMA has read it), then one bulk copy per token: with a store per thread
    // and token the 64 tokens of a tile took 2.8 us.
    for (int c = 0; c < a.T; c += 16) {
      uint32_t v[16];
      tmem_ld_32x16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c, v);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 16; ++e)  // (the rows up to n_pad exist in the ring)
        sts32(smem_base + (uint32_t)((c + e) * 512 + (quarter * 32 + lane) * 4), v[e]);
    }
    fence_proxy_async_smem();
    named_bar_sync(2, 128);
    const int token = tid - 128;
    if (token < a.T) {
      bulk_s2g(a.part + ((int64_t)part * a.T + token) * a.out + row0, smem_base + (uint32_t)token * 512u, (uint32_t)min(128, a.out - row0) * 4u);
      bulk_commit_group();
      bulk_wait_all();
    }
    tc_fence_before_sync();
  }
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, (uint32_t)tmem_cols);
  if (tid == 0 && abort_flag != 0) atomicOr(&g_b200_status, kStatusWaitGaveUp);
}

// GEMM CTAs first (they are all in use), then the buckets of the delta kernel, in clusters of one size.
template <bool kFullK, int kKind, bool kWide>
__global__ void __launch_bounds__(kBgmvThreads, 2)
decode_linear_kernel(const __grid_constant__ DecGemmMaps maps, const DecGemmArgs g, const __grid_constant__ BgmvParams p, const int gemm_rows) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((int)blockIdx.y < gemm_rows) decode_gemm_body(maps, g, smem, (int)blockIdx.y * (int)gridDim.x + (int)blockIdx.x);
  else bgmv_body<4, kFullK, kKind, kWide>(p, smem, (int)blockIdx.y - gemm_rows, (int)gridDim.y - gemm_rows);
}
__global__ void __launch_bounds__(kBgmvThreads, 2)
decode_gemm_kernel(const __grid_constant__ DecGemmMaps maps, const DecGemmArgs g) {
  extern __shared__ __align__(1024) uint8_t smem[];
  decode_gemm_body(maps, g, smem, (int)blockIdx.x);
}

// K parts of a projection: about 128 CTAs, at most 8 parts of at least one 64-column step
inline int decode_gemm_parts(int in_dim, int out) {
  const int tiles = ceil_div_i(out, 128), steps = ceil_div_i(in_dim, kDecBK);
  int parts = 1;
  while (parts < 8 && tiles * parts * 2 <= 148 && ceil_div_i(steps, 2 * parts) * (2 * parts - 1) < steps) parts *= 2;
  return parts;
}
// ... and the CTAs that it counts beside the clusters of the delta (two to an SM)
inline int decode_gemm_ctas(int in_dim, int out) { return std::min(ceil_div_i(out, 128) * decode_gemm_parts(in_dim, out), 148); }

// planes of x . W^T, and (lora != nullptr) the delta in the plane behind them
inline int decode_linear_launch(float* planes, const void* x, int64_t x_ld, int T, int in_dim, const void* w, int64_t w_ld, int out,
                                const BgmvParams* lora, cudaStream_t stream) {
  DecGemmArgs a = {};
  DecGemmMaps maps;
  a.part = planes; a.T = T; a.in_dim = in_dim; a.out = out; a.n_pad = round_up_i(T, 16);
  a.parts = decode_gemm_parts(in_dim, out); a.tiles = ceil_div_i(out, 128);
  a.k_part = round_up_i(ceil_div_i(in_dim, a.parts), kDecBK);
  const int stage = 128 * kDecBK * 2 + round_up_i(a.n_pad * kDecBK * 2, 1024);
  a.stages = std::min(kDecGemmMaxStages, 98 * 1024 / stage);
  if (int rc = make_tmap_2d(&maps.w, w, (uint64_t)out, (uint64_t)in_dim, (uint64_t)w_ld, 128, kDecBK)) return rc;
  if (int rc = make_tmap_2d(&maps.x, x, (uint64_t)T, (uint64_t)in_dim, (uint64_t)x_ld, (uint32_t)a.n_pad, kDecBK)) return rc;
  size_t smem = (size_t)a.stages * stage + 1024 + kDecGemmBars;
  if (lora == nullptr) {
    const cudaError_t e = cudaFuncSetAttribute(decode_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return fail(B200_LORA_ECUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    return launch_dependent(decode_gemm_kernel, "decode_gemm_kernel", dim3((unsigned)(a.tiles * a.parts)), kBgmvThreads, smem, stream, maps, a);
  }
  a.delta = planes + (size_t)a.parts * T * out;
  const BgmvParams& p = *lora;
  a.token_to_slot = p.token_to_slot; a.rank_per_slot = p.rank_per_slot; a.S = p.S;
  smem = std::max(smem, (size_t)p.off_bar + 256);
  const int C = 1 << p.c_shift, gemm_rows = ceil_div_i(a.tiles * a.parts, C);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)C, (unsigned)(gemm_rows + p.clusters), 1);
  cfg.blockDim = dim3(kBgmvThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = (unsigned)C;
  attrs[0].val.clusterDim.y = attrs[0].val.clusterDim.z = 1;
  attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = p.use_pdl ? 2 : 1;
  cudaError_t e = cudaSuccess;
#define B200_DEC_LINEAR(F, K, W)                                                                                              \
  {                                                                                                                           \
    e = cudaFuncSetAttribute(decode_linear_kernel<F, K, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBgmvSmemMax); \
    if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, decode_linear_kernel<F, K, W>, maps, a, p, gemm_rows);                 \
  }
  const int which = (p.full_k ? 4 : 0) + (p.kind ? 2 : 0) + (p.ER == 256 ? 0 : 1);
  switch (which) {
    case 0: B200_DEC_LINEAR(false, 0, false) break;
    case 1: B200_DEC_LINEAR(false, 0, true) break;
    case 2: B200_DEC_LINEAR(false, 1, false) break;
    case 3: B200_DEC_LINEAR(false, 1, true) break;
    case 4: B200_DEC_LINEAR(true, 0, false) break;
    case 5: B200_DEC_LINEAR(true, 0, true) break;
    case 6: B200_DEC_LINEAR(true, 1, false) break;
    default: B200_DEC_LINEAR(true, 1, true) break;
  }
#undef B200_DEC_LINEAR
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(B200_LORA_ECUDA, "decode_linear_kernel launch: %s", cudaGetErrorString(e));
  }
  return B200_LORA_OK;
}

// ============================================================================ glue over planes
// Four consecutive columns of a row of a projection's result, N of them: the planes [planes, T, ld] added in fp32. All loads
// of a thread are issued before the first sum waits, hence the unrolled forms (up to kP planes; the last plane is read again
// in place of the missing ones and left out of the sum).
template <int N, int kP>
__device__ __forceinline__ void planes_load4_upto(const float* part, int planes, int64_t plane, const int64_t (&at)[N], float (&v)[N][4]) {
  float4 got[kP][N];
#pragma unroll
  for (int p = 0; p < kP; ++p)
#pragma unroll
    for (int n = 0; n < N; ++n) got[p][n] = __ldcg(reinterpret_cast<const float4*>(part + min(p, planes - 1) * plane + at[n]));
#pragma unroll
  for (int n = 0; n < N; ++n) {
    v[n][0] = v[n][1] = v[n][2] = v[n][3] = 0.f;
#pragma unroll
    for (int p = 0; p < kP; ++p) {
      const bool live = p < planes;
      v[n][0] += live ? got[p][n].x : 0.f; v[n][1] += live ? got[p][n].y : 0.f;
      v[n][2] += live ? got[p][n].z : 0.f; v[n][3] += live ? got[p][n].w : 0.f;
    }
  }
}
template <int N>
__device__ __forceinline__ void planes_load4(const float* part, int planes, int64_t plane, const int64_t (&at)[N], float (&v)[N][4]) {
  if (planes <= 2) planes_load4_upto<N, 2>(part, planes, plane, at, v);
  else if (planes == 3) planes_load4_upto<N, 3>(part, planes, plane, at, v);
  else if (planes <= 5) planes_load4_upto<N, 5>(part, planes, plane, at, v);
  else planes_load4_upto<N, kDecMaxPlanes>(part, planes, plane, at, v);
}
__device__ __forceinline__ uint2 pack4(const float (&v)[4]) { return make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3])); }
__device__ __forceinline__ void unpack4(uint2 r, float (&v)[4]) {
  const float2 a = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&r.x)), b = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&r.y));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

// hidden_out = residual + sum of planes (bf16); normed = rms_norm(hidden_out) * weight. One CTA per row, four columns per
// thread: a row's loads are all in flight at once.
__global__ void __launch_bounds__(1024) decode_add_rmsnorm_kernel(__nv_bfloat16* __restrict__ normed, __nv_bfloat16* hidden_out,
                                                                  const float* part, int planes, const __nv_bfloat16* residual,
                                                                  const __nv_bfloat16* __restrict__ weight, int T, int H, float eps) {
  __shared__ float sums[32];
  griddep_launch_dependents();
  const int row = blockIdx.x, col = threadIdx.x * 4, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float w[4], res[4], v[1][4], ss = 0.f;
  const bool live = col < H;
  if (live) unpack4(*reinterpret_cast<const uint2*>(weight + col), w);
  griddep_wait();
  if (live) {
    const int64_t at[1] = {(int64_t)row * H + col};
    const uint2 old = *reinterpret_cast<const uint2*>(residual + at[0]);
    planes_load4<1>(part, planes, (int64_t)T * H, at, v);
    unpack4(old, res);
#pragma unroll
    for (int e = 0; e < 4; ++e) v[0][e] += res[e];
    const uint2 sum = pack4(v[0]);
    *reinterpret_cast<uint2*>(hidden_out + at[0]) = sum;
    unpack4(sum, v[0]);  // the norm sees the rounded sum
#pragma unroll
    for (int e = 0; e < 4; ++e) ss += v[0][e] * v[0][e];
  }
  ss = warp_sum(ss);
  if (lane == 0) sums[warp] = ss;
  __syncthreads();
  ss = warp_sum(lane < (int)(blockDim.x >> 5) ? sums[lane] : 0.f);
  if (!live) return;
  const float rstd = rsqrtf(ss / (float)H + eps);
#pragma unroll
  for (int e = 0; e < 4; ++e) v[0][e] *= rstd * w[e];
  *reinterpret_cast<uint2*>(normed + (int64_t)row * H + col) = pack4(v[0]);
}

// out = silu(gate) * up of the summed planes [planes, T, 2 I]
__global__ void __launch_bounds__(256) decode_silu_mul_kernel(__nv_bfloat16* __restrict__ out, const float* part, int planes, int T, int I) {
  griddep_launch_dependents();
  griddep_wait();
  const int nvec = I >> 2, total = T * nvec;
  for (int i = blockIdx.x * 256 + threadIdx.x; i < total; i += gridDim.x * 256) {
    const int row = i / nvec, col = (i - row * nvec) * 4;
    float v[2][4], o[4];
    const int64_t gate = (int64_t)row * 2 * I + col, at[2] = {gate, gate + I};
    planes_load4<2>(part, planes, (int64_t)T * 2 * I, at, v);
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = v[0][e] / (1.f + expf(-v[0][e])) * v[1][e];
    *reinterpret_cast<uint2*>(out + (int64_t)row * I + col) = pack4(o);
  }
}

// ============================================================================ attention
// One CTA per (kv head, request): sums the planes of the request's q heads of that kv head, k and v, rotates q and k, stores k
// and v to the paged cache and attends over the cached tokens (mma.sync m16n8k16 with the up to 16 q heads as rows, online
// softmax per warp, merged at the end). Every warp has blocks of 16 tokens of its own and stages of its own for their K and V
// rows: the first ones are requested (cp.async) before the wait, the next one as soon as a stage is free, and no warp waits for
// another before the merge. us a launch in a chain of its own, chunks of 368 tokens shared by the CTA / this, 64 requests around 200,
// 352 and 640 tokens: 2 kv heads of 64, 4.6 / 4.8, 6.7 / 6.5 and 11.7 / 10.1; of 128, 7.3 / 7.6, 10.7 / 9.9 and 17.6 / 14.4; one
// request around 200 3.3 / 3.6: short contexts lose 3 to 7 % to what long ones gain. Beyond 368 tokens a block's probabilities are
// rounded to bf16 against the running maximum of its own warp, not of the CTA's chunk: the same widths, other last bits.
struct DecAttnArgs {
  const float* part; int planes, ld;       // [planes, T, (Hq + 2 Hk) D]
  int T, Hq, Hk;
  const int64_t* positions;
  const void* cos; const void* sin;        // [max_pos, D / 2] or [max_pos, D]
  int table_dim, table_dtype, max_pos;
  __nv_bfloat16 *k_cache, *v_cache;        // [blocks, block_size, Hk, D]
  const int32_t* block_tables; int max_blocks, block_size;
  const int32_t* context_lens;             // tokens to attend to, the new one included
  const int64_t* slot_mapping;             // where the new token's k and v go (< 0: nowhere)
  __nv_bfloat16* out;                      // [T, Hq D]
  float scale;
};

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

constexpr int kDecAttnWarps = 8;
// A warp's items are the K and V rows of its blocks together (heads of 64), or K and V in turn (128: one and a half blocks are all
// that fits, two CTAs per SM); slots of an item
template <int D>
__host__ __device__ constexpr int dec_attn_slots() { return 3; }
template <int D>
__host__ __device__ constexpr int dec_attn_smem() {
  const int kv = kDecAttnWarps * dec_attn_slots<D>() * (D == 64 ? 2 : 1) * 16 * (D * 2 + 16), merge = kDecAttnWarps * 16 * (D + 2) * 4;
  return (kv > merge ? kv : merge) + 16 * (D * 2 + 16);
}
template <int N>
__device__ __forceinline__ void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int D>
__global__ void __launch_bounds__(kDecAttnWarps * 32) decode_attention_kernel(const DecAttnArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  constexpr int kPitch = D * 2 + 16, kHalf = D / 2, kWarps = kDecAttnWarps, kThreads = kWarps * 32, kSlots = dec_attn_slots<D>();
  constexpr bool kTurn = D == 128;  // K and V in turn
  constexpr int kRows = 16 * kPitch, kItem = (kTurn ? 1 : 2) * kRows;  // bytes of the K or V rows of a block, of an item
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int kvh = blockIdx.x, req = blockIdx.y, group = a.Hq / a.Hk;
  griddep_launch_dependents();
  const uint32_t q_u32 = smem_u32(smem), kv_u32 = q_u32 + kRows + (uint32_t)(warp * kSlots * kItem);  // this warp's slots
  // (the cache rows of earlier steps were written before this chain of dependent launches began: see the header)
  const int ctx = a.context_lens[req];
  const int32_t* table = a.block_tables + (int64_t)req * a.max_blocks;
  const int n_old = max(ctx - 1, 0);  // tokens whose k and v are in the cache already
  const int n_blocks = (ctx + 15) >> 4;

  // A warp's blocks are warp, warp + 8, ... First element of the cache rows of its block j (lane l: row l % 16):
  auto rows_of = [&](int j) {
    const int tok = 16 * (warp + j * kWarps) + (lane & 15);
    if (16 * (warp + j * kWarps) >= n_old || tok >= n_old) return (int64_t)0;
    const int blk = table[tok / a.block_size];
    return (blk * (int64_t)a.block_size + tok % a.block_size) * ((int64_t)a.Hk * D) + (int64_t)kvh * D;
  };
  // K (which 0), V (1) or both (2) of block j into a slot: cached rows; that of the new token is written below, rows behind the
  // context are zero (their probabilities are zero, their values must be finite). A group is committed for missing blocks too.
  auto load_item = [&](int j, int which, uint32_t slot, int64_t at) {
    const int b = warp + j * kWarps;
    if (b < n_blocks) {
      constexpr int kPieces = D / 8;  // 16-byte pieces of a row
      const int p = lane % kPieces;
#pragma unroll
      for (int q = 0; q < kPieces / 2; ++q) {
        const int r = lane / kPieces + q * (32 / kPieces);
        const int64_t row = __shfl_sync(0xffffffffu, at, r) + p * 8;
        if (16 * b + r == n_old && ctx > 0) continue;
        const bool live = 16 * b + r < n_old;
        const uint32_t dst = slot + (uint32_t)(r * kPitch + p * 16);
        if (which != 1) cp_async_16(dst, a.k_cache + (live ? row : 0), live ? 16u : 0u);
        if (which != 0) cp_async_16(dst + (which == 2 ? (uint32_t)kRows : 0u), a.v_cache + (live ? row : 0), live ? 16u : 0u);
      }
    }
    cp_async_commit();
  };
  int64_t at = 0;  // (in turn) of the block whose K was asked for last
#pragma unroll
  for (int i = 0; i < kSlots; ++i) {
    if (!kTurn || (i & 1) == 0) at = rows_of(kTurn ? i >> 1 : i);
    load_item(kTurn ? i >> 1 : i, kTurn ? i & 1 : 2, kv_u32 + (uint32_t)(i * kItem), at);
  }

  // ---- q, k, v of the new token: a thread takes four pairs (j, j + D / 2) of a head
  int64_t pos = a.positions[req];
  pos = pos < 0 ? 0 : (pos >= a.max_pos ? a.max_pos - 1 : pos);
  const int64_t slot = a.slot_mapping[req];
  const int64_t plane = (int64_t)a.T * a.ld, row_at = (int64_t)req * a.ld;
  const int hi_off = a.table_dim == D ? kHalf : 0;
  __shared__ __align__(16) __nv_bfloat16 kv_new[2][D];
  bool waited = false;
  for (int i = tid; i < (group + 2) * (kHalf / 4) || !waited; i += kThreads) {
    const int head = i / (kHalf / 4), j = (i - head * (kHalf / 4)) * 4;  // heads 0 .. group - 1: q; group: k; group + 1: v
    const bool item = head < group + 2, turned = head <= group;
    float c1[4], s1[4], c2[4], s2[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      c1[e] = c2[e] = 1.f;
      s1[e] = s2[e] = 0.f;
      if (turned) {
        const int64_t tb = pos * a.table_dim + j + e;
        c1[e] = table_at(a.cos, a.table_dtype, tb); s1[e] = table_at(a.sin, a.table_dtype, tb);
        c2[e] = table_at(a.cos, a.table_dtype, tb + hi_off); s2[e] = table_at(a.sin, a.table_dtype, tb + hi_off);
      }
    }
    if (!waited) griddep_wait();  // (tables, positions and the cache do not depend on the launches ahead)
    waited = true;
    if (!item) break;
    const int64_t col = head < group ? (int64_t)(kvh * group + head) * D : (int64_t)(a.Hq + (head - group) * a.Hk + kvh) * D;
    const int64_t at[2] = {row_at + col + j, row_at + col + kHalf + j};
    float x[2][4], lo[4], hi[4];
    planes_load4<2>(a.part, a.planes, plane, at, x);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      lo[e] = turned ? __fadd_rn(__fmul_rn(x[0][e], c1[e]), __fmul_rn(-x[1][e], s1[e])) : x[0][e];
      hi[e] = turned ? __fadd_rn(__fmul_rn(x[1][e], c2[e]), __fmul_rn(x[0][e], s2[e])) : x[1][e];
    }
    __nv_bfloat16* dst = head < group ? reinterpret_cast<__nv_bfloat16*>(smem + head * kPitch) : kv_new[head - group];
    *reinterpret_cast<uint2*>(dst + j) = pack4(lo);
    *reinterpret_cast<uint2*>(dst + kHalf + j) = pack4(hi);
  }
  for (int i = tid; i < (16 - group) * D; i += kThreads)  // unused rows of the q tile
    reinterpret_cast<__nv_bfloat16*>(smem + (group + i / D) * kPitch)[i % D] = __float2bfloat16_rn(0.f);
  __syncthreads();
  if (tid < 2 * (D / 8)) {
    const int which = tid / (D / 8), p = tid - which * (D / 8);
    const uint4 piece = *reinterpret_cast<const uint4*>(&kv_new[which][8 * p]);
    if (slot >= 0) *reinterpret_cast<uint4*>((which ? a.v_cache : a.k_cache) + slot * a.Hk * D + (int64_t)kvh * D + 8 * p) = piece;
  }

  uint32_t qf[D / 16][4];
  {
    const uint32_t addr = q_u32 + (uint32_t)((lane & 15) * kPitch + (lane >> 4) * 16);
#pragma unroll
    for (int k = 0; k < D / 16; ++k) ldsm_x4(addr + 32u * k, qf[k]);
  }
  float o[D / 8][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int d = 0; d < D / 8; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;
  const float sc = a.scale * 1.4426950408889634f;  // scores in units of log2(e)

  auto put_new = [&](int b, int which, uint32_t slot) {  // the new token's row
    if (n_old >> 4 == b && lane < D / 8)
      sts128(slot + (uint32_t)((n_old & 15) * kPitch + 16 * lane), *reinterpret_cast<const uint4*>(&kv_new[which][8 * lane]));
  };
  uint32_t here = kv_u32;  // the slot of the item at hand
  auto advance = [&]() {
    here += kItem;
    if (here == kv_u32 + kSlots * kItem) here = kv_u32;
  };
  for (int j = 0, b = warp; b < n_blocks; ++j, b += kWarps) {
    cp_async_wait_group<kSlots - 1>();
    const uint32_t k_st = here;
    if (kTurn) {
      put_new(b, 0, k_st);
    } else if (n_old >> 4 == b && lane < 2 * (D / 8)) {
      const int which = lane / (D / 8), p = lane - which * (D / 8);
      sts128(k_st + (uint32_t)(which * kRows + (n_old & 15) * kPitch + 16 * p), *reinterpret_cast<const uint4*>(&kv_new[which][8 * p]));
    }
    __syncwarp();
    {
      float s[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) s[h][0] = s[h][1] = s[h][2] = s[h][3] = 0.f;
      // matrices: tokens 0-7 / dims 0-7, tokens 0-7 / dims 8-15, tokens 8-15 / dims 0-7, tokens 8-15 / dims 8-15
      const uint32_t ka = k_st + (uint32_t)(((lane & 7) + ((lane >> 4) << 3)) * kPitch + ((lane >> 3) & 1) * 16);
#pragma unroll
      for (int k = 0; k < D / 16; ++k) {
        uint32_t kf[4];
        ldsm_x4(ka + 32u * k, kf);
        mma_bf16_16816(s[0], qf[k][0], qf[k][1], qf[k][2], qf[k][3], kf[0], kf[1]);
        mma_bf16_16816(s[1], qf[k][0], qf[k][1], qf[k][2], qf[k][3], kf[2], kf[3]);
      }
      if (kTurn) {
        __syncwarp();  // every lane has read the slot: V of the next block goes there
        load_item(j + 1, 1, here, at);
        advance();
      }
      float mx[2] = {m[0], m[1]};
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const bool live = 16 * b + 8 * h + 2 * t + (e & 1) < ctx;
          s[h][e] = live ? s[h][e] * sc : -INFINITY;
          mx[e >> 1] = fmaxf(mx[e >> 1], s[h][e]);
        }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        mx[q] = fmaxf(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], 1));
        mx[q] = fmaxf(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], 2));
        const float f = exp2f(m[q] - mx[q]);  // (token b of the tile is live, so mx is finite)
        m[q] = mx[q];
        l[q] *= f;
#pragma unroll
        for (int d = 0; d < D / 8; ++d) { o[d][2 * q] *= f; o[d][2 * q + 1] *= f; }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s[h][e] = exp2f(s[h][e] - m[e >> 1]);
          l[e >> 1] += s[h][e];
        }
      const uint32_t p0 = pack_bf16x2(s[0][0], s[0][1]), p1 = pack_bf16x2(s[0][2], s[0][3]);
      const uint32_t p2 = pack_bf16x2(s[1][0], s[1][1]), p3 = pack_bf16x2(s[1][2], s[1][3]);
      if (kTurn) {
        cp_async_wait_group<kSlots - 1>();
        put_new(b, 1, here);
        __syncwarp();
      }
      const uint32_t va = (kTurn ? here : k_st + kRows) + (uint32_t)((lane & 15) * kPitch + (lane >> 4) * 16);
#pragma unroll
      for (int d = 0; d < D / 16; ++d) {
        uint32_t vf[4];
        ldsm_x4_t(va + 32u * d, vf);
        mma_bf16_16816(o[2 * d], p0, p1, p2, p3, vf[0], vf[1]);
        mma_bf16_16816(o[2 * d + 1], p0, p1, p2, p3, vf[2], vf[3]);
      }
    }
    __syncwarp();
    if (kTurn) load_item(j + 2, 0, here, at = rows_of(j + 2));
    else load_item(j + kSlots, 2, here, rows_of(j + kSlots));
    advance();
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    l[q] += __shfl_xor_sync(0xffffffffu, l[q], 1);
    l[q] += __shfl_xor_sync(0xffffffffu, l[q], 2);
  }
  // ---- merge the warps: [warp][head][D] sums, then m and l (every warp has waited for the copies of its blocks)
  __syncthreads();
  float* acc = reinterpret_cast<float*>(smem + 16 * kPitch);
  float* ml = acc + kWarps * 16 * D;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int head = g + 8 * q;
    if (head < group) {
#pragma unroll
      for (int d = 0; d < D / 8; ++d)
        *reinterpret_cast<float2*>(acc + (warp * 16 + head) * D + 8 * d + 2 * t) = make_float2(o[d][2 * q], o[d][2 * q + 1]);
      if (t == 0) { ml[(warp * 16 + head) * 2] = m[q]; ml[(warp * 16 + head) * 2 + 1] = l[q]; }
    }
  }
  __syncthreads();
  for (int i = tid; i < group * D / 2; i += kThreads) {
    const int head = i / (D / 2), d = (i - head * (D / 2)) * 2;
    float top = -INFINITY;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) top = fmaxf(top, ml[(w * 16 + head) * 2]);
    float total = 0.f, x = 0.f, y = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float mw = ml[(w * 16 + head) * 2];
      const float f = mw == -INFINITY ? 0.f : exp2f(mw - top);
      const float2 v = *reinterpret_cast<const float2*>(acc + (w * 16 + head) * D + d);
      total += f * ml[(w * 16 + head) * 2 + 1];
      x += f * v.x;
      y += f * v.y;
    }
    const float inv = total > 0.f ? 1.f / total : 0.f;
    *reinterpret_cast<uint32_t*>(a.out + (int64_t)req * a.Hq * D + (int64_t)(kvh * group + head) * D + d) = pack_bf16x2(x * inv, y * inv);
  }
}

// ------------------------------------------------------------------ host side
inline int decode_attention_launch(const DecAttnArgs& a, int D, cudaStream_t stream) {
  const dim3 grid((unsigned)a.Hk, (unsigned)a.T);
#define B200_DEC_ATTN(DIM)                                                                                                          \
  {                                                                                                                                 \
    const cudaError_t e = cudaFuncSetAttribute(decode_attention_kernel<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, dec_attn_smem<DIM>()); \
    if (e != cudaSuccess) return fail(B200_LORA_ECUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));                          \
    return launch_dependent(decode_attention_kernel<DIM>, "decode_attention_kernel", grid, kDecAttnWarps * 32, dec_attn_smem<DIM>(), stream, a); \
  }
  if (D == 64) B200_DEC_ATTN(64)
  B200_DEC_ATTN(128)
#undef B200_DEC_ATTN
}

}  // namespace b200lora
