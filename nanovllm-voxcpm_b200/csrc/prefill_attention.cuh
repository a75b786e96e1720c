// Causal attention over packed prompts: q, k and v as columns of the packed projection [T, (Hq + 2 Hk) D], bf16.
//
// A CTA takes 128 (position, q head) rows of one request and one kv head: up to eight heads of a group share it, so that a
// K / V tile brought in once serves them all, and a CTA covers few positions (16 with eight heads), which leaves little
// masked work and cuts ragged prompts into many CTAs of even length. Tiles of 64 keys in a two-stage cp.async pipeline; each
// of eight warps keeps 16 rows (mma.sync m16n8k16, online softmax in registers, as in Dao, "FlashAttention-2", 2023). The
// blocks with the longest key ranges are launched first. mma.sync and not tcgen05: for 4001 rows of 12 prompts the arithmetic
// is 4 GFLOP, the time is latency of loads and of the softmax chain. Measured (16 / 2 heads of 64): 12 prompts of 330 rows 23 us,
// one of 4000 135 us, one of 8000 465 us = 282 TFLOP/s of the causal half, which is what mma.sync with two 64-key stages gives; a
// caller with a faster kernel for long prompts takes that (backbone.py has the line and both sides of it).
#pragma once

#include "decode_step.cuh"

namespace b200lora {

constexpr int kPreAttnThreads = 256;
constexpr int kPreAttnRows = 128;  // (position, head) rows of a CTA
constexpr int kPreAttnKeys = 64;   // keys of a tile

struct PreAttnArgs {
  const __nv_bfloat16* qkv; int64_t ld;   // [T, (Hq + 2 Hk) D]
  __nv_bfloat16* out; int64_t out_ld;     // [T, Hq D]
  const int32_t* cu_seqlens;              // [n_req + 1]
  int Hq, Hk, T;
  int h_shift;                            // heads of a CTA = 1 << h_shift
  float scale;
};

template <int D>
__host__ __device__ constexpr int pre_attn_smem() { return 4 * kPreAttnKeys * (D * 2 + 16); }

template <int D>
__global__ void __launch_bounds__(kPreAttnThreads, D == 64 ? 2 : 1) prefill_attention_kernel(const PreAttnArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  constexpr int kPitch = D * 2 + 16, kPieces = D / 8, kTile = kPreAttnKeys * kPitch;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int heads = 1 << a.h_shift, per_cta = kPreAttnRows >> a.h_shift, group = a.Hq / a.Hk;
  const int head0 = (int)blockIdx.x << a.h_shift, kvh = head0 / group, req = blockIdx.y;
  const int q0 = ((int)gridDim.z - 1 - (int)blockIdx.z) * per_cta;
  glue_enter();
  const int begin = a.cu_seqlens[req], len = a.cu_seqlens[req + 1] - begin;
  if (q0 >= len || begin < 0 || begin + len > a.T) return;
  const int n_keys = min(len, q0 + per_cta), n_tiles = (n_keys + kPreAttnKeys - 1) / kPreAttnKeys;
  const uint32_t k_u32 = smem_u32(smem), v_u32 = k_u32 + 2 * kTile;

  const __nv_bfloat16* const k_rows = a.qkv + (int64_t)begin * a.ld + (int64_t)(a.Hq + kvh) * D;
  auto load_tile = [&](int i) {
    const int p = tid % kPieces, stage = (i & 1) * kTile;
#pragma unroll
    for (int j = 0; j < kPreAttnKeys * kPieces / kPreAttnThreads; ++j) {
      const int r = tid / kPieces + j * (kPreAttnThreads / kPieces), key = i * kPreAttnKeys + r;
      const bool live = key < n_keys;  // (rows beyond are zero: their probabilities are zero, their values must be finite)
      const __nv_bfloat16* src = k_rows + (int64_t)(live ? key : 0) * a.ld + p * 8;
      const uint32_t off = (uint32_t)(stage + r * kPitch + p * 16);
      cp_async_16(k_u32 + off, src, live ? 16u : 0u);
      cp_async_16(v_u32 + off, src + (int64_t)a.Hk * D, live ? 16u : 0u);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load_tile(0);

  // q fragments: rows g and g + 8 of the warp's 16
  const int row_lo = warp * 16 + g, row_hi = row_lo + 8;
  const int pos_lo = q0 + (row_lo >> a.h_shift), pos_hi = q0 + (row_hi >> a.h_shift);
  const int head_lo = head0 + (row_lo & (heads - 1)), head_hi = head0 + (row_hi & (heads - 1));
  uint32_t qf[D / 16][4];
  {
    const uint32_t* lo = reinterpret_cast<const uint32_t*>(a.qkv + (int64_t)(begin + min(pos_lo, len - 1)) * a.ld + (int64_t)head_lo * D);
    const uint32_t* hi = reinterpret_cast<const uint32_t*>(a.qkv + (int64_t)(begin + min(pos_hi, len - 1)) * a.ld + (int64_t)head_hi * D);
#pragma unroll
    for (int k = 0; k < D / 16; ++k) {
      qf[k][0] = lo[8 * k + t]; qf[k][1] = hi[8 * k + t];
      qf[k][2] = lo[8 * k + 4 + t]; qf[k][3] = hi[8 * k + 4 + t];
    }
  }
  float o[D / 8][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int d = 0; d < D / 8; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;
  const float sc = a.scale * 1.4426950408889634f;  // scores in units of log2(e)
  const int warp_first = q0 + ((warp * 16) >> a.h_shift);  // first position of the warp: keys up to it need no mask

  for (int i = 0; i < n_tiles; ++i) {
    if (i + 1 < n_tiles) {
      load_tile(i + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const int key0 = i * kPreAttnKeys;
    const uint32_t ks = k_u32 + (uint32_t)((i & 1) * kTile), vs = v_u32 + (uint32_t)((i & 1) * kTile);
    float s[kPreAttnKeys / 8][4];
#pragma unroll
    for (int n = 0; n < kPreAttnKeys / 8; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
    for (int k = 0; k < D / 16; ++k) {
#pragma unroll
      for (int b = 0; b < kPreAttnKeys / 16; ++b) {
        uint32_t kf[4];
        ldsm_x4(ks + (uint32_t)((16 * b + (lane & 7) + ((lane >> 4) << 3)) * kPitch + ((lane >> 3) & 1) * 16) + 32u * k, kf);
        mma_bf16_16816(s[2 * b], qf[k][0], qf[k][1], qf[k][2], qf[k][3], kf[0], kf[1]);
        mma_bf16_16816(s[2 * b + 1], qf[k][0], qf[k][1], qf[k][2], qf[k][3], kf[2], kf[3]);
      }
    }
    float mx[2] = {m[0], m[1]};
    if (key0 + kPreAttnKeys - 1 > warp_first) {
#pragma unroll
      for (int n = 0; n < kPreAttnKeys / 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int key = key0 + 8 * n + 2 * t + (e & 1);
          if (key > ((e >> 1) ? pos_hi : pos_lo) || key >= n_keys) s[n][e] = -INFINITY;
        }
    }
#pragma unroll
    for (int n = 0; n < kPreAttnKeys / 8; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) mx[e >> 1] = fmaxf(mx[e >> 1], s[n][e] * sc);
    float m_use[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      mx[q] = fmaxf(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], 1));
      mx[q] = fmaxf(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], 2));
      m_use[q] = mx[q] == -INFINITY ? 0.f : mx[q];  // (no key of this row so far)
      const float f = exp2f(m[q] - m_use[q]);
      m[q] = mx[q];
      l[q] *= f;
#pragma unroll
      for (int d = 0; d < D / 8; ++d) { o[d][2 * q] *= f; o[d][2 * q + 1] *= f; }
    }
#pragma unroll
    for (int n = 0; n < kPreAttnKeys / 8; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        s[n][e] = exp2f(s[n][e] * sc - m_use[e >> 1]);
        l[e >> 1] += s[n][e];
      }
#pragma unroll
    for (int b = 0; b < kPreAttnKeys / 16; ++b) {
      const uint32_t p0 = pack_bf16x2(s[2 * b][0], s[2 * b][1]), p1 = pack_bf16x2(s[2 * b][2], s[2 * b][3]);
      const uint32_t p2 = pack_bf16x2(s[2 * b + 1][0], s[2 * b + 1][1]), p3 = pack_bf16x2(s[2 * b + 1][2], s[2 * b + 1][3]);
      const uint32_t va = vs + (uint32_t)((16 * b + (lane & 15)) * kPitch + (lane >> 4) * 16);
#pragma unroll
      for (int d = 0; d < D / 16; ++d) {
        uint32_t vf[4];
        ldsm_x4_t(va + 32u * d, vf);
        mma_bf16_16816(o[2 * d], p0, p1, p2, p3, vf[0], vf[1]);
        mma_bf16_16816(o[2 * d + 1], p0, p1, p2, p3, vf[2], vf[3]);
      }
    }
    __syncthreads();  // every warp is done with this stage before it is filled again
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    l[q] += __shfl_xor_sync(0xffffffffu, l[q], 1);
    l[q] += __shfl_xor_sync(0xffffffffu, l[q], 2);
    const int pos = q ? pos_hi : pos_lo;
    if (pos >= len) continue;
    const float inv = l[q] > 0.f ? 1.f / l[q] : 0.f;
    uint32_t* dst = reinterpret_cast<uint32_t*>(a.out + (int64_t)(begin + pos) * a.out_ld + (int64_t)(q ? head_hi : head_lo) * D);
#pragma unroll
    for (int d = 0; d < D / 8; ++d) dst[4 * d + t] = pack_bf16x2(o[d][2 * q] * inv, o[d][2 * q + 1] * inv);
  }
}

inline int prefill_attention_launch(PreAttnArgs a, int D, int n_req, int max_seqlen, cudaStream_t stream) {
  const int group = a.Hq / a.Hk;
  a.h_shift = 0;
  while (a.h_shift < 3 && group % (2 << a.h_shift) == 0) ++a.h_shift;
  const int per_cta = kPreAttnRows >> a.h_shift;
  const dim3 grid((unsigned)(a.Hq >> a.h_shift), (unsigned)n_req, (unsigned)ceil_div_i(max_seqlen, per_cta));
#define B200_PRE_ATTN(DIM)                                                                                                              \
  {                                                                                                                                     \
    const cudaError_t e = cudaFuncSetAttribute(prefill_attention_kernel<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, pre_attn_smem<DIM>()); \
    if (e != cudaSuccess) return fail(B200_LORA_ECUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));                              \
    return launch_dependent(prefill_attention_kernel<DIM>, "prefill_attention_kernel", grid, kPreAttnThreads, pre_attn_smem<DIM>(), stream, a); \
  }
  if (D == 64) B200_PRE_ATTN(64)
  B200_PRE_ATTN(128)
#undef B200_PRE_ATTN
}

}  // namespace b200lora
