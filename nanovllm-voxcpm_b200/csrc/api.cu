// C ABI of the B200 multi-LoRA library: argument checks + kernel dispatch.
// Declarations and the reference interface each entry point replaces: include/b200_lora.h
#include "common.cuh"
#include "generic.cuh"
#include "bgmv_fused.cuh"
#include "metadata.cuh"
#include "tp_exchange.cuh"
#include "slot_loader.cuh"
#include "glue.cuh"
#include "sgmv_tc.cuh"
#include "gemm_tc.cuh"
#include "prefill_cluster.cuh"
#include "linear_pair.cuh"
#include "grouped_tc.cuh"
#include "decode_step.cuh"
#include "prefill_attention.cuh"

using namespace b200lora;

namespace {

int fill_slices(SliceTable& st, int n_slices, const void* const* a_slabs,
                const void* const* b_slabs, const int32_t* out_sizes,
                const int32_t* col_offsets, bool need_a, bool need_b) {
  if (n_slices < 1 || n_slices > B200_LORA_MAX_SLICES)
    return fail(B200_LORA_EINVAL, "n_slices=%d outside [1,%d]", n_slices, B200_LORA_MAX_SLICES);
  st.n = n_slices;
  for (int s = 0; s < B200_LORA_MAX_SLICES; ++s) {
    st.a[s] = st.b[s] = nullptr;
    st.out[s] = st.col[s] = 0;
  }
  for (int s = 0; s < n_slices; ++s) {
    st.out[s] = out_sizes ? out_sizes[s] : 1;
    st.col[s] = col_offsets ? col_offsets[s] : 0;
    if (st.out[s] < 0 || st.col[s] < 0)
      return fail(B200_LORA_EINVAL, "slice %d: negative width/offset", s);
    if (need_a) {
      st.a[s] = a_slabs ? a_slabs[s] : nullptr;
      if (st.a[s] == nullptr && st.out[s] > 0) return fail(B200_LORA_EINVAL, "slice %d: null lora_A slab", s);
    }
    if (need_b) {
      st.b[s] = b_slabs ? b_slabs[s] : nullptr;
      if (st.b[s] == nullptr && st.out[s] > 0) return fail(B200_LORA_EINVAL, "slice %d: null lora_B slab", s);
    }
  }
  return B200_LORA_OK;
}

// y[row, slice columns] = -0.0 (sign bit only) for every slice; elem = bytes per element
__global__ void fill_neg_zero_kernel(void* y, int64_t y_ld, const SliceTable st, int elem) {
  const int64_t row = blockIdx.x;
  for (int s = 0; s < st.n; ++s) {
    if (elem == 2) {
      uint16_t* dst = static_cast<uint16_t*>(y) + row * y_ld + st.col[s];
      for (int i = threadIdx.x; i < st.out[s]; i += blockDim.x) dst[i] = 0x8000u;
    } else {
      uint32_t* dst = static_cast<uint32_t*>(y) + row * y_ld + st.col[s];
      for (int i = threadIdx.x; i < st.out[s]; i += blockDim.x) dst[i] = 0x80000000u;
    }
  }
}

bool valid_dtype(int d) { return d == B200_LORA_BF16 || d == B200_LORA_F16 || d == B200_LORA_F32; }

template <typename T>
int launch_generic_add(void* y, int64_t y_ld, const void* x, int64_t x_ld, int T_rows, int in_dim,
                       const SliceTable& st, int S, int r_max, const int32_t* rank_per_slot,
                       const float* scale_per_slot, const int32_t* token_to_slot, float scaling,
                       cudaStream_t stream) {
  const size_t smem = sizeof(float) * st.n * r_max;
  generic_add_kernel<T><<<T_rows, kGenericThreads, smem, stream>>>(
      static_cast<T*>(y), y_ld, static_cast<const T*>(x), x_ld, in_dim, st, S, r_max,
      rank_per_slot, scale_per_slot, token_to_slot, scaling);
  return check_launch("generic_add_kernel");
}

template <typename T, typename TO>
int launch_generic_shrink(void* out, const void* x, int64_t x_ld, int T_rows, int in_dim,
                          const SliceTable& st, int S, int r_max, const int32_t* token_to_slot,
                          float scaling, cudaStream_t stream) {
  generic_shrink_kernel<T, TO><<<T_rows, kGenericThreads, 0, stream>>>(
      static_cast<TO*>(out), static_cast<const T*>(x), x_ld, T_rows, in_dim, st, S, r_max,
      token_to_slot, scaling);
  return check_launch("generic_shrink_kernel");
}

template <typename T, typename TI>
int launch_generic_expand(void* y, int64_t y_ld, const void* tmp, int T_rows, const SliceTable& st,
                          int S, int r_max, const int32_t* token_to_slot, int add_inputs,
                          cudaStream_t stream) {
  const size_t smem = sizeof(float) * st.n * r_max;
  generic_expand_kernel<T, TI><<<T_rows, kGenericThreads, smem, stream>>>(
      static_cast<T*>(y), y_ld, static_cast<const TI*>(tmp), T_rows, st, S, r_max, token_to_slot,
      add_inputs);
  return check_launch("generic_expand_kernel");
}

}  // namespace

namespace {

// Whether a bf16 batch is large enough for the prefill kernels rather than the bucket kernel (an adapter read once per 16 rows of it),
// by the adapter bytes that the bucket kernel would read; 16 rank rows take it as long as 32.
//   prefill_cluster_kernel (adds): us per projection, bucket / prefill kernel, eight prompts: 1024-wide, rank 32: 1000 rows, qkv (18
//   MB) 6.9 / 10.1, gate_up (41 MB) 9.4 / 11.9, 2048 rows, qkv (36 MB) 8.2 / 11.5, 2400 (42 MB) 12.7 / 11.1, o (20 MB) 6.2 / 8.6;
//   2048-wide, rank 32: 1000 rows, qkv (35 MB) 9.1 / 12.1, 1200 (42 MB) 14.9 / 12.9; rank 64: gate_up of 400 rows (52 MB) 12.7 / 13.0,
//   of 511 (67 MB) 21.4 / 13.5. The bucket kernel's time goes up in steps, a wave of clusters each, so that some batches lie on the
//   wrong side of any line by bytes (the 41 MB above). Over 1560 measured points (200 to 3300 rows of one to eight prompts, three widths,
//   ranks 16 to 64) the line is 2.4 % slower than the better choice each time, one at 75 windows and 50 MB 5.2. Adapters of rank 16 that
//   went to the bucket kernel, which keeps their intermediate as two numbers, still do: up to 1184 rows and 50 MB. Rank 64 is not
//   asked for its bytes from 512 rows on, as it never was: 5.3 % behind the better choice there, most with few bytes (1024 -> 1024,
//   512 rows, 8 MB 4.8 / 7.9; 2048 -> 2048, 724 rows, 24 MB 7.9 / 9.4).
//   sgmv_shrink_kernel and the launch behind it (operators, slices that do not tile the output; at least 11 us for the pair): bucket /
//   pair, six prompts: 1024-wide, rank 32, 900 rows, qkv (16 MB) 6.7 / 13.5, gate_up (37 MB) 8.9 / 15.1, 1500 rows 11.5 / 13.8 and
//   (61 MB) 18.6 / 20.4; 2048-wide, rank 32, 900 rows, gate_up (59 MB) 19.0 / 19.1, 1500 rows (98 MB) 32.9 / 24.7; rank 64, 900
//   rows, qkv (63 MB) 18.8 / 17.0, 1500 rows 33.2 / 19.3.
inline bool prefill_sized(int32_t T, const SliceTable& st, int32_t r_max, int32_t in_dim, bool expand, bool one_launch) {
  constexpr int64_t kMB = 1000 * 1000;
  const int windows = ceil_div_i(T, kBgmvTok);
  int64_t bytes = 0;
  for (int s = 0; s < st.n; ++s)
    if (st.out[s] > 0 || !expand) bytes += 2 * (int64_t)r_max * (in_dim + (expand ? st.out[s] : 0));
  bytes *= windows;
  const bool pair_sized = T >= kSgmvAutoMinTokens && (r_max > 32 || bytes > 50 * kMB);
  if (pair_sized || !one_launch) return pair_sized;
  if (r_max <= 16 && windows <= 74) return false;
  return bytes * (r_max <= 16 ? 2 : 1) > (T < kSgmvAutoMinTokens ? 52 : 38) * kMB || windows > 240;
}

// Rows a bucket from which a batch may be one of whole prompts. The prefill kernels take the rows of a block's slots apart (the one-launch
// kernel wherever they lie, the pair run by run), so a decode batch that is taken for one costs a pass over x for every one to four
// slots of a block. Batches of fewer than 512 rows are more often that: at 64 rows a bucket rows that lie scattered cost adds of rank 64
// (2048- and 4096-wide) 0.63 to 1.08 of the bucket kernel's time a layer, of rank 32 (4096-wide) up to 1.18, at 32 up to 1.9; whole prompts 0.7.
inline bool rows_for_prefill(int32_t T, int32_t n_buckets) { return T >= (T < kSgmvAutoMinTokens ? 64 : 32) * (int64_t)n_buckets; }

}  // namespace

extern "C" {

int lora_b200_version(void) { return B200_LORA_ABI_VERSION; }

const char* lora_b200_last_error(void) { return error_buffer(); }

int lora_b200_set_option(int32_t key, int32_t value) {
  if (key == B200_LORA_OPT_CLUSTER) {
    if (value != 0 && value != 1 && value != 2 && value != 4 && value != 8)
      return fail(B200_LORA_EINVAL, "cluster size %d not in {0,1,2,4,8}", value);
    bgmv_options().cluster = value;
    return B200_LORA_OK;
  }
  if (key == B200_LORA_OPT_PDL) {
    bgmv_options().pdl = value != 0;
    return B200_LORA_OK;
  }
  if (key == B200_LORA_OPT_RING_KB) {
    if (value < 0 || value > 227) return fail(B200_LORA_EINVAL, "ring size %d KB outside [0, 227]", value);
    bgmv_options().ring_kb = value;
    return B200_LORA_OK;
  }
  if (key == B200_LORA_OPT_PEER_POLL_LIMIT) {
    if (value < 0) return fail(B200_LORA_EINVAL, "poll limit %d is negative", value);
    tp_spin_limit() = value == 0 ? kTpSpinLimit : value;
    return B200_LORA_OK;
  }
  if (key == B200_LORA_OPT_KSPLIT) {
    bgmv_options().ksplit = value != 0;
    return B200_LORA_OK;
  }
  return fail(B200_LORA_EINVAL, "unknown option %d", key);
}

int lora_b200_build_metadata(const int32_t* token_to_slot, int32_t T, int32_t S, int32_t convention,
                             int32_t* sorted_idx, int32_t* slot_ids, int32_t* counts, int32_t* offsets,
                             int32_t* info, void* stream) {
  return build_metadata(token_to_slot, T, S, convention, sorted_idx, slot_ids, counts, offsets, info,
                        static_cast<cudaStream_t>(stream));
}

int lora_b200_load_slot(const void* staging, int32_t n_desc, int64_t max_elems, void* stream) {
  return slot_load_launch(staging, n_desc, max_elems, static_cast<cudaStream_t>(stream));
}

int lora_b200_glue_add_rmsnorm(void* normed, int64_t normed_ld, void* hidden_out, int64_t hidden_ld, const void* x,
                               int64_t x_ld, const void* residual, int64_t residual_ld, const void* weight, int32_t T,
                               int32_t hidden, float eps, int32_t norm_of_rounded_sum, int32_t dtype, void* stream) {
  return add_rmsnorm_launch(normed, normed_ld, hidden_out, hidden_ld, x, x_ld, residual, residual_ld, weight, T, hidden, eps,
                            norm_of_rounded_sum, dtype, static_cast<cudaStream_t>(stream));
}

int lora_b200_glue_rope_kv_store(void* qkv, int64_t qkv_ld, int32_t T, int32_t num_heads, int32_t num_kv_heads,
                                 int32_t head_dim, const int64_t* positions, const void* cos_table, const void* sin_table,
                                 int32_t table_dim, int32_t table_dtype, int32_t max_position, void* k_cache, void* v_cache,
                                 const int32_t* slot_mapping, int32_t dtype, void* stream) {
  RopeKvParams p;
  p.qkv = qkv; p.qkv_ld = qkv_ld; p.T = T; p.Hq = num_heads; p.Hk = num_kv_heads; p.D = head_dim;
  p.positions = positions; p.cos = cos_table; p.sin = sin_table;
  p.table_dim = table_dim; p.table_dtype = table_dtype; p.max_pos = max_position;
  p.k_cache = k_cache; p.v_cache = v_cache; p.slot_mapping = slot_mapping;
  p.apply_rope = (cos_table != nullptr || sin_table != nullptr || positions != nullptr) ? 1 : 0;
  return rope_kv_store_launch(p, dtype, static_cast<cudaStream_t>(stream));
}

int lora_b200_glue_silu_mul(void* out, int64_t out_ld, const void* gate_up, int64_t gate_up_ld, int32_t T,
                            int32_t intermediate, int32_t dtype, void* stream) {
  return silu_mul_launch(out, out_ld, gate_up, gate_up_ld, T, intermediate, dtype, static_cast<cudaStream_t>(stream));
}

int lora_b200_decode_planes(int32_t in_dim, int32_t out) {
  if (in_dim < 1 || out < 1) return 0;
  return decode_gemm_parts(in_dim, out) + 1;
}

// Argument checks of a projection of the decode chain, and the plan of the adapters' part of the launch. Reads no pointer.
static int decode_linear_plan(BgmvParams* plan, float* planes, const void* x, int64_t x_ld, int32_t T, int32_t in_dim, const void* weight,
                              int64_t w_ld, int32_t out_total, int32_t n_slices, const void* const* a_slabs,
                              const void* const* b_slabs, const int32_t* out_sizes, const int32_t* col_offsets, int32_t S,
                              int32_t r_max, const int32_t* rank_per_slot, const int32_t* token_to_slot,
                              const int32_t* sorted_idx, const int32_t* slot_ids, const int32_t* counts, const int32_t* offsets,
                              int32_t n_buckets) {
  if (T < 1 || T > kDecMaxRows || in_dim < 1 || out_total < 1) return fail(B200_LORA_EINVAL, "decode_linear: bad sizes T=%d in=%d out=%d", T, in_dim, out_total);
  if (planes == nullptr || x == nullptr || weight == nullptr) return fail(B200_LORA_EINVAL, "decode_linear: null pointer");
  if (in_dim % 64 != 0 || x_ld % 8 != 0 || w_ld % 8 != 0 || x_ld < in_dim || w_ld < in_dim || out_total % 8 != 0 || !aligned16(planes) || !aligned16(x) ||
      !aligned16(weight))
    return fail(B200_LORA_EUNSUPPORTED, "decode_linear: in_dim must be a multiple of 64, out of 8, rows 16-byte aligned");
  if (n_slices <= 0) return B200_LORA_OK;
  if (out_sizes == nullptr || col_offsets == nullptr || token_to_slot == nullptr) return fail(B200_LORA_EINVAL, "decode_linear: null slice or slot array");
  BgmvProblem bp = {};
  if (int rc = fill_slices(bp.st, n_slices, a_slabs, b_slabs, out_sizes, col_offsets, true, true)) return rc;
  int covered = 0;
  for (int s = 0; s < bp.st.n; ++s) {
    if (bp.st.col[s] + bp.st.out[s] > out_total) return fail(B200_LORA_EINVAL, "slice %d exceeds the output width", s);
    covered += bp.st.out[s];
  }
  if (covered != out_total) return fail(B200_LORA_EUNSUPPORTED, "decode_linear: the slices must cover the output");
  const int parts = decode_gemm_parts(in_dim, out_total);
  bp.y = planes + (size_t)parts * T * out_total; bp.y_ld = out_total;
  bp.x = x; bp.x_ld = x_ld; bp.T = T; bp.in_dim = in_dim; bp.S = S; bp.r_max = r_max;
  bp.rank_per_slot = rank_per_slot; bp.scale_per_slot = nullptr;
  bp.sorted_idx = sorted_idx; bp.slot_ids = slot_ids; bp.counts = counts; bp.offsets = offsets; bp.n_buckets = n_buckets;
  bp.scaling = 1.0f; bp.mode = 4; bp.kind = r_max % 32 != 0 ? 1 : 0; bp.token_to_slot = token_to_slot;
  bp.beside = decode_gemm_ctas(in_dim, out_total);
  if (S < 1 || r_max < 1) return fail(B200_LORA_EINVAL, "decode_linear: bad sizes S=%d r_max=%d", S, r_max);
  if (sorted_idx == nullptr || slot_ids == nullptr || counts == nullptr || offsets == nullptr)
    return fail(B200_LORA_EINVAL, "decode_linear: needs the bucket arrays");
  const char* why = nullptr;
  if (!bgmv_plan(bp, plan, &why)) return fail(B200_LORA_EUNSUPPORTED, "decode_linear: %s", why);
  return B200_LORA_OK;
}

int lora_b200_decode_linear_check(int32_t T, int32_t in_dim, const void* weight, int64_t w_ld, int32_t out_total, int32_t n_slices,
                                  const void* const* a_slabs, const void* const* b_slabs, const int32_t* out_sizes,
                                  const int32_t* col_offsets, int32_t S, int32_t r_max, int32_t n_buckets) {
  BgmvParams plan;
  float* const some = reinterpret_cast<float*>(uintptr_t(256));  // (stands for the arrays of a step; not read)
  const int32_t* const index = reinterpret_cast<const int32_t*>(some);
  return decode_linear_plan(&plan, some, some, in_dim, T, in_dim, weight, w_ld, out_total, n_slices, a_slabs, b_slabs, out_sizes, col_offsets,
                               S, r_max, nullptr, index, index, index, index, index, n_buckets);
}

int lora_b200_decode_linear(float* planes, const void* x, int64_t x_ld, int32_t T, int32_t in_dim, const void* weight, int64_t w_ld,
                            int32_t out_total, int32_t n_slices, const void* const* a_slabs, const void* const* b_slabs,
                            const int32_t* out_sizes, const int32_t* col_offsets, int32_t S, int32_t r_max,
                            const int32_t* rank_per_slot, const int32_t* token_to_slot, const int32_t* sorted_idx,
                            const int32_t* slot_ids, const int32_t* counts, const int32_t* offsets, int32_t n_buckets,
                            void* stream) {
  BgmvParams plan;
  if (int rc = decode_linear_plan(&plan, planes, x, x_ld, T, in_dim, weight, w_ld, out_total, n_slices, a_slabs, b_slabs, out_sizes, col_offsets, S,
                                  r_max, rank_per_slot, token_to_slot, sorted_idx, slot_ids, counts, offsets, n_buckets))
    return rc;
  return decode_linear_launch(planes, x, x_ld, T, in_dim, weight, w_ld, out_total, n_slices > 0 ? &plan : nullptr, static_cast<cudaStream_t>(stream));
}

int lora_b200_decode_add_rmsnorm(void* normed, void* hidden_out, const float* planes, int32_t n_planes, const void* residual,
                                 const void* weight, int32_t T, int32_t hidden, float eps, void* stream) {
  if (T < 1 || hidden < 8 || hidden % 8 != 0 || hidden > 4096) return fail(B200_LORA_EUNSUPPORTED, "decode_add_rmsnorm: bad shape T=%d H=%d", T, hidden);
  if (n_planes < 1 || n_planes > kDecMaxPlanes) return fail(B200_LORA_EINVAL, "decode_add_rmsnorm: %d planes", n_planes);
  if (!normed || !hidden_out || !planes || !residual || !weight) return fail(B200_LORA_EINVAL, "decode_add_rmsnorm: null pointer");
  if (!aligned16(normed) || !aligned16(hidden_out) || !aligned16(planes) || !aligned16(residual) || !aligned16(weight))
    return fail(B200_LORA_EUNSUPPORTED, "decode_add_rmsnorm: rows must be 16-byte aligned");
  using B = __nv_bfloat16;
  return launch_dependent(decode_add_rmsnorm_kernel, "decode_add_rmsnorm_kernel", dim3((unsigned)T), round_up_i(hidden / 4, 32), 0,
                          static_cast<cudaStream_t>(stream), static_cast<B*>(normed), static_cast<B*>(hidden_out), planes, n_planes,
                          static_cast<const B*>(residual), static_cast<const B*>(weight), T, hidden, eps);
}

int lora_b200_decode_silu_mul(void* out, const float* planes, int32_t n_planes, int32_t T, int32_t intermediate, void* stream) {
  if (T < 1 || intermediate < 8 || intermediate % 8 != 0) return fail(B200_LORA_EUNSUPPORTED, "decode_silu_mul: bad shape T=%d I=%d", T, intermediate);
  if (n_planes < 1 || n_planes > kDecMaxPlanes) return fail(B200_LORA_EINVAL, "decode_silu_mul: %d planes", n_planes);
  if (!out || !planes || !aligned16(out) || !aligned16(planes)) return fail(B200_LORA_EINVAL, "decode_silu_mul: null or misaligned pointer");
  const int ctas = std::min(4 * 148, ceil_div_i(T * (intermediate / 4), 256));
  return launch_dependent(decode_silu_mul_kernel, "decode_silu_mul_kernel", dim3((unsigned)ctas), 256, 0, static_cast<cudaStream_t>(stream),
                          static_cast<__nv_bfloat16*>(out), planes, n_planes, T, intermediate);
}

int lora_b200_decode_attention(void* out, const float* planes, int32_t n_planes, int32_t T, int32_t num_heads, int32_t num_kv_heads,
                               int32_t head_dim, const int64_t* positions, const void* cos_table, const void* sin_table,
                               int32_t table_dim, int32_t table_dtype, int32_t max_position, void* k_cache, void* v_cache,
                               const int32_t* block_tables, int32_t max_blocks, int32_t block_size, const int32_t* context_lens,
                               const int64_t* slot_mapping, float scale, void* stream) {
  if (T < 1 || T > 65535 || num_kv_heads < 1 || num_heads % num_kv_heads != 0 || num_heads / num_kv_heads > 16 || (head_dim != 64 && head_dim != 128))
    return fail(B200_LORA_EUNSUPPORTED, "decode_attention: T=%d heads=%d / %d of %d", T, num_heads, num_kv_heads, head_dim);
  if (n_planes < 1 || n_planes > kDecMaxPlanes || max_blocks < 1 || block_size < 1 || max_position < 1)
    return fail(B200_LORA_EINVAL, "decode_attention: bad sizes");
  if ((table_dim != head_dim && table_dim != head_dim / 2) || !valid_dtype(table_dtype)) return fail(B200_LORA_EINVAL, "decode_attention: bad rotation table");
  if (!out || !planes || !positions || !cos_table || !sin_table || !k_cache || !v_cache || !block_tables || !context_lens || !slot_mapping)
    return fail(B200_LORA_EINVAL, "decode_attention: null pointer");
  if (!aligned16(k_cache) || !aligned16(v_cache) || !aligned16(planes) || (reinterpret_cast<uintptr_t>(out) & 3u))
    return fail(B200_LORA_EUNSUPPORTED, "decode_attention: caches must be 16-byte aligned");
  DecAttnArgs a;
  a.part = planes; a.planes = n_planes; a.ld = (num_heads + 2 * num_kv_heads) * head_dim; a.T = T; a.Hq = num_heads; a.Hk = num_kv_heads;
  a.positions = positions; a.cos = cos_table; a.sin = sin_table; a.table_dim = table_dim; a.table_dtype = table_dtype; a.max_pos = max_position;
  a.k_cache = static_cast<__nv_bfloat16*>(k_cache); a.v_cache = static_cast<__nv_bfloat16*>(v_cache);
  a.block_tables = block_tables; a.max_blocks = max_blocks; a.block_size = block_size; a.context_lens = context_lens; a.slot_mapping = slot_mapping;
  a.out = static_cast<__nv_bfloat16*>(out); a.scale = scale;
  return decode_attention_launch(a, head_dim, static_cast<cudaStream_t>(stream));
}

int lora_b200_prefill_attention(void* out, int64_t out_ld, const void* qkv, int64_t qkv_ld, int32_t T, int32_t num_heads,
                                int32_t num_kv_heads, int32_t head_dim, const int32_t* cu_seqlens, int32_t n_seqs,
                                int32_t max_seqlen, float scale, void* stream) {
  if (T < 0 || n_seqs < 0 || max_seqlen < 0) return fail(B200_LORA_EINVAL, "prefill_attention: bad sizes");
  if (T == 0 || n_seqs == 0 || max_seqlen == 0) return B200_LORA_OK;
  if (num_kv_heads < 1 || num_heads < 1 || num_heads % num_kv_heads != 0 || (head_dim != 64 && head_dim != 128) || n_seqs > 65535 ||
      max_seqlen > (1 << 19))
    return fail(B200_LORA_EUNSUPPORTED, "prefill_attention: heads=%d / %d of %d, %d sequences", num_heads, num_kv_heads, head_dim, n_seqs);
  if (!out || !qkv || !cu_seqlens) return fail(B200_LORA_EINVAL, "prefill_attention: null pointer");
  const int width = (num_heads + 2 * num_kv_heads) * head_dim;
  if (qkv_ld < width || out_ld < num_heads * head_dim) return fail(B200_LORA_EINVAL, "prefill_attention: row stride smaller than row");
  if (!aligned16(qkv) || qkv_ld % 8 != 0 || out_ld % 2 != 0 || (reinterpret_cast<uintptr_t>(out) & 3u))
    return fail(B200_LORA_EUNSUPPORTED, "prefill_attention: rows must be 16-byte aligned");
  PreAttnArgs a = {};
  a.qkv = static_cast<const __nv_bfloat16*>(qkv); a.ld = qkv_ld; a.out = static_cast<__nv_bfloat16*>(out); a.out_ld = out_ld;
  a.cu_seqlens = cu_seqlens; a.Hq = num_heads; a.Hk = num_kv_heads; a.T = T; a.scale = scale;
  return prefill_attention_launch(a, head_dim, n_seqs, max_seqlen, static_cast<cudaStream_t>(stream));
}

size_t lora_b200_tp_exchange_bytes(int32_t tp, int32_t capacity) { return tp_exchange_bytes(tp, capacity); }

int lora_b200_tp_allreduce(const float* partial, float* out, int32_t count, void* const* peer_buffers, int32_t rank,
                           int32_t tp, int32_t capacity, void* stream) {
  return tp_allreduce_launch(partial, out, count, peer_buffers, rank, tp, capacity, static_cast<cudaStream_t>(stream));
}

#ifdef B200_TRACE
// Tuning builds only: copies the phase timeline of the last fused-decode launch.
int lora_b200_debug_trace(long long* out, int32_t n_values) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_b200_trace, sizeof(long long) * (size_t)n_values);
  return e == cudaSuccess ? 0 : B200_LORA_ECUDA;
}
#endif

int lora_b200_device_status(int32_t* status, int32_t reset) {
  if (status == nullptr) return fail(B200_LORA_EINVAL, "null status pointer");
  int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_b200_status, sizeof(int));
  if (e != cudaSuccess) return fail(B200_LORA_ECUDA, "cudaMemcpyFromSymbol: %s", cudaGetErrorString(e));
  *status = v;
  if (reset) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_b200_status, &zero, sizeof(int));
    if (e != cudaSuccess) return fail(B200_LORA_ECUDA, "cudaMemcpyToSymbol: %s", cudaGetErrorString(e));
  }
  return B200_LORA_OK;
}

static int linear_lora_checked(bool silu, void* y, int64_t y_ld, const void* x, int64_t x_ld, int32_t T, int32_t in_dim,
                          const void* weight, int64_t w_ld, int32_t out_total, const void* bias, int32_t n_slices,
                          const void* const* a_slabs, const void* const* b_slabs, const int32_t* out_sizes,
                          const int32_t* col_offsets, int32_t S, int32_t r_max, const float* scale_per_slot,
                          const int32_t* token_to_slot, float scaling, void* workspace, size_t workspace_bytes,
                          void* stream) {
  if (T < 0 || in_dim < 1 || out_total < 1) return fail(B200_LORA_EINVAL, "bad sizes T=%d in=%d out=%d", T, in_dim, out_total);
  if (T == 0) return B200_LORA_OK;
  if (y == nullptr || x == nullptr || weight == nullptr) return fail(B200_LORA_EINVAL, "null y / x / weight");
  if (y_ld < (silu ? out_total / 2 : out_total) || x_ld < in_dim || w_ld < in_dim) return fail(B200_LORA_EINVAL, "row stride smaller than row");
  LinearProblem lp;
  lp.weight = weight; lp.w_ld = w_ld; lp.n_total = out_total; lp.bias = bias; lp.silu = silu;
  SliceTable st;
  st.n = 0;
  for (int s = 0; s < B200_LORA_MAX_SLICES; ++s) { st.a[s] = st.b[s] = nullptr; st.out[s] = st.col[s] = 0; }
  if (n_slices > 0 && token_to_slot != nullptr) {
    if (S < 1 || r_max < 1) return fail(B200_LORA_EINVAL, "bad sizes S=%d r_max=%d", S, r_max);
    if (out_sizes == nullptr || col_offsets == nullptr) return fail(B200_LORA_EINVAL, "null out_sizes / col_offsets");
    if (int rc = fill_slices(st, n_slices, a_slabs, b_slabs, out_sizes, col_offsets, true, true)) return rc;
    for (int s = 0; s < st.n; ++s)
      if (st.col[s] + st.out[s] > out_total) return fail(B200_LORA_EINVAL, "slice %d exceeds the output width", s);
  }
  lp.lora.y = y; lp.lora.y_ld = y_ld; lp.lora.x = x; lp.lora.x_ld = x_ld; lp.lora.T = T; lp.lora.in_dim = in_dim;
  lp.lora.S = S; lp.lora.r_max = r_max; lp.lora.st = st; lp.lora.scale_per_slot = scale_per_slot;
  lp.lora.token_to_slot = token_to_slot; lp.lora.scaling = scaling;
  return linear_lora_launch(lp, workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}

int lora_b200_linear_lora(void* y, int64_t y_ld, const void* x, int64_t x_ld, int32_t T, int32_t in_dim, const void* weight, int64_t w_ld, int32_t out_total,
                          const void* bias, int32_t n_slices, const void* const* a_slabs, const void* const* b_slabs, const int32_t* out_sizes,
                          const int32_t* col_offsets, int32_t S, int32_t r_max, const float* scale_per_slot, const int32_t* token_to_slot,
                          float scaling, void* workspace, size_t workspace_bytes, void* stream) {
  return linear_lora_checked(false, y, y_ld, x, x_ld, T, in_dim, weight, w_ld, out_total, bias, n_slices, a_slabs, b_slabs, out_sizes, col_offsets, S,
                             r_max, scale_per_slot, token_to_slot, scaling, workspace, workspace_bytes, stream);
}

int lora_b200_linear_lora_silu(void* y, int64_t y_ld, const void* x, int64_t x_ld, int32_t T, int32_t in_dim, const void* weight, int64_t w_ld, int32_t out_total,
                          int32_t n_slices, const void* const* a_slabs, const void* const* b_slabs, const int32_t* out_sizes,
                          const int32_t* col_offsets, int32_t S, int32_t r_max, const float* scale_per_slot, const int32_t* token_to_slot,
                          float scaling, void* workspace, size_t workspace_bytes, void* stream) {
  return linear_lora_checked(true, y, y_ld, x, x_ld, T, in_dim, weight, w_ld, out_total, nullptr, n_slices, a_slabs, b_slabs, out_sizes, col_offsets, S,
                             r_max, scale_per_slot, token_to_slot, scaling, workspace, workspace_bytes, stream);
}

size_t lora_b200_workspace_bytes(int32_t T, int32_t n_slices, int32_t r_max) {
  if (T < 0 || n_slices < 1 || r_max < 1) return 0;
  return std::max(sgmv_workspace_bytes(T, n_slices, r_max), grouped_workspace_bytes(T, n_slices, r_max));
}

size_t lora_b200_grouped_workspace_bytes(int32_t T, int32_t in_dim, int32_t n_slices, int32_t r_max, int32_t n_buckets) {
  if (T < 0 || in_dim < 1 || n_slices < 1 || n_slices > B200_LORA_MAX_SLICES || n_buckets < 1 || (r_max != 16 && r_max != 32 && r_max != 64)) return 0;
  GroupedProblem b = {};
  b.T = T; b.in_dim = in_dim; b.r_max = r_max; b.n_buckets = n_buckets; b.st.n = n_slices;
  for (int s = 0; s < n_slices; ++s) b.st.out[s] = 8;
  int parts;
  return grouped_need(b, &parts);
}

int32_t lora_b200_bucket_cluster(int32_t T, int32_t in_dim, int32_t n_slices, const int32_t* out_sizes, int32_t r_max, int32_t n_buckets,
                                 int32_t dtype, int32_t beside_gemm) {
  if (T < 1 || in_dim < 1 || r_max < 1 || out_sizes == nullptr || n_slices < 1 || n_slices > B200_LORA_MAX_SLICES ||
      (dtype != B200_LORA_BF16 && dtype != B200_LORA_F16))
    return 0;
  void* const some = reinterpret_cast<void*>(uintptr_t(256));  // (stands for the arrays of a call; not read)
  BgmvProblem b = {};
  int out_total = 0;
  b.st.n = n_slices;
  for (int s = 0; s < n_slices; ++s) {
    if (out_sizes[s] < 0) return 0;
    b.st.a[s] = b.st.b[s] = some; b.st.out[s] = out_sizes[s]; b.st.col[s] = out_total;
    out_total += out_sizes[s];
  }
  b.y = some; b.y_ld = out_total; b.x = some; b.x_ld = in_dim; b.T = T; b.in_dim = in_dim; b.S = 1; b.r_max = r_max; b.n_buckets = n_buckets;
  b.kind = dtype == B200_LORA_F16 ? 2 : (r_max % 32 != 0 ? 1 : 0);
  if (beside_gemm) { b.mode = 4; b.beside = decode_gemm_ctas(in_dim, out_total); }
  BgmvParams p;
  return bgmv_plan(b, &p, nullptr) ? 1 << p.c_shift : 0;
}

int32_t lora_b200_prefill_plan(int32_t T, int32_t in_dim, int32_t n_slices, const int32_t* out_sizes, int32_t r_max, int32_t form, int32_t* split) {
  if (T < 1 || in_dim < 1 || r_max < 1 || out_sizes == nullptr || n_slices < 1 || n_slices > B200_LORA_MAX_SLICES || form < 0 || form > 2 || split == nullptr)
    return 0;
  void* const some = reinterpret_cast<void*>(uintptr_t(256));  // (stands for the arrays of a call; not read)
  LinearProblem p = {};
  SgmvProblem& b = p.lora;
  int n = 0;
  b.st.n = n_slices;
  for (int s = 0; s < n_slices; ++s) {
    if (out_sizes[s] < 0) return 0;
    b.st.a[s] = b.st.b[s] = some; b.st.out[s] = out_sizes[s]; b.st.col[s] = p.n_total;
    p.n_total += out_sizes[s];
    n += out_sizes[s] > 0;
  }
  b.y = some; b.x = some; b.y_ld = p.n_total; b.x_ld = in_dim; b.T = T; b.in_dim = in_dim; b.S = 1; b.r_max = r_max;
  p.silu = form == 2;
  if (!sgmv_supported(b, nullptr)) return 0;
  PcArgs a = {};
  int kernel;
  if (form == 0) {
    if (!prefill_cluster_add_ok(b)) return kLinearTiles;
    if (!prefill_cluster_plan(b, n, p.n_total, false, &a)) return 0;
    kernel = kLinearCluster;
  } else {
    kernel = linear_kernel(p, true, &a);
  }
  if (kernel != kLinearCluster) return kernel;
  const int width = (a.groups > 1 ? prefill_cluster_need(a, n, a.group_cols) : n) * r_max, nk_part = ceil_div_i(in_dim / kSgmvBK, a.ck);
  split[0] = a.ck; split[1] = a.groups; split[2] = a.bm;
  split[3] = form == 0 ? ceil_div_i(ceil_div_i(a.group_cols, a.tile_cols), a.ck) : ceil_div_i(std::min(a.cta_cols, a.group_cols), a.tile_cols);
  split[4] = a.gmax; split[5] = ceil_div_i(width, a.part_cols); split[6] = a.stages;
  split[7] = 0;
  for (int g = 1; g <= a.gmax; ++g)
    if (form != 0 || a.off_part / (kSgmvBM * kSgmvBK * 2 + g * width * kSgmvBK * 2) >= std::min(nk_part, 4)) split[7] = g;
  return kernel;
}

int lora_b200_shrink_allreduce_expand(void* y, int64_t y_ld, const void* x, int64_t x_ld, int32_t T, int32_t in_dim,
                                      int32_t n_slices, const void* const* a_slabs, const void* const* b_slabs,
                                      const int32_t* out_sizes, const int32_t* col_offsets, int32_t S, int32_t r_max,
                                      const int32_t* rank_per_slot, const float* scale_per_slot,
                                      const int32_t* token_to_slot, const int32_t* sorted_idx, const int32_t* slot_ids,
                                      const int32_t* counts, const int32_t* offsets, int32_t n_buckets, float scaling,
                                      int32_t dtype, float* tmp, void* const* peer_buffers, int32_t rank, int32_t tp,
                                      int32_t capacity, void* stream) {
  if (!valid_dtype(dtype)) return fail(B200_LORA_EINVAL, "unknown dtype %d", dtype);
  if (T < 0 || in_dim < 1 || S < 1 || r_max < 1)
    return fail(B200_LORA_EINVAL, "bad sizes T=%d in=%d S=%d r_max=%d", T, in_dim, S, r_max);
  if (T == 0) return B200_LORA_OK;
  if (y == nullptr || x == nullptr || token_to_slot == nullptr || tmp == nullptr)
    return fail(B200_LORA_EINVAL, "null y / x / token_to_slot / tmp");
  if (out_sizes == nullptr || col_offsets == nullptr) return fail(B200_LORA_EINVAL, "null out_sizes / col_offsets");
  if (tp < 1 || rank < 0 || rank >= tp) return fail(B200_LORA_EINVAL, "rank %d of %d", rank, tp);
  if (tp > 1 && peer_buffers == nullptr) return fail(B200_LORA_EINVAL, "null peer_buffers with tp=%d", tp);
  SliceTable st;
  if (int rc = fill_slices(st, n_slices, a_slabs, b_slabs, out_sizes, col_offsets, true, true)) return rc;
  int n_act = 0;
  int64_t width = 0;
  for (int s = 0; s < st.n; ++s) {
    if (st.out[s] == 0) return fail(B200_LORA_EUNSUPPORTED, "tensor-parallel exchange: zero-width slice %d", s);
    width = width > (int64_t)st.col[s] + st.out[s] ? width : (int64_t)st.col[s] + st.out[s];
    ++n_act;
  }
  if (y_ld < width || x_ld < in_dim)
    return fail(B200_LORA_EINVAL, "row stride smaller than row: y_ld=%lld (need %lld) x_ld=%lld (need %d)",
                (long long)y_ld, (long long)width, (long long)x_ld, in_dim);
  const int64_t count64 = (int64_t)n_act * T * r_max;
  if (count64 > (int64_t)INT32_MAX || (count64 & 3)) return fail(B200_LORA_EINVAL, "n_slices * T * r_max must be a multiple of 4 below 2^31");
  const int count = (int)count64;
  cudaStream_t st_ = static_cast<cudaStream_t>(stream);
  const bool have_buckets = sorted_idx && slot_ids && counts && offsets && n_buckets > 0;

  BgmvProblem bp;
  bp.y = y; bp.y_ld = y_ld; bp.x = x; bp.x_ld = x_ld; bp.T = T; bp.in_dim = in_dim; bp.st = st;
  bp.S = S; bp.r_max = r_max; bp.rank_per_slot = rank_per_slot; bp.scale_per_slot = scale_per_slot;
  bp.sorted_idx = sorted_idx; bp.slot_ids = slot_ids; bp.counts = counts; bp.offsets = offsets;
  bp.n_buckets = n_buckets; bp.scaling = scaling; bp.tmp_io = tmp;
  BgmvProblem shrink_p = bp, expand_p = bp;
  shrink_p.mode = 1;
  expand_p.mode = 2; expand_p.scaling = 1.0f; expand_p.scale_per_slot = nullptr;  // the scale is already in tmp
  BgmvParams shrink_plan, expand_plan;
  const bool fused_kernels = dtype == B200_LORA_BF16 && have_buckets && bgmv_plan(shrink_p, &shrink_plan, nullptr) &&
                             bgmv_plan(expand_p, &expand_plan, nullptr);
  if (fused_kernels) {
    if (int rc = bgmv_launch(shrink_plan, st_)) return rc;
  } else {
    // any dtype / shape: one CTA per token; rows without adapter are zero-filled (they are exchanged too)
    if (r_max > 2048) return fail(B200_LORA_EUNSUPPORTED, "generic kernel: r_max=%d > 2048", r_max);
    if (scale_per_slot != nullptr) return fail(B200_LORA_EUNSUPPORTED, "per-slot scales need the bf16 bucket kernels here");
    int rc;
    if (dtype == B200_LORA_BF16)
      rc = launch_generic_shrink<__nv_bfloat16, float>(tmp, x, x_ld, T, in_dim, st, S, r_max, token_to_slot, scaling, st_);
    else if (dtype == B200_LORA_F16)
      rc = launch_generic_shrink<__half, float>(tmp, x, x_ld, T, in_dim, st, S, r_max, token_to_slot, scaling, st_);
    else
      rc = launch_generic_shrink<float, float>(tmp, x, x_ld, T, in_dim, st, S, r_max, token_to_slot, scaling, st_);
    if (rc) return rc;
  }
  if (tp > 1)
    if (int rc = tp_allreduce_launch(tmp, tmp, count, peer_buffers, rank, tp, capacity, st_)) return rc;
  if (fused_kernels) return bgmv_launch(expand_plan, st_);
  if (dtype == B200_LORA_BF16) return launch_generic_expand<__nv_bfloat16, float>(y, y_ld, tmp, T, st, S, r_max, token_to_slot, 1, st_);
  if (dtype == B200_LORA_F16) return launch_generic_expand<__half, float>(y, y_ld, tmp, T, st, S, r_max, token_to_slot, 1, st_);
  return launch_generic_expand<float, float>(y, y_ld, tmp, T, st, S, r_max, token_to_slot, 1, st_);
}

// overwrite = 0: y += delta (lora_b200_add); 1: y = delta, -0.0 in rows without one (lora_b200_delta)
static int add_or_delta(void* y, int64_t y_ld, const void* x, int64_t x_ld, int32_t T, int32_t in_dim,
                        int32_t n_slices, const void* const* a_slabs, const void* const* b_slabs,
                        const int32_t* out_sizes, const int32_t* col_offsets, int32_t S, int32_t r_max,
                        const int32_t* rank_per_slot, const float* scale_per_slot,
                        const int32_t* token_to_slot, const int32_t* sorted_idx, const int32_t* slot_ids,
                        const int32_t* counts, const int32_t* offsets, int32_t n_buckets, float scaling,
                        int32_t dtype, int32_t impl, void* workspace, size_t workspace_bytes,
                        void* stream, int overwrite) {
  if (!valid_dtype(dtype)) return fail(B200_LORA_EINVAL, "unknown dtype %d", dtype);
  if (T < 0 || in_dim < 1 || S < 1 || r_max < 1)
    return fail(B200_LORA_EINVAL, "bad sizes T=%d in=%d S=%d r_max=%d", T, in_dim, S, r_max);
  if (T == 0) return B200_LORA_OK;
  if (y == nullptr || x == nullptr || token_to_slot == nullptr)
    return fail(B200_LORA_EINVAL, "null y / x / token_to_slot");
  if (out_sizes == nullptr || col_offsets == nullptr)
    return fail(B200_LORA_EINVAL, "null out_sizes / col_offsets");
  SliceTable st;
  if (int rc = fill_slices(st, n_slices, a_slabs, b_slabs, out_sizes, col_offsets, true, true)) return rc;
  int64_t width = 0;
  bool any = false;
  for (int s = 0; s < st.n; ++s) {
    width = width > (int64_t)st.col[s] + st.out[s] ? width : (int64_t)st.col[s] + st.out[s];
    any = any || st.out[s] > 0;
  }
  if (!any) return B200_LORA_OK;
  if (y_ld < width || x_ld < in_dim)
    return fail(B200_LORA_EINVAL, "row stride smaller than row: y_ld=%lld (need %lld) x_ld=%lld (need %d)",
                (long long)y_ld, (long long)width, (long long)x_ld, in_dim);
  cudaStream_t st_ = static_cast<cudaStream_t>(stream);
  const bool have_buckets = sorted_idx && slot_ids && counts && offsets && n_buckets > 0;

  BgmvProblem bp;
  bp.y = y; bp.y_ld = y_ld; bp.x = x; bp.x_ld = x_ld; bp.T = T; bp.in_dim = in_dim; bp.st = st;
  bp.S = S; bp.r_max = r_max; bp.rank_per_slot = rank_per_slot; bp.scale_per_slot = scale_per_slot;
  bp.sorted_idx = sorted_idx; bp.slot_ids = slot_ids; bp.counts = counts; bp.offsets = offsets;
  bp.n_buckets = n_buckets; bp.scaling = scaling;
  const bool is16 = dtype == B200_LORA_BF16 || dtype == B200_LORA_F16;
  bp.kind = dtype == B200_LORA_F16 ? 2 : (r_max % 32 != 0 ? 1 : 0);

  SgmvProblem sp;
  sp.y = y; sp.y_ld = y_ld; sp.x = x; sp.x_ld = x_ld; sp.T = T; sp.in_dim = in_dim; sp.S = S; sp.r_max = r_max;
  sp.st = st; sp.scale_per_slot = scale_per_slot; sp.token_to_slot = token_to_slot; sp.scaling = scaling;

  GroupedProblem gp;
  gp.y = y; gp.y_ld = y_ld; gp.x = x; gp.x_ld = x_ld; gp.T = T; gp.in_dim = in_dim; gp.S = S; gp.r_max = r_max; gp.st = st;
  gp.rank_per_slot = rank_per_slot; gp.scale_per_slot = scale_per_slot; gp.sorted_idx = sorted_idx; gp.slot_ids = slot_ids;
  gp.counts = counts; gp.offsets = offsets; gp.n_buckets = n_buckets; gp.scaling = scaling; gp.dtype = dtype;

  // Scratch of the prefill pair. The one-launch kernel uses none: AUTO takes it without, a call that asks for the prefill kernels by
  // name is refused without (which of them runs is not the caller's to know).
  int n_act = 0;
  for (int s = 0; s < st.n; ++s) n_act += st.out[s] > 0;
  const bool one_launch = prefill_cluster_add_ok(sp), auto_impl = impl == B200_LORA_IMPL_AUTO;
  const bool scratch_ok = (auto_impl && one_launch) || (workspace != nullptr && workspace_bytes >= sgmv_workspace_bytes(T, n_act, r_max));

  BgmvParams plan;
  if (overwrite) {
    // decode batches: the row-split kernel writes the delta (and the -0.0 rows) itself; everything else
    // fills y with -0.0 first and then adds as usual (-0.0 + d == d)
    const int kind = bp.kind;
    bp.kind = 0;
    bp.mode = 3;
    bp.token_to_slot = token_to_slot;
    // (Without bucket arrays, or at rank 16, which the bucket kernel cannot overwrite, a batch that is its own takes a fill and an add.)
    const bool bucket_form = have_buckets && r_max % 32 == 0;
    // (What the prefill kernels refuse is no batch of theirs, however large: one bucket launch instead of a fill and an add.)
    const bool prefill = sgmv_supported(sp, nullptr) && scratch_ok &&
                         (prefill_sized(T, st, r_max, in_dim, true, one_launch) || (!bucket_form && one_launch && ceil_div_i(T, kBgmvTok) > 74));
    const bool decode_like = !rows_for_prefill(T, n_buckets) || !prefill;
    if (dtype == B200_LORA_BF16 && have_buckets &&
        (impl == B200_LORA_IMPL_BGMV || (auto_impl && decode_like)) && bgmv_plan(bp, &plan, nullptr))
      return bgmv_launch(plan, st_);
    bp.mode = 0;
    bp.kind = kind;
    bp.token_to_slot = nullptr;
    // prefill batches: the tiles of the delta are stored instead of reduce-added
    if (dtype == B200_LORA_BF16 && (impl == B200_LORA_IMPL_SGMV || (auto_impl && !decode_like)) && sgmv_supported(sp, nullptr) &&
        prefill_overwrite_ok(st) && scratch_ok)
      return prefill_add(sp, workspace, workspace_bytes, st_, true);
    fill_neg_zero_kernel<<<(unsigned)T, 128, 0, st_>>>(y, y_ld, st, dtype == B200_LORA_F32 ? 4 : 2);
    if (int rc = check_launch("fill_neg_zero_kernel")) return rc;
  }

  bool planned = false;
  if (auto_impl) {
    // Long batches (prefill) go to the tensor-core kernels, where they have the scratch they use, decode
    // batches to the fused kernel, everything else (other dtypes, odd shapes) to the generic one.
    int parts;
    const bool bgmv_ok = planned = is16 && have_buckets && bgmv_plan(bp, &plan, nullptr);
    // The prefill kernels take the rows in token order: with bucket arrays at hand, few rows a bucket on average mean a decode-like
    // batch (slots scattered over the rows), which goes to the bucket kernel.
    const bool scattered = bgmv_ok && !rows_for_prefill(T, n_buckets);
    if (dtype == B200_LORA_BF16 && !scattered && (!bgmv_ok ? T >= kSgmvAutoMinTokens : prefill_sized(T, st, r_max, in_dim, true, one_launch)) && sgmv_supported(sp, nullptr) &&
        scratch_ok)
      impl = B200_LORA_IMPL_SGMV;
    else if (bgmv_ok && grouped_preferred(gp) && grouped_supported(gp, nullptr) && workspace != nullptr &&
             workspace_bytes >= grouped_need(gp, &parts))
      impl = B200_LORA_IMPL_GROUPED;
    else if (bgmv_ok)
      impl = B200_LORA_IMPL_BGMV;
    else
      impl = B200_LORA_IMPL_GENERIC;
  }
  switch (impl) {
    case B200_LORA_IMPL_GENERIC:
      if (r_max > 2048) return fail(B200_LORA_EUNSUPPORTED, "generic kernel: r_max=%d > 2048", r_max);
      if (dtype == B200_LORA_BF16)
        return launch_generic_add<__nv_bfloat16>(y, y_ld, x, x_ld, T, in_dim, st, S, r_max, rank_per_slot,
                                                 scale_per_slot, token_to_slot, scaling, st_);
      if (dtype == B200_LORA_F16)
        return launch_generic_add<__half>(y, y_ld, x, x_ld, T, in_dim, st, S, r_max, rank_per_slot,
                                          scale_per_slot, token_to_slot, scaling, st_);
      return launch_generic_add<float>(y, y_ld, x, x_ld, T, in_dim, st, S, r_max, rank_per_slot,
                                       scale_per_slot, token_to_slot, scaling, st_);
    case B200_LORA_IMPL_BGMV: {
      if (!is16) return fail(B200_LORA_EUNSUPPORTED, "fused decode kernel is bf16 / fp16 only");
      if (!have_buckets) return fail(B200_LORA_EINVAL, "fused decode kernel needs the bucket arrays");
      const char* why = nullptr;
      if (planned || bgmv_plan(bp, &plan, &why)) return bgmv_launch(plan, st_);
      return fail(B200_LORA_EUNSUPPORTED, "fused decode kernel: %s", why);
    }
    case B200_LORA_IMPL_SGMV:
      if (dtype != B200_LORA_BF16) return fail(B200_LORA_EUNSUPPORTED, "prefill kernels are bf16 only");
      if (!scratch_ok && sgmv_supported(sp, nullptr))
        if (int rc = sgmv_workspace_check(sp, n_act, workspace, workspace_bytes)) return rc;
      return prefill_add(sp, workspace, workspace_bytes, st_);
    case B200_LORA_IMPL_GROUPED:
      // (where the fused decode kernel takes the batch too, the delta is rounded to bf16 and added at the L2 as there)
      return grouped_add_launch(gp, workspace, workspace_bytes, dtype == B200_LORA_BF16 && r_max % 32 == 0, st_);
    default:
      return fail(B200_LORA_EUNSUPPORTED, "impl %d is not available", impl);
  }
}

int lora_b200_add(void* y, int64_t y_ld, const void* x, int64_t x_ld, int32_t T, int32_t in_dim,
                  int32_t n_slices, const void* const* a_slabs, const void* const* b_slabs,
                  const int32_t* out_sizes, const int32_t* col_offsets, int32_t S, int32_t r_max,
                  const int32_t* rank_per_slot, const float* scale_per_slot,
                  const int32_t* token_to_slot, const int32_t* sorted_idx, const int32_t* slot_ids,
                  const int32_t* counts, const int32_t* offsets, int32_t n_buckets, float scaling,
                  int32_t dtype, int32_t impl, void* workspace, size_t workspace_bytes,
                  void* stream) {
  return add_or_delta(y, y_ld, x, x_ld, T, in_dim, n_slices, a_slabs, b_slabs, out_sizes, col_offsets, S, r_max,
                      rank_per_slot, scale_per_slot, token_to_slot, sorted_idx, slot_ids, counts, offsets, n_buckets,
                      scaling, dtype, impl, workspace, workspace_bytes, stream, 0);
}

int lora_b200_delta(void* delta, int64_t delta_ld, const void* x, int64_t x_ld, int32_t T, int32_t in_dim,
                    int32_t n_slices, const void* const* a_slabs, const void* const* b_slabs,
                    const int32_t* out_sizes, const int32_t* col_offsets, int32_t S, int32_t r_max,
                    const int32_t* rank_per_slot, const float* scale_per_slot,
                    const int32_t* token_to_slot, const int32_t* sorted_idx, const int32_t* slot_ids,
                    const int32_t* counts, const int32_t* offsets, int32_t n_buckets, float scaling,
                    int32_t dtype, int32_t impl, void* workspace, size_t workspace_bytes,
                    void* stream) {
  return add_or_delta(delta, delta_ld, x, x_ld, T, in_dim, n_slices, a_slabs, b_slabs, out_sizes, col_offsets, S, r_max,
                      rank_per_slot, scale_per_slot, token_to_slot, sorted_idx, slot_ids, counts, offsets, n_buckets,
                      scaling, dtype, impl, workspace, workspace_bytes, stream, 1);
}

int lora_b200_shrink_buckets(void* out, int32_t out_dtype, const void* x, int64_t x_ld, int32_t T, int32_t in_dim,
                             int32_t n_slices, const void* const* a_slabs, int32_t S, int32_t r_max,
                             const int32_t* token_to_slot, const int32_t* sorted_idx, const int32_t* slot_ids,
                             const int32_t* counts, const int32_t* offsets, int32_t n_buckets, float scaling, int32_t dtype,
                             void* stream) {
  if (!valid_dtype(dtype) || !valid_dtype(out_dtype)) return fail(B200_LORA_EINVAL, "unknown dtype");
  if (out_dtype != dtype && out_dtype != B200_LORA_F32)
    return fail(B200_LORA_EUNSUPPORTED, "shrink output must have the input dtype or be f32");
  if (T < 0 || in_dim < 1 || S < 1 || r_max < 1) return fail(B200_LORA_EINVAL, "bad sizes");
  if (T == 0) return B200_LORA_OK;
  if (!out || !x || !token_to_slot) return fail(B200_LORA_EINVAL, "null out / x / token_to_slot");
  if (x_ld < in_dim) return fail(B200_LORA_EINVAL, "x_ld < in_dim");
  SliceTable st;
  if (int rc = fill_slices(st, n_slices, a_slabs, nullptr, nullptr, nullptr, true, false)) return rc;
  cudaStream_t st_ = static_cast<cudaStream_t>(stream);
  // With bucket arrays: the shrink half of the fused decode kernel (same sums as the per-token kernel, which reads an
  // adapter again for every row). Batches of prefill size go to the tensor-core shrink if their rows are contiguous: with
  // bucket arrays the two are launched together and look for themselves (rows_scattered).
  const bool buckets = sorted_idx && slot_ids && counts && offsets && n_buckets > 0;
  BgmvProblem bp = {};
  bp.y = nullptr; bp.y_ld = 8; bp.x = x; bp.x_ld = x_ld; bp.T = T; bp.in_dim = in_dim; bp.st = st; bp.S = S; bp.r_max = r_max;
  for (int s = 0; s < st.n; ++s) bp.st.out[s] = 8;  // (no output columns here)
  bp.rank_per_slot = nullptr; bp.scale_per_slot = nullptr;
  bp.sorted_idx = sorted_idx; bp.slot_ids = slot_ids; bp.counts = counts; bp.offsets = offsets;
  bp.n_buckets = n_buckets; bp.scaling = scaling; bp.mode = 1; bp.kind = dtype == B200_LORA_F16 ? 2 : 1;
  bp.tmp_io = out; bp.io16 = out_dtype != B200_LORA_F32; bp.zero_rows = 1; bp.token_to_slot = token_to_slot;
  BgmvParams plan;
  const bool by_bucket = buckets && (dtype == B200_LORA_BF16 || dtype == B200_LORA_F16) && aligned16(out) && bgmv_plan(bp, &plan, nullptr);
  const bool prefill = by_bucket ? T >= 32 * n_buckets && prefill_sized(T, st, r_max, in_dim, false, false) : T >= kSgmvAutoMinTokens;
  if (dtype == B200_LORA_BF16 && out_dtype == B200_LORA_BF16 && prefill) {
    // prefill-sized bf16 batches: the tensor-core shrink (rows without adapter are written as zeros, as the
    // per-token kernel does); anything it does not take falls through
    SgmvProblem sp;
    sp.y = nullptr; sp.y_ld = 0; sp.x = x; sp.x_ld = x_ld; sp.T = T; sp.in_dim = in_dim; sp.S = S; sp.r_max = r_max;
    sp.st = st; sp.scale_per_slot = nullptr; sp.token_to_slot = token_to_slot; sp.scaling = scaling;
    if (sgmv_supported(sp, nullptr, true, false) && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
      SgmvMaps sm;
      SgmvArgs sa;
      if (int rc = sgmv_prepare_tmp(sp, out, (uint64_t)st.n * T, true, false, &sm, &sa)) return rc;
      sa.zero_fill = 1;
      sa.gate = by_bucket ? 1 : 0;
      const int rc = sgmv_launch_shrink(sm, sa, st_);
      if (rc != B200_LORA_OK || !by_bucket) return rc;
      plan.gate = 1;
    }
  }
  if (by_bucket) return bgmv_launch(plan, st_);
#define B200_SHRINK(TT)                                                                              \
  (out_dtype == B200_LORA_F32 && dtype != B200_LORA_F32)                                             \
      ? launch_generic_shrink<TT, float>(out, x, x_ld, T, in_dim, st, S, r_max, token_to_slot, scaling, st_) \
      : launch_generic_shrink<TT, TT>(out, x, x_ld, T, in_dim, st, S, r_max, token_to_slot, scaling, st_)
  if (dtype == B200_LORA_BF16) return B200_SHRINK(__nv_bfloat16);
  if (dtype == B200_LORA_F16) return B200_SHRINK(__half);
  return launch_generic_shrink<float, float>(out, x, x_ld, T, in_dim, st, S, r_max, token_to_slot, scaling, st_);
#undef B200_SHRINK
}

int lora_b200_expand_buckets(void* y, int64_t y_ld, const void* tmp, int32_t tmp_dtype, int32_t T, int32_t n_slices,
                             const void* const* b_slabs, const int32_t* out_sizes, const int32_t* col_offsets, int32_t S,
                             int32_t r_max, const int32_t* token_to_slot, const int32_t* sorted_idx, const int32_t* slot_ids,
                             const int32_t* counts, const int32_t* offsets, int32_t n_buckets, int32_t add_inputs, int32_t dtype,
                             void* stream) {
  if (!valid_dtype(dtype) || !valid_dtype(tmp_dtype)) return fail(B200_LORA_EINVAL, "unknown dtype");
  if (tmp_dtype != dtype && tmp_dtype != B200_LORA_F32)
    return fail(B200_LORA_EUNSUPPORTED, "expand input must have the weight dtype or be f32");
  if (T < 0 || S < 1 || r_max < 1) return fail(B200_LORA_EINVAL, "bad sizes");
  if (T == 0) return B200_LORA_OK;
  if (!y || !tmp || !token_to_slot || !out_sizes || !col_offsets)
    return fail(B200_LORA_EINVAL, "null pointer argument");
  if (r_max > 2048) return fail(B200_LORA_EUNSUPPORTED, "r_max=%d > 2048", r_max);
  SliceTable st;
  if (int rc = fill_slices(st, n_slices, nullptr, b_slabs, out_sizes, col_offsets, false, true)) return rc;
  for (int s = 0; s < st.n; ++s)
    if (y_ld < (int64_t)st.col[s] + st.out[s]) return fail(B200_LORA_EINVAL, "y_ld smaller than slice end");
  cudaStream_t st_ = static_cast<cudaStream_t>(stream);
  // (as in the shrink: one of two launches for prefill-sized batches with bucket arrays)
  const bool buckets = sorted_idx && slot_ids && counts && offsets && n_buckets > 0;
  bool dense = true;  // no zero-width slice: tmp is indexed by slice position
  for (int s = 0; s < st.n; ++s) dense = dense && st.out[s] > 0;
  BgmvProblem bp = {};
  bp.y = y; bp.y_ld = y_ld; bp.x = nullptr; bp.x_ld = 32; bp.T = T; bp.in_dim = 32; bp.st = st; bp.S = S; bp.r_max = r_max;
  bp.rank_per_slot = nullptr; bp.scale_per_slot = nullptr;
  bp.sorted_idx = sorted_idx; bp.slot_ids = slot_ids; bp.counts = counts; bp.offsets = offsets;
  bp.n_buckets = n_buckets; bp.scaling = 1.0f; bp.mode = 2; bp.kind = dtype == B200_LORA_F16 ? 2 : 1;
  bp.tmp_io = const_cast<void*>(tmp); bp.io16 = tmp_dtype != B200_LORA_F32; bp.no_add = add_inputs ? 0 : 1; bp.token_to_slot = token_to_slot;
  BgmvParams plan;
  const bool by_bucket = buckets && (dtype == B200_LORA_BF16 || dtype == B200_LORA_F16) && dense && aligned16(tmp) && bgmv_plan(bp, &plan, nullptr);
  const bool prefill = by_bucket ? T >= 32 * n_buckets && prefill_sized(T, st, r_max, 0, true, false) : T >= kSgmvAutoMinTokens;
  if (dtype == B200_LORA_BF16 && tmp_dtype == B200_LORA_BF16 && add_inputs && prefill) {
    // prefill-sized bf16 batches: the tensor-core expand (reduce-add tile kernel when the slices tile the
    // columns they cover in 64-column units, run-based kernel otherwise)
    int first = -1;
    for (int s = 0; s < st.n; ++s)
      if (st.out[s] > 0 && (first < 0 || st.col[s] < first)) first = st.col[s];
    if (dense && first >= 0 && first % 8 == 0) {
      SgmvProblem sp;
      sp.y = static_cast<char*>(y) + (size_t)first * 2; sp.y_ld = y_ld; sp.x = nullptr; sp.x_ld = 0; sp.T = T; sp.in_dim = 0;
      sp.S = S; sp.r_max = r_max; sp.st = st; sp.scale_per_slot = nullptr; sp.token_to_slot = token_to_slot; sp.scaling = 1.0f;
      for (int s = 0; s < st.n; ++s) sp.st.col[s] -= first;
      if (sgmv_supported(sp, nullptr, false, true) && (reinterpret_cast<uintptr_t>(tmp) & 15u) == 0) {
        SgmvMaps sm;
        SgmvArgs sa;
        if (int rc = sgmv_prepare_tmp(sp, const_cast<void*>(tmp), (uint64_t)st.n * T, false, true, &sm, &sa)) return rc;
        sa.gate = by_bucket ? 1 : 0;
        int rc;
        if (tc_expand_fast_path_ok(sa)) {
          int n_total = 0;
          for (int s = 0; s < sa.n; ++s) n_total = std::max(n_total, sa.col[s] + sa.out[s]);
          GemmMaps gm;
          GemmArgs ga;
          if (int rc2 = tc_tile_prepare(sm, sa, nullptr, 0, n_total, nullptr, true, true, &gm, &ga, false, false)) return rc2;
          rc = tc_tile_launch(gm, ga, st_);
        } else {
          rc = sgmv_launch_expand(sm, sa, st_);
        }
        if (rc != B200_LORA_OK || !by_bucket) return rc;
        plan.gate = 1;
      }
    }
  }
  if (by_bucket) return bgmv_launch(plan, st_);
#define B200_EXPAND(TT)                                                                               \
  (tmp_dtype == B200_LORA_F32 && dtype != B200_LORA_F32)                                              \
      ? launch_generic_expand<TT, float>(y, y_ld, tmp, T, st, S, r_max, token_to_slot, add_inputs, st_) \
      : launch_generic_expand<TT, TT>(y, y_ld, tmp, T, st, S, r_max, token_to_slot, add_inputs, st_)
  if (dtype == B200_LORA_BF16) return B200_EXPAND(__nv_bfloat16);
  if (dtype == B200_LORA_F16) return B200_EXPAND(__half);
  return launch_generic_expand<float, float>(y, y_ld, tmp, T, st, S, r_max, token_to_slot, add_inputs, st_);
#undef B200_EXPAND
}

int lora_b200_shrink(void* out, int32_t out_dtype, const void* x, int64_t x_ld, int32_t T, int32_t in_dim, int32_t n_slices,
                     const void* const* a_slabs, int32_t S, int32_t r_max, const int32_t* token_to_slot, float scaling,
                     int32_t dtype, void* stream) {
  return lora_b200_shrink_buckets(out, out_dtype, x, x_ld, T, in_dim, n_slices, a_slabs, S, r_max, token_to_slot, nullptr, nullptr,
                                  nullptr, nullptr, 0, scaling, dtype, stream);
}

int lora_b200_expand(void* y, int64_t y_ld, const void* tmp, int32_t tmp_dtype, int32_t T, int32_t n_slices,
                     const void* const* b_slabs, const int32_t* out_sizes, const int32_t* col_offsets, int32_t S, int32_t r_max,
                     const int32_t* token_to_slot, int32_t add_inputs, int32_t dtype, void* stream) {
  return lora_b200_expand_buckets(y, y_ld, tmp, tmp_dtype, T, n_slices, b_slabs, out_sizes, col_offsets, S, r_max, token_to_slot,
                                  nullptr, nullptr, nullptr, nullptr, 0, add_inputs, dtype, stream);
}

}  // extern "C"

// ------------------------------------------------------------------------------------------
// Prefill entry point for callers that cannot allocate device memory.
//
// The tensor-core prefill kernels keep the rank-r shrink result in scratch memory that
// lora_b200_add expects from its caller. Some callers have nowhere to get that from: code
// running inside an already captured or replaying CUDA graph, plug-ins that are handed
// input / output buffers by a host framework and are forbidden to call the allocator, and
// latency-critical loops that must not touch cudaMalloc (it synchronises the device). For them
// the same kernels run on a fixed scratch array that is part of the library image (the one-launch kernel uses
// none of it; what is refused depends on the sizes alone).
//
// The array is one per GPU (every device that loads this library carries these bytes until
// the process exits) and is shared by every call on that GPU: it still holds the previous
// call's intermediate, and two calls that overlap on the GPU (different streams) would
// overwrite each other's intermediate. Nothing in it has to start at zero: each row that a
// call reads and uses was written by that same call's shrink kernel, rows of tokens without
// an adapter are read but masked out.
namespace {

constexpr size_t kStaticScratchBytes = 8u << 20;  // 8 MiB: e.g. 3 slices x 8192 tokens x rank 64 in bf16 = 3 MiB
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

constexpr int kMaxDevices = 64;
void* g_static_scratch_addr[kMaxDevices] = {};

// Device address of the scratch array on the current device. In host code the array's name is
// only a handle of the runtime, not a device pointer, so the address is asked for once per
// device (with that device current) and remembered.
int static_scratch_for_current_device(void** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(B200_LORA_ECUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices) return fail(B200_LORA_EUNSUPPORTED, "device ordinal %d not supported", dev);
  if (g_static_scratch_addr[dev] == nullptr) {
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_static_scratch);
    if (e != cudaSuccess || ptr == nullptr)
      return fail(B200_LORA_ECUDA, "cudaGetSymbolAddress(static scratch): %s", cudaGetErrorString(e));
    g_static_scratch_addr[dev] = ptr;
  }
  *out = g_static_scratch_addr[dev];
  return B200_LORA_OK;
}

}  // namespace

extern "C" {

size_t lora_b200_static_scratch_bytes(void) { return kStaticScratchBytes; }

int lora_b200_add_prefill_noalloc(void* y, int64_t y_ld, const void* x, int64_t x_ld, int32_t T, int32_t in_dim,
                                  int32_t n_slices, const void* const* a_slabs, const void* const* b_slabs,
                                  const int32_t* out_sizes, const int32_t* col_offsets, int32_t S, int32_t r_max,
                                  const float* scale_per_slot, const int32_t* token_to_slot, float scaling,
                                  void* stream) {
  if (T < 0 || in_dim < 1 || S < 1 || r_max < 1)
    return fail(B200_LORA_EINVAL, "bad sizes T=%d in=%d S=%d r_max=%d", T, in_dim, S, r_max);
  if (T == 0) return B200_LORA_OK;
  if (y == nullptr || x == nullptr || token_to_slot == nullptr || out_sizes == nullptr || col_offsets == nullptr)
    return fail(B200_LORA_EINVAL, "null pointer argument");
  SliceTable st;
  if (int rc = fill_slices(st, n_slices, a_slabs, b_slabs, out_sizes, col_offsets, true, true)) return rc;
  int n_act = 0;
  int64_t width = 0;
  for (int s = 0; s < st.n; ++s) {
    n_act += st.out[s] > 0;
    width = width > (int64_t)st.col[s] + st.out[s] ? width : (int64_t)st.col[s] + st.out[s];
  }
  if (n_act == 0) return B200_LORA_OK;
  if (y_ld < width || x_ld < in_dim) return fail(B200_LORA_EINVAL, "row stride smaller than row");
  const size_t need = sgmv_workspace_bytes(T, n_act, r_max);
  if (need > kStaticScratchBytes)
    return fail(B200_LORA_EWORKSPACE,
                "batch needs %zu bytes of scratch (slices %d x tokens %d x rank %d, bf16) but the built-in scratch "
                "holds %zu; use lora_b200_add with caller-provided scratch",
                need, n_act, T, r_max, kStaticScratchBytes);
  SgmvProblem sp;
  sp.y = y; sp.y_ld = y_ld; sp.x = x; sp.x_ld = x_ld; sp.T = T; sp.in_dim = in_dim; sp.S = S; sp.r_max = r_max;
  sp.st = st; sp.scale_per_slot = scale_per_slot; sp.token_to_slot = token_to_slot; sp.scaling = scaling;
  void* scratch = nullptr;
  if (int rc = static_scratch_for_current_device(&scratch)) return rc;
  return prefill_add(sp, scratch, kStaticScratchBytes, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
