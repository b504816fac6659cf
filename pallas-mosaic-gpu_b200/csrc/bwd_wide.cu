// Launcher of the 128-row-per-step fused backward (bwd_wide_kernel.cuh).
#include "bwd_launch.cuh"
#include "bwd_wide_kernel.cuh"
#include "dispatch.h"

namespace splash {

template <int D, bool BF16>
static int launch_bwd_wide_typed(const SplashParams& p, cudaStream_t stream) {
  using L = WideLayout<D>;
  const bool seg = p.seg_q != nullptr;
  const CUtensorMapDataType dt = tmap_dtype(p.dtype);
  const uint64_t q_rows = static_cast<uint64_t>(p.batch) * p.heads * p.q_len;
  const uint64_t kv_rows = static_cast<uint64_t>(p.batch) * p.kv_heads * p.kv_len;
  CUtensorMap tm_q, tm_k, tm_v, tm_do, tm_dk, tm_dv, tm_dqacc;
  int rc;
  if ((rc = make_tmap_2d(&tm_q, p.q, dt, 2, q_rows, D, 128, 64, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  if ((rc = make_tmap_2d(&tm_do, p.d_out, dt, 2, q_rows, D, 128, 64, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  if ((rc = make_tmap_2d(&tm_k, p.k, dt, 2, kv_rows, D, 128, 64, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  if ((rc = make_tmap_2d(&tm_v, p.v, dt, 2, kv_rows, D, 128, 64, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  if ((rc = make_tmap_2d(&tm_dk, p.dk, dt, 2, kv_rows, D, 128, 64, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  if ((rc = make_tmap_2d(&tm_dv, p.dv, dt, 2, kv_rows, D, 128, 64, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  // f32 accumulator, tiles of 32 x 32: [batch * heads * head_dim, q_len], at head_dim 64
  // [batch * heads * q_len, head_dim].
  const uint64_t acc_rows = L::kRoomy ? q_rows : static_cast<uint64_t>(p.batch) * p.heads * D;
  if ((rc = make_tmap_2d(&tm_dqacc, p.dq_acc, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, acc_rows, L::kRoomy ? D : p.q_len, 32, 32,
                         CU_TENSOR_MAP_SWIZZLE_128B)))
    return rc;
  if (reinterpret_cast<uintptr_t>(p.partial_blocks) & 15)
    return fail(SPLASH_INVALID_ARGUMENT, "partial_blocks not 16-byte aligned");
  BwdArgs a;
  fill_bwd_args(a, p, p.partial_blocks != nullptr, seg);
  a.stages = L::kSlots;
  a.aux_lse = fold_operand_lse(p);  // filled by the caller
  a.aux_delta = fold_operand_delta(p);
  // Segment skipping when what is left of the CTA's block steps fits the room set aside for it.
  const bool skipping = seg && p.seg_ranges != nullptr && L::steps_fit(p.mask_heads > 1 ? p.heads / p.kv_heads : 1, p.max_steps);
  a.seg_q_ranges = skipping ? seg_q_ranges(p) : nullptr;
  a.seg_kv_ranges = skipping ? seg_kv_ranges(p) : nullptr;
  const bool plain = p.soft_cap == 0.f && !seg;
  auto kernel = plain ? splash_bwd_wide_kernel<D, true, BF16> : splash_bwd_wide_kernel<D, false, BF16>;
  if ((rc = opt_in_smem(kernel, L::kSmemBytes))) return rc;
  const unsigned grid = static_cast<unsigned>(a.kv_blocks) * p.kv_heads * p.batch;
  kernel<<<grid, L::kThreads, L::kSmemBytes, stream>>>(tm_q, tm_k, tm_v, tm_do, tm_dk, tm_dv, tm_dqacc, a);
  SPLASH_CUDA_CHECK(cudaGetLastError());
  return SPLASH_OK;
}

int launch_bwd_wide(const SplashParams& p, cudaStream_t stream) {
  if (p.head_dim != p.head_dim_v || (p.head_dim != 64 && p.head_dim != 128))
    return fail(SPLASH_UNSUPPORTED, "the fused backward needs head_dim == head_dim_v in {64, 128}");
  if (p.head_dim == 64) {
    if (p.dtype == SPLASH_DTYPE_BF16) return launch_bwd_wide_typed<64, true>(p, stream);
    return launch_bwd_wide_typed<64, false>(p, stream);
  }
  if (p.dtype == SPLASH_DTYPE_BF16) return launch_bwd_wide_typed<128, true>(p, stream);
  return launch_bwd_wide_typed<128, false>(p, stream);
}

}  // namespace splash
