// Host launcher for the forward kernel template: builds the TMA tensor maps for one
// call and enqueues the grid.  Included by the translation units that instantiate
// the kernel for a given (head_dim, head_dim_v, block_kv, tiles) combination.
#pragma once

#include "dispatch.h"
#include "fwd_kernel.cuh"
#include "host_common.cuh"

namespace splash {

template <int D, int DV, int BKV, int NT, int AW, bool PLAIN, bool SPLIT, bool BF16>
int launch_fwd_plain(const SplashParams& p, int splits, void* workspace, cudaStream_t stream) {
  using L = FwdLayout<D, DV, BKV, NT, AW>;
  const bool dense = p.partial_blocks != nullptr;
  const bool seg = p.seg_q != nullptr;
  // The list of steps that survive segment skipping needs max_steps 16-bit entries; without room
  // for it (or with more than 2^15 steps) every scheduled block is computed.
  bool skipping = seg && p.seg_ranges != nullptr && p.max_steps < (1 << 15);
  if (skipping && L::smem_bytes(p.num_stages, dense, seg, p.max_steps) > kMaxDynamicSmem) skipping = false;
  const size_t smem = L::smem_bytes(p.num_stages, dense, seg, skipping ? p.max_steps : 0);
  if (smem > kMaxDynamicSmem) {
    char d[96];
    snprintf(d, sizeof d, "%zu > %zu bytes; reduce num_stages or block_kv", smem, kMaxDynamicSmem);
    return fail(SPLASH_BUDGET_EXCEEDED, "Shared memory budget exceeded", d);
  }
  if (!L::kOStageInQ && p.num_stages * BKV < 128)
    return fail(SPLASH_BUDGET_EXCEEDED, "Shared memory budget exceeded", "output staging needs num_stages * block_kv >= 128");

  const CUtensorMapDataType dt = tmap_dtype(p.dtype);
  const uint64_t q_rows = static_cast<uint64_t>(p.batch) * p.heads * p.q_len;
  const uint64_t kv_rows = static_cast<uint64_t>(p.batch) * p.kv_heads * p.kv_len;
  CUtensorMap tm_q, tm_k, tm_v, tm_o;
  int rc;
  if ((rc = make_tmap_2d(&tm_q, p.q, dt, 2, q_rows, D, 128, 64, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  if ((rc = make_tmap_2d(&tm_k, p.k, dt, 2, kv_rows, D, BKV, 64, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  if ((rc = make_tmap_2d(&tm_v, p.v, dt, 2, kv_rows, DV, BKV, 64, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  if ((rc = make_tmap_2d(&tm_o, p.out, dt, 2, q_rows, DV, 128, 64, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  if (dense && (reinterpret_cast<uintptr_t>(p.partial_blocks) & 15))
    return fail(SPLASH_INVALID_ARGUMENT, "partial_blocks not 16-byte aligned");

  FwdArgs a;
  a.num_steps = p.num_steps;
  a.block_order = p.block_order;
  a.block_list = p.block_list;
  a.block_kind = p.block_kind;
  a.mask_block = p.mask_block;
  a.mask_desc = p.mask_desc;
  a.seg_q = p.seg_q;
  a.seg_kv = p.seg_kv;
  a.partial_blocks = reinterpret_cast<const uint8_t*>(p.partial_blocks);
  a.seg_q_ranges = skipping ? seg_q_ranges(p) : nullptr;
  a.seg_kv_ranges = skipping ? seg_kv_ranges(p) : nullptr;
  a.out = p.out;
  a.lse_out = p.lse_out;
  a.status = p.status;
  a.batch = p.batch;
  a.heads = p.heads;
  a.kv_heads = p.kv_heads;
  a.q_len = p.q_len;
  a.kv_len = p.kv_len;
  a.mask_heads = p.mask_heads;
  a.max_steps = p.max_steps;
  a.q_blocks = p.q_len / (128 * NT);
  a.stages = p.num_stages;
  a.has_dense = dense;
  a.has_seg = seg;
  a.head_group = 8;
  a.mask_value = p.mask_value;
  a.soft_cap = p.soft_cap;
  a.splits = splits;
  a.part_o = static_cast<float*>(workspace);
  a.part_ml = splits > 1 ? reinterpret_cast<float2*>(a.part_o + static_cast<size_t>(splits) * q_rows * DV) : nullptr;

  auto kernel = splash_fwd_kernel<D, DV, BKV, NT, AW, PLAIN, SPLIT, BF16>;
  if ((rc = opt_in_smem(kernel, smem))) return rc;
  const unsigned grid = static_cast<unsigned>(a.q_blocks) * p.heads * p.batch * splits;
  kernel<<<grid, L::kThreads, smem, stream>>>(tm_q, tm_k, tm_v, tm_o, a);
  SPLASH_CUDA_CHECK(cudaGetLastError());
  return SPLASH_OK;
}

// The kernel without its soft-cap, segment and streamed-mask code when the call uses none.
template <int D, int DV, int BKV, int NT, int AW, bool SPLIT, bool BF16>
int launch_fwd_form(const SplashParams& p, int splits, void* workspace, cudaStream_t stream) {
  const bool plain = p.soft_cap == 0.f && p.seg_q == nullptr && p.partial_blocks == nullptr;
  return plain ? launch_fwd_plain<D, DV, BKV, NT, AW, true, SPLIT, BF16>(p, splits, workspace, stream)
               : launch_fwd_plain<D, DV, BKV, NT, AW, false, SPLIT, BF16>(p, splits, workspace, stream);
}

template <int D, int DV, int BKV, int NT, int AW, bool BF16>
int launch_fwd_typed(const SplashParams& p, int splits, void* workspace, cudaStream_t stream) {
  return splits > 1 ? launch_fwd_form<D, DV, BKV, NT, AW, true, BF16>(p, splits, workspace, stream)
                    : launch_fwd_form<D, DV, BKV, NT, AW, false, BF16>(p, splits, workspace, stream);
}

// Softmax warpgroups per q tile of the one-tile kernel.  Two that alternate over the KV steps where
// tensor memory has room for P beside S: 128-wide blocks always (causal, 16 heads, seq 8192, D = 128:
// 449 us against 532 with one group), 64-wide blocks where the softmax bounds the step (two CTAs per SM,
// D = 64, 64 heads, seq 8192 causal: 742 against 786 us; packed documents 734 against 750) or a step is
// long enough for its latency to show (one CTA per SM, D = 256, 64 heads, block-sparse seq 8192: 1092
// against 1145 us; D = 192: 348 against 356).  At DV = 128 with 64-wide blocks P lies over S in the 256
// columns each of two CTAs has, and one group is better (causal seq 8192: 457 against 490 us).
template <int DV, int BKV, int NT>
constexpr int fwd_softmax_groups() {
  if (NT == 2) return 1;
  if (BKV == 64) return (DV == 64 || DV > 128) ? 2 : 1;
  return 3 * BKV + DV <= 512 ? 2 : 1;
}

// Rows of few steps, where two groups hardly take turns and their hand-over and larger start only cost: one group.
// Up to head_dim 128 by the longest row (one group against two, bf16, seq 8192, D = 64, 64 heads: window 64, 3 steps,
// 101.7 against 108.0 us, window 256, 6 steps, 136.5 / 137.5, window 512, 10 steps, 178.4 / 171.8; batch 32, 16 heads, seq
// 128 13.1 / 14.7; batch 16, seq 512 33.8 / 34.4).  Above it, where one CTA has the SM, where a row spans all keys, as in
// batches of short sequences (batch 16, 16 heads, seq 512, D = 256 full 88.5 / 96.4, causal 75.6 / 79.6; batch 8, seq 1024
// 142.5 / 150.6, 102.0 / 108.8; D = 192 112.4 / 115.4, 85.6 / 87.4); windows are even there (+-1.5 %) and keep two.
template <int D, int DV>
bool fwd_short_rows(const SplashParams& p) {
  if (D <= 128 && DV <= 128) return p.max_steps <= 8;
  return p.max_steps <= 16 && p.max_steps * p.block_kv >= p.kv_len;
}

template <int D, int DV, int BKV, int NT>
int launch_fwd(const SplashParams& p, int splits, void* workspace, cudaStream_t stream) {
  const bool bf16 = p.dtype == SPLASH_DTYPE_BF16;
  constexpr int AW = fwd_softmax_groups<DV, BKV, NT>();
  if constexpr (NT == 1 && BKV == 64 && AW == 2) {
    if (splits == 1 && fwd_short_rows<D, DV>(p))
      return bf16 ? launch_fwd_form<D, DV, BKV, NT, 1, false, true>(p, 1, nullptr, stream)
                  : launch_fwd_form<D, DV, BKV, NT, 1, false, false>(p, 1, nullptr, stream);
  }
  if (bf16) return launch_fwd_typed<D, DV, BKV, NT, AW, true>(p, splits, workspace, stream);
  return launch_fwd_typed<D, DV, BKV, NT, AW, false>(p, splits, workspace, stream);
}

}  // namespace splash
