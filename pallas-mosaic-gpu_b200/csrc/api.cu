// extern "C" entry points of libsplash_sm100.so: argument validation, dispatch to
// the compiled kernel configuration, status helpers.
#include "dispatch.h"
#include "fwd_launch.cuh"
#include "host_common.cuh"

namespace splash {

constexpr int kBwdStagesMax = 4;

static int check_common(const SplashParams* p, bool backward) {
  if (!p) return fail(SPLASH_INVALID_ARGUMENT, "params is null");
  if (!p->q || !p->k || !p->v || !p->status) return fail(SPLASH_INVALID_ARGUMENT, "q, k, v and status must be non-null");
  if (!p->num_steps || !p->block_order || !p->block_list || !p->block_kind)
    return fail(SPLASH_INVALID_ARGUMENT, "schedule arrays must be non-null");
  if (p->batch <= 0 || p->heads <= 0 || p->kv_heads <= 0 || p->q_len <= 0 || p->kv_len <= 0)
    return fail(SPLASH_INVALID_ARGUMENT, "sizes must be positive");
  if (p->heads % p->kv_heads) return fail(SPLASH_INVALID_ARGUMENT, "heads not a multiple of kv_heads");
  if (p->dtype != SPLASH_DTYPE_BF16 && p->dtype != SPLASH_DTYPE_F16) return fail(SPLASH_UNSUPPORTED, "Only bf16/f16 are supported");
  if (p->head_dim % 64 || p->head_dim_v % 64 || p->head_dim > 256 || p->head_dim_v > 256 || p->head_dim <= 0 ||
      p->head_dim_v <= 0)
    return fail(SPLASH_UNSUPPORTED, "head dims must be multiples of 64 and <= 256");
  if (p->mask_heads != 1 && p->mask_heads != p->heads) return fail(SPLASH_INVALID_ARGUMENT, "mask_heads must be 1 or heads");
  if (p->max_steps < 1) return fail(SPLASH_INVALID_ARGUMENT, "max_steps must be >= 1");
  if ((p->seg_q == nullptr) != (p->seg_kv == nullptr)) return fail(SPLASH_INVALID_ARGUMENT, "seg_q and seg_kv go together");
  if (p->partial_blocks && (!p->mask_block || p->num_partial_blocks <= 0))
    return fail(SPLASH_INVALID_ARGUMENT, "dense partial blocks need mask_block ids");
  if (p->partial_blocks && p->mask_desc) return fail(SPLASH_INVALID_ARGUMENT, "give dense partial blocks or a band descriptor, not both");
  if (static_cast<int64_t>(p->batch) * p->heads * p->q_len >= (1ll << 31) ||
      static_cast<int64_t>(p->batch) * p->kv_heads * p->kv_len >= (1ll << 31))
    return fail(SPLASH_INVALID_ARGUMENT, "batch * heads * length must fit in 31 bits");
  if (backward && (!p->d_out || !p->lse || !p->delta)) return fail(SPLASH_INVALID_ARGUMENT, "backward needs d_out, lse and delta");
  return SPLASH_OK;
}

static int check_fwd(const SplashParams* p, int tiles) {
  if (int rc = check_common(p, false)) return rc;
  if (!p->out) return fail(SPLASH_INVALID_ARGUMENT, "out is null");
  if (p->block_q != 128 * tiles) return fail(SPLASH_INVALID_ARGUMENT, "block_q does not match this entry point");
  if (p->block_kv != 64 && p->block_kv != 128) return fail(SPLASH_INVALID_ARGUMENT, "block_kv must be 64 or 128");
  if (p->num_stages < 2 || p->num_stages > 8) return fail(SPLASH_INVALID_ARGUMENT, "num_stages must be in [2, 8]");
  if (p->q_len % p->block_q || p->kv_len % p->block_kv)
    return fail(SPLASH_INVALID_ARGUMENT, "Sequence lengths must be multiples of the block sizes");
  return SPLASH_OK;
}

#define SPLASH_FWD_CASE(D_, DV_, NT_)                                                               \
  if (p->head_dim == D_ && p->head_dim_v == DV_) {                                                  \
    return p->block_kv == 64 ? launch_fwd<D_, DV_, 64, NT_>(*p, splits, ws, st)                      \
                             : launch_fwd<D_, DV_, 128, NT_>(*p, splits, ws, st);                    \
  }

}  // namespace splash

using namespace splash;

extern "C" int64_t splash_seg_ranges_bytes(const SplashParams* p) {
  if (!p || !p->seg_q || p->q_len % 64 || p->kv_len % 64) return 0;
  return static_cast<int64_t>(p->batch) * (p->q_len / 64 + p->kv_len / 64) * 8;
}

static int fwd128(const SplashParams* p, int splits, void* ws, cudaStream_t st) {
  if (int rc = check_fwd(p, 1)) return rc;
  if (int rc = launch_seg_ranges(*p, st)) return rc;
  SPLASH_FWD_CASE(64, 64, 1)
  SPLASH_FWD_CASE(64, 128, 1)
  SPLASH_FWD_CASE(128, 128, 1)
  SPLASH_FWD_CASE(128, 64, 1)
  SPLASH_FWD_CASE(192, 192, 1)
  SPLASH_FWD_CASE(256, 256, 1)
  return fail(SPLASH_UNSUPPORTED, "this (head_dim, head_dim_v) pair is not compiled for the 128-row forward");
}

static int fwd256(const SplashParams* p, int splits, void* ws, cudaStream_t st) {
  if (int rc = check_fwd(p, 2)) return rc;
  if (int rc = launch_seg_ranges(*p, st)) return rc;
  if (p->head_dim != p->head_dim_v) return fail(SPLASH_UNSUPPORTED, "ping-pong kernel needs head_dim == head_dim_v");
  SPLASH_FWD_CASE(64, 64, 2)
  SPLASH_FWD_CASE(128, 128, 2)
  return fail(SPLASH_UNSUPPORTED, "ping-pong kernel supports head_dim 64/128");
}

extern "C" int splash_fwd128(const SplashParams* p, void* stream) {
  return fwd128(p, 1, nullptr, static_cast<cudaStream_t>(stream));
}

extern "C" int splash_fwd256(const SplashParams* p, void* stream) {
  return fwd256(p, 1, nullptr, static_cast<cudaStream_t>(stream));
}

// Whether two CTAs of the one-tile kernel share an SM: built for it at 64-wide blocks and head dims up to 128, and
// their shared memory fits (two stages at head_dim 128, five at 64).
template <int D, int DV>
static bool fwd_two_fit(const SplashParams& p) {
  using L = FwdLayout<D, DV, 64, 1, fwd_softmax_groups<DV, 64, 1>()>;
  const int list_steps = p.seg_q && p.seg_ranges ? p.max_steps : 0;
  const size_t smem = L::smem_bytes(p.num_stages, p.partial_blocks != nullptr, p.seg_q != nullptr, list_steps);
  return L::kCtasPerSm == 2 && 2 * (smem + kSmemPerCtaReserved) <= kSmemPerSm;
}

static bool fwd_two_per_sm(const SplashParams& p) {
  if (p.block_q != 128 || p.block_kv != 64) return false;
  if (p.head_dim == 64 && p.head_dim_v == 64) return fwd_two_fit<64, 64>(p);
  if (p.head_dim == 64 && p.head_dim_v == 128) return fwd_two_fit<64, 128>(p);
  if (p.head_dim == 128 && p.head_dim_v == 64) return fwd_two_fit<128, 64>(p);
  return p.head_dim == 128 && p.head_dim_v == 128 && fwd_two_fit<128, 128>(p);
}

// CTAs per q tile that fill the GPU once.  A grid of one CTA per tile leaves SMs idle when tiles are few
// (a chunk of queries against a long cache, small batches), and the heaviest tile then sets the time.
// Shares of fewer than 512 keys are not made, and at least 2048 keys have to come off the longest tile:
// the combining pass and its launch cost what about that many do.  Scheduled steps count, not those that segment ids
// leave (1 head, 4096 tokens, D = 128, GPU time: documents of 256-4096 tokens 66.9 -> 21.5 us, of 64-256 13.7 -> 15.5).
static int fwd_splits(const SplashParams* p) {
  if (!p || p->block_q <= 0 || p->q_len <= 0 || p->batch <= 0 || p->heads <= 0) return 1;
  const int64_t keys = static_cast<int64_t>(p->max_steps) * p->block_kv;
  if (keys <= 2048) return 1;  // (short calls, whose host time counts, ask no further)
  const int64_t tiles = static_cast<int64_t>(p->q_len / p->block_q) * p->heads * p->batch;
  if (tiles <= 0) return 1;
  const int64_t slots = static_cast<int64_t>(sm_count()) * (fwd_two_per_sm(*p) ? 2 : 1);
  int64_t splits = slots / tiles;
  if (splits > keys / 512) splits = keys / 512;
  if (splits > 32) splits = 32;
  if (splits < 2 || keys - keys / splits < 2048) return 1;
  return static_cast<int>(splits);
}

extern "C" int64_t splash_fwd_split_bytes(const SplashParams* p) {
  const int splits = fwd_splits(p);
  if (splits < 2) return 0;
  return splits * q_row_count(*p) * (static_cast<int64_t>(p->head_dim_v) * 4 + 8);
}

extern "C" int splash_fwd_split(const SplashParams* p, void* workspace, int64_t bytes, void* stream) {
  const int splits = fwd_splits(p);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool two_tiles = p && p->block_q == 256;
  if (splits < 2) return two_tiles ? fwd256(p, 1, nullptr, st) : fwd128(p, 1, nullptr, st);
  if (!workspace || bytes < splash_fwd_split_bytes(p) || (reinterpret_cast<uintptr_t>(workspace) & 15))
    return fail(SPLASH_INVALID_ARGUMENT, "the workspace of a split forward is null, too small or not 16-byte aligned");
  if (int rc = two_tiles ? fwd256(p, splits, workspace, st) : fwd128(p, splits, workspace, st)) return rc;
  return launch_fwd_combine(*p, splits, workspace, st);
}

static int check_bwd(const SplashParams* p) {
  if (int rc = check_common(p, true)) return rc;
  if (p->block_q != 128 || p->block_kv != 128) return fail(SPLASH_INVALID_ARGUMENT, "the backward schedule is 128x128");
  if (p->num_stages < 1 || p->num_stages > kBwdStagesMax) return fail(SPLASH_INVALID_ARGUMENT, "num_stages_bwd must be in [1, 4]");
  if (p->q_len % 128 || p->kv_len % 128) return fail(SPLASH_INVALID_ARGUMENT, "Sequence lengths must be multiples of 128");
  if (p->sub_block != 0 && p->sub_block != 64 && p->sub_block != 128)
    return fail(SPLASH_INVALID_ARGUMENT, "sub_block must be 0, 64 or 128");
  if ((p->head_dim != 64 && p->head_dim != 128) || (p->head_dim_v != 64 && p->head_dim_v != 128))
    return fail(SPLASH_UNSUPPORTED, "the backward pass supports head dims 64 and 128");
  return SPLASH_OK;
}

static int check_bwd_fused(const SplashParams* p) {
  if (int rc = check_bwd(p)) return rc;
  if (p->head_dim != p->head_dim_v) return fail(SPLASH_UNSUPPORTED, "the fused backward needs head_dim == head_dim_v");
  return SPLASH_OK;
}

extern "C" int splash_bwd_delta(const void* o, const void* d_out, float* delta, int64_t rows, int32_t head_dim_v,
                                int32_t dtype, void* stream) {
  return launch_delta(o, d_out, delta, rows, head_dim_v, dtype, static_cast<cudaStream_t>(stream));
}

extern "C" int splash_bwd_dq(const SplashParams* p, void* stream) {
  if (int rc = check_bwd(p)) return rc;
  if (!p->dq) return fail(SPLASH_INVALID_ARGUMENT, "dq is null");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (int rc = launch_seg_ranges(*p, st)) return rc;
  // The requested sub-block is a preference: 128 keys per step when it fits in shared
  // memory, else 64.
  const bool want128 = p->sub_block != 64;
#define SPLASH_DQ_CASE(D_, DV_)                                                                                  \
  if (p->head_dim == D_ && p->head_dim_v == DV_) {                                                               \
    if (want128 && bwd_row_smem<D_, DV_, 128>(*p) <= kMaxDynamicSmem) return launch_bwd_row<D_, DV_, 128>(*p, st); \
    return launch_bwd_row<D_, DV_, 64>(*p, st);                                                                  \
  }
  SPLASH_DQ_CASE(64, 64)
  SPLASH_DQ_CASE(128, 128)
  SPLASH_DQ_CASE(128, 64)
  SPLASH_DQ_CASE(64, 128)
#undef SPLASH_DQ_CASE
  return fail(SPLASH_UNSUPPORTED, "this (head_dim, head_dim_v) pair is not compiled for the dQ kernel");
}

extern "C" int splash_bwd_dkv(const SplashParams* p, void* stream) {
  if (int rc = check_bwd(p)) return rc;
  if (!p->dk || !p->dv) return fail(SPLASH_INVALID_ARGUMENT, "dk / dv is null");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (int rc = launch_seg_ranges(*p, st)) return rc;
  // The kernel works in steps of 64 q rows with double-buffered scores; `sub_block`
  // is accepted for compatibility and does not change the tiling.
  if (p->head_dim == 64) return p->head_dim_v == 64 ? launch_bwd_col<64, 64>(*p, st) : launch_bwd_col<64, 128>(*p, st);
  return p->head_dim_v == 128 ? launch_bwd_col<128, 128>(*p, st) : launch_bwd_col<128, 64>(*p, st);
}

// The f32 dQ accumulator alone.
static int64_t dq_acc_bytes(const SplashParams* p) {
  return static_cast<int64_t>(p->batch) * p->heads * p->q_len * p->head_dim * 4;
}

extern "C" int64_t splash_bwd_fused_workspace_bytes(const SplashParams* p) {
  if (!p) return 0;
  // Accumulator; at head_dim 64 also 32 bytes per q row for the folded lse / delta operands.
  return dq_acc_bytes(p) + fold_operand_bytes(*p);
}

extern "C" int splash_bwd_fused(const SplashParams* p, void* stream) {
  if (int rc = check_bwd_fused(p)) return rc;
  if (!p->dq || !p->dk || !p->dv || !p->dq_acc) return fail(SPLASH_INVALID_ARGUMENT, "dq, dk, dv and dq_acc must be non-null");

  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (int rc = launch_seg_ranges(*p, st)) return rc;
  if (p->out) {
    // One pass streams O and dO for delta, clears the accumulator on the way and (head_dim 64) writes
    // the folded operands.
    if (int rc = launch_delta(p->out, p->d_out, p->delta, q_row_count(*p), p->head_dim_v, p->dtype, st, p->dq_acc,
                              p->head_dim, p->lse, fold_operand_lse(*p), fold_operand_delta(*p), p->mask_value))
      return rc;
  } else {
    SPLASH_CUDA_CHECK(cudaMemsetAsync(p->dq_acc, 0, static_cast<size_t>(dq_acc_bytes(p)), st));
    if (fold_operand_lse(*p)) {
      if (int rc = launch_fold_operands(p->lse, p->delta, fold_operand_lse(*p), fold_operand_delta(*p), q_row_count(*p),
                                        p->mask_value, p->dtype, st))
        return rc;
    }
  }
  if (int rc = launch_bwd_wide(*p, st)) return rc;
  return launch_dq_cast(p->dq_acc, p->dq, static_cast<long long>(p->batch) * p->heads, p->head_dim, p->q_len,
                                  p->dtype, st);
}

// ---------------------------------------------------------------------------
// Fused backward for callers that cannot allocate
// ---------------------------------------------------------------------------
// The f32 dQ accumulator lives in a fixed array inside the library image instead of
// caller-provided scratch.  In host code `g_static_dq_acc` is only a handle for the
// symbol, not a device address; the address a kernel can use comes from
// cudaGetSymbolAddress, looked up once per device with that device current.
constexpr size_t kStaticDqAccBytes = SPLASH_STATIC_DQ_ACC_BYTES;
static __device__ __align__(256) float g_static_dq_acc[kStaticDqAccBytes / sizeof(float)];

static int static_dq_acc_address(float** out) {
  constexpr int kMaxDevices = 64;
  static float* cache[kMaxDevices] = {};
  int dev = -1;
  SPLASH_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail(SPLASH_INVALID_ARGUMENT, "device ordinal out of range");
  float* ptr = __atomic_load_n(&cache[dev], __ATOMIC_ACQUIRE);
  if (!ptr) {
    void* sym = nullptr;
    SPLASH_CUDA_CHECK(cudaGetSymbolAddress(&sym, g_static_dq_acc));
    if (!sym) return fail(SPLASH_CUDA_ERROR, "cudaGetSymbolAddress returned a null address");
    ptr = static_cast<float*>(sym);
    __atomic_store_n(&cache[dev], ptr, __ATOMIC_RELEASE);
  }
  *out = ptr;
  return SPLASH_OK;
}

extern "C" int splash_bwd_fused_static(const SplashParams* p, void* stream) {
  if (int rc = check_bwd_fused(p)) return rc;
  SplashParams q = *p;
  const int64_t need = splash_bwd_fused_workspace_bytes(&q);
  if (need <= 0 || static_cast<uint64_t>(need) > kStaticDqAccBytes) {
    char d[160];
    snprintf(d, sizeof d, "the scratch for these shapes is %lld bytes, the built-in one holds %zu",
             static_cast<long long>(need), kStaticDqAccBytes);
    return fail(SPLASH_BUDGET_EXCEEDED, "problem too large for splash_bwd_fused_static", d);
  }
  float* acc = nullptr;
  if (int rc = static_dq_acc_address(&acc)) return rc;
  q.dq_acc = acc;  // whatever the caller put there is ignored
  return splash_bwd_fused(&q, stream);
}

extern "C" int splash_read_status(const int32_t* status, int32_t* host_out, void* stream) {
  int32_t h[4] = {0, 0, 0, 0};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SPLASH_CUDA_CHECK(cudaMemcpyAsync(h, status, sizeof h, cudaMemcpyDeviceToHost, st));
  SPLASH_CUDA_CHECK(cudaStreamSynchronize(st));
  if (host_out) memcpy(host_out, h, sizeof h);
  if (h[0] != 0) {
    char d[128];
    snprintf(d, sizeof d, "code %d at wait site %d, block %d, step %d", h[0], h[1], h[2], h[3]);
    return fail(SPLASH_DEVICE_TIMEOUT, "a kernel gave up waiting", d);
  }
  return SPLASH_OK;
}

extern "C" int splash_status_copy(const int32_t* status, int32_t* host, void* stream, void* side_stream, void* launched,
                                  void* copied) {
  if (!status || !host || !side_stream || !launched || !copied)
    return fail(SPLASH_INVALID_ARGUMENT, "splash_status_copy needs the word, its host copy, a side stream and two events");
  cudaStream_t side = static_cast<cudaStream_t>(side_stream);
  SPLASH_CUDA_CHECK(cudaEventRecord(static_cast<cudaEvent_t>(launched), static_cast<cudaStream_t>(stream)));
  SPLASH_CUDA_CHECK(cudaStreamWaitEvent(side, static_cast<cudaEvent_t>(launched), 0));
  SPLASH_CUDA_CHECK(cudaMemcpyAsync(host, status, 4 * sizeof(int32_t), cudaMemcpyDeviceToHost, side));
  SPLASH_CUDA_CHECK(cudaEventRecord(static_cast<cudaEvent_t>(copied), side));
  return SPLASH_OK;
}

extern "C" const char* splash_status_string(int status) {
  switch (status) {
    case SPLASH_OK: return "ok";
    case SPLASH_INVALID_ARGUMENT: return "invalid argument";
    case SPLASH_UNSUPPORTED: return "unsupported configuration";
    case SPLASH_BUDGET_EXCEEDED: return "shared/tensor memory budget exceeded";
    case SPLASH_CUDA_ERROR: return "CUDA error";
    case SPLASH_DEVICE_TIMEOUT: return "device-side wait timed out";
    default: return "unknown status";
  }
}

extern "C" const char* splash_last_error(void) { return last_error_buf(); }
