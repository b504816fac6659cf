// Second pass of a forward whose q tiles were shared by several CTAs (splits > 1):
//   m = max_i m_i, w_i = 2^((m_i - m) log2 e), l = sum_i w_i l_i, out = sum_i w_i O_i / l,
//   lse = m + ln l (mask_value and zeros where no part saw a key),
// all in f32, as one CTA per tile would have it.  One warp per q row, a float4 of the row per lane;
// bound by the read of the parts, which the first pass has just left in L2.
#include "dispatch.h"
#include "fwd_kernel.cuh"
#include "host_common.cuh"

namespace splash {

template <bool BF16>
__global__ void __launch_bounds__(256) fwd_combine_kernel(const float4* __restrict__ part_o,
                                                          const float2* __restrict__ part_ml, uint2* __restrict__ out,
                                                          float* __restrict__ lse, long long rows, int vecs, int splits,
                                                          float mask_value) {
  const long long row = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  float m = -INFINITY;
  for (int i = 0; i < splits; ++i) {
    const float2 ml = part_ml[i * rows + row];
    if (ml.y != 0.f) m = fmaxf(m, ml.x);  // a part without a sum has seen no key
  }
  float l = 0.f;
  for (int i = 0; i < splits; ++i) {
    const float2 ml = part_ml[i * rows + row];
    if (ml.y != 0.f) l = fmaf(ml.y, ex2_approx((ml.x - m) * kLog2e), l);
  }
  const float inv_l = l > 0.f ? 1.f / l : 0.f;
  for (int c = lane; c < vecs; c += 32) {
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = 0; i < splits; ++i) {
      const float2 ml = part_ml[i * rows + row];
      if (ml.y == 0.f) continue;
      const float w = ex2_approx((ml.x - m) * kLog2e);
      const float4 x = part_o[(i * rows + row) * vecs + c];
      o.x = fmaf(x.x, w, o.x);
      o.y = fmaf(x.y, w, o.y);
      o.z = fmaf(x.z, w, o.z);
      o.w = fmaf(x.w, w, o.w);
    }
    out[row * vecs + c] = make_uint2(pack2<BF16>(o.x * inv_l, o.y * inv_l), pack2<BF16>(o.z * inv_l, o.w * inv_l));
  }
  if (lse && lane == 0) lse[row] = l > 0.f ? m + lg2_approx(l) * kLn2 : mask_value;
}

int launch_fwd_combine(const SplashParams& p, int splits, const void* workspace, cudaStream_t stream) {
  const long long rows = q_row_count(p);
  const float* part_o = static_cast<const float*>(workspace);
  const float2* part_ml = reinterpret_cast<const float2*>(part_o + static_cast<size_t>(splits) * rows * p.head_dim_v);
  const unsigned grid = static_cast<unsigned>((rows + 7) / 8);
  auto kernel = p.dtype == SPLASH_DTYPE_BF16 ? fwd_combine_kernel<true> : fwd_combine_kernel<false>;
  kernel<<<grid, 256, 0, stream>>>(reinterpret_cast<const float4*>(part_o), part_ml, static_cast<uint2*>(p.out), p.lse_out,
                                   rows, p.head_dim_v / 4, splits, p.mask_value);
  SPLASH_CUDA_CHECK(cudaGetLastError());
  return SPLASH_OK;
}

}  // namespace splash
