// Weights of the 16-bit parts that -lse and -delta are split into where the fused backward folds them into its
// score products (head_dim 64): written by the pre-pass (bwd_misc.cu), multiplied in bwd_wide_kernel.cuh.
#pragma once

#include <stdint.h>

namespace splash {

template <bool BF16>
struct FoldWeights;

template <>
struct FoldWeights<true> {
  static constexpr int kParts = 3;
  static constexpr uint32_t kLo = 0x3f803f80u, kHi = 0x00003f80u;  // {1, 1}, {1, 0} as bf16
};

// Each weight is small enough for the remainder that the part before it leaves (2^-12 of what it was given, or
// half a subnormal step of f16, 2^-25 of the weight) and large enough not to overflow there.
template <>
struct FoldWeights<false> {
  static constexpr int kParts = 4;
  static constexpr uint32_t kLo = 0x4c007800u, kHi = 0x04002000u;  // {2^15, 2^4}, {2^-7, 2^-14} as f16
  __host__ __device__ static constexpr float weight(int i) {
    return i == 0 ? 32768.f : i == 1 ? 16.f : i == 2 ? 1.f / 128.f : 1.f / 16384.f;
  }
};

}  // namespace splash
