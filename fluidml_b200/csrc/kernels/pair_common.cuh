// What the half-precision-pair kernels share (gemm_pair.cu, conv_pair.cu): the split of an fp32 value into
// two fp16 ones, the power-of-two scales, and the packed form of constant right-hand sides.
#pragma once
#include "tc_common.cuh"
#include <cuda_fp16.h>

namespace fml {

constexpr int kPK = 32;                // k values per block: 128 bytes of fp32, 64 of fp16
constexpr int kPairB = kPK * 4;        // bytes of B per block and column: hi and lo
constexpr int kAtom = 8 * kPK * 2;     // bytes of an atom: 8 columns x 32 k values of fp16

// 2^k for -126 <= k <= 127.
__device__ __forceinline__ float pow2(int k) { return __uint_as_float((uint32_t)(127 + k) << 23); }
// The exponent that brings a largest magnitude m into [2^target, 2^(target + 1)), limited so that the
// power and its inverse are normal numbers.
__device__ __forceinline__ int scale_exponent(float m, int target) {
  return min(max(target - ((int)(__float_as_uint(m) >> 23) - 127), -126), 126);
}

// Two fp32 values -> (hi pair, lo pair) of x * s.
__device__ __forceinline__ void split_pair(float x0, float x1, float s, uint32_t &hi, uint32_t &lo) {
  const __half2 h = __floats2half2_rn(x0 * s, x1 * s);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(fmaf(x0, s, -f.x), fmaf(x1, s, -f.y));
  hi = *reinterpret_cast<const uint32_t *>(&h);
  lo = *reinterpret_cast<const uint32_t *>(&l);
}

// Largest magnitude of src[k0, k1) (16-byte aligned at k0, a multiple of 4), by the whole warp.
__device__ __forceinline__ float warp_row_max(const float *src, int64_t k0, int64_t k1, int lane) {
  float m = 0.0f;
  const int64_t whole = k0 + ((k1 - k0) & ~3ll);
#pragma unroll 4
  for (int64_t k = k0 + lane * 4; k < whole; k += 128) {
    const float4 x = *reinterpret_cast<const float4 *>(src + k);
    m = fmaxf(m, fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w))));
  }
  if (whole + lane < k1) m = fmaxf(m, fabsf(src[whole + lane]));
  return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));  // non-negative floats order as their bits
}

}  // namespace fml
