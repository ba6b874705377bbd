// Arithmetic on pairs of 16-bit elements (bf16 or fp16) held in 32-bit words, shared by all kernels.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cstdint>

namespace fo {

template <bool BF16>
__device__ __forceinline__ float2 unpack2(uint32_t w) {
  if constexpr (BF16) {
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&w));
  } else {
    return __half22float2(*reinterpret_cast<__half2*>(&w));
  }
}

template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (BF16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}

// round16(a + b) per element, added in fp32: what `a + b` on 16-bit tensors computes.
template <bool BF16>
__device__ __forceinline__ uint32_t add2(uint32_t a, uint32_t b) {
  const float2 x = unpack2<BF16>(a), y = unpack2<BF16>(b);
  return pack2<BF16>(x.x + y.x, x.y + y.y);
}

__device__ __forceinline__ float silu(float x) { return x / (1.f + expf(-x)); }

}  // namespace fo
