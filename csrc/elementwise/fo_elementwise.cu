#include "fo_elementwise.h"

#include <cstdint>

#include "../common/fo_pack16.cuh"

namespace fo {

namespace {

constexpr int kThreads = 256;

// Bound by memory: 4096 tokens x 9 heads of 128 (19 MB moved) took 284 us as the fourteen eager
// operators of the two rotations (fp32 intermediates, strided pairs) and take 9 us here.
// A thread owns 8 adjacent elements (4 pairs) of one position and walks kHeadsPerThread heads, whose
// loads are all in flight while it computes the four angles they share.
constexpr int kHeadsPerThread = 8;

template <bool BF16>
__global__ void __launch_bounds__(kThreads)
    rope_kernel(uint16_t* __restrict__ qkv, int tokens, int seq, int heads, int head_dim, int row_elems, float theta) {
  const int per_head = head_dim / 8;
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;
  const int64_t token = idx / per_head;
  if (token >= tokens) return;
  const int d = static_cast<int>(idx - token * per_head) * 8;
  const int h0 = blockIdx.y * kHeadsPerThread;
  const int h1 = min(heads, h0 + kHeadsPerThread);
  uint16_t* row = qkv + token * row_elems + d;
  uint4 x[kHeadsPerThread];
#pragma unroll
  for (int i = 0; i < kHeadsPerThread; ++i) {
    if (h0 + i < h1) x[i] = *reinterpret_cast<const uint4*>(row + static_cast<int64_t>(h0 + i) * head_dim);
  }
  const float pos = static_cast<float>(token % seq);
  float c[4], s[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float inv = powf(theta, -static_cast<float>(d + 2 * k) / static_cast<float>(head_dim));
    sincosf(pos * inv, &s[k], &c[k]);
  }
#pragma unroll
  for (int i = 0; i < kHeadsPerThread; ++i) {
    if (h0 + i < h1) {
      uint32_t* u = reinterpret_cast<uint32_t*>(&x[i]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 v = unpack2<BF16>(u[k]);
        u[k] = pack2<BF16>(v.x * c[k] - v.y * s[k], v.x * s[k] + v.y * c[k]);
      }
      *reinterpret_cast<uint4*>(row + static_cast<int64_t>(h0 + i) * head_dim) = x[i];
    }
  }
}

template <bool BF16>
__device__ __forceinline__ uint32_t silu_mul(uint32_t g, uint32_t u) {
  const float2 a = unpack2<BF16>(g);
  // silu is rounded to the storage type before the product, as two operators in a row round it
  const uint32_t r = pack2<BF16>(silu(a.x), silu(a.y));
  const float2 p = unpack2<BF16>(r), q = unpack2<BF16>(u);
  return pack2<BF16>(p.x * q.x, p.y * q.y);
}

template <bool BF16>
__device__ __forceinline__ uint4 silu_mul8(const uint4& g, const uint4& u) {
  return make_uint4(silu_mul<BF16>(g.x, u.x), silu_mul<BF16>(g.y, u.y), silu_mul<BF16>(g.z, u.z),
                    silu_mul<BF16>(g.w, u.w));
}

// Bound by memory: 4096 x 7168 -> 3584 (88 MB) took 81 us as silu and a product over strided halves
// and takes 20 us here.  One row at a time per CTA (grid-strided), two vectors of each operand in flight per thread.
template <bool BF16>
__global__ void __launch_bounds__(kThreads)
    swiglu_kernel(const uint16_t* __restrict__ gu, uint16_t* __restrict__ y, int rows, int f) {
  const int nvec = f / 8;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const uint4* g = reinterpret_cast<const uint4*>(gu + static_cast<int64_t>(r) * 2 * f);
    const uint4* u = g + nvec;
    uint4* o = reinterpret_cast<uint4*>(y + static_cast<int64_t>(r) * f);
    for (int j = threadIdx.x; j < nvec; j += 2 * kThreads) {
      const bool two = j + kThreads < nvec;
      const uint4 g0 = __ldcs(g + j), u0 = __ldcs(u + j);
      uint4 g1 = {}, u1 = {};
      if (two) {
        g1 = __ldcs(g + j + kThreads);
        u1 = __ldcs(u + j + kThreads);
      }
      o[j] = silu_mul8<BF16>(g0, u0);
      if (two) o[j + kThreads] = silu_mul8<BF16>(g1, u1);
    }
  }
}

}  // namespace

cudaError_t rope_launch(void* QKV, int tokens, int seq, int heads, int head_dim, int row_elems, float theta, bool bf16,
                        cudaStream_t stream) {
  if (head_dim < 8 || head_dim % 8 != 0 || row_elems % 8 != 0 || seq < 1) return cudaErrorInvalidValue;
  if (tokens == 0 || heads == 0) return cudaSuccess;
  const int64_t threads = static_cast<int64_t>(tokens) * (head_dim / 8);
  const dim3 grid(static_cast<unsigned>((threads + kThreads - 1) / kThreads),
                  static_cast<unsigned>((heads + kHeadsPerThread - 1) / kHeadsPerThread));
  uint16_t* q = static_cast<uint16_t*>(QKV);
  if (bf16) {
    rope_kernel<true><<<grid, kThreads, 0, stream>>>(q, tokens, seq, heads, head_dim, row_elems, theta);
  } else {
    rope_kernel<false><<<grid, kThreads, 0, stream>>>(q, tokens, seq, heads, head_dim, row_elems, theta);
  }
  return cudaGetLastError();
}

cudaError_t swiglu_launch(const void* GU, void* Y, int rows, int f, bool bf16, int sm_count, cudaStream_t stream) {
  if (f % 8 != 0) return cudaErrorInvalidValue;
  if (rows == 0 || f == 0) return cudaSuccess;
  const int grid = rows < sm_count * 32 ? rows : sm_count * 32;
  const uint16_t* g = static_cast<const uint16_t*>(GU);
  uint16_t* y = static_cast<uint16_t*>(Y);
  if (bf16) {
    swiglu_kernel<true><<<grid, kThreads, 0, stream>>>(g, y, rows, f);
  } else {
    swiglu_kernel<false><<<grid, kThreads, 0, stream>>>(g, y, rows, f);
  }
  return cudaGetLastError();
}

}  // namespace fo
