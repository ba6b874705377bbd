// Device helpers shared by the tcgen05 GEMM kernels: tile order, wave groups.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>

#include "../common/fo_pack16.cuh"
#include "../common/fo_ptx.cuh"
#include "fo_gemm_params.h"

namespace fo {

struct TileCoord {
  int m, n;
};

// Position in the launch order -> tile coordinates.  Tiles are swept in column strips
// `sw` tiles wide, M-major inside a strip; sw == tiles_n gives row-panel-major order.
__device__ __forceinline__ TileCoord tile_of_position(int pos, int tiles_m, int tiles_n, int sw) {
  const int per_strip = tiles_m * sw;
  const int s = pos / per_strip;
  const int q = pos - s * per_strip;
  const int w = min(sw, tiles_n - s * sw);
  TileCoord c;
  c.m = q / w;
  c.n = s * sw + (q - c.m * w);
  return c;
}

// Wave group of reordered position r: groups are runs of cseg[g] consecutive positions.
__device__ __forceinline__ void group_of_position(const GemmParams& p, int r, int* g, int* need) {
  // No grouping, or as many groups as tiles (every group then holds exactly one tile).
  if (p.num_groups <= 0 || p.cseg == nullptr || p.num_groups == p.num_tiles) {
    *g = r;
    *need = 1;
    return;
  }
  int acc = 0, i = 0, n = 1;
  for (; i < p.num_groups; ++i) {
    n = p.cseg[i];
    acc += n;
    if (r < acc) break;
  }
  if (i >= p.num_groups) i = p.num_groups - 1;
  *g = i;
  *need = n;
}

// Reordered position of natural tile t.  A value outside [0, tiles) - a corrupted RA, or one
// built for another shape - would become an out-of-range address and counter index: it is
// reported (kStatusBadArgument) and replaced by t, so the kernel stays inside its buffers;
// the result is then wrong and the status words say why.
__device__ __forceinline__ int tile_position(const GemmParams& p, int t, int32_t* status) {
  if (p.RA == nullptr) return t;
  const int r = p.RA[t];
  if (static_cast<unsigned>(r) >= static_cast<unsigned>(p.num_tiles)) {
    ptx::report_status(status, kStatusBadArgument, 1, t, r);
    return t;
  }
  return r;
}

template <bool BF16>
__device__ __forceinline__ void unpack_add(uint32_t w, float& lo, float& hi) {
  const float2 f = unpack2<BF16>(w);
  lo += f.x;
  hi += f.y;
}

}  // namespace fo
