// Host-side launch helper shared by the translation units that instantiate the GEMM kernels.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "fo_gemm_params.h"

namespace fo {

// Common part of every launch.  query != nullptr: do not launch, report the largest co-resident
// grid instead.  programmatic: the kernel calls ptx::grid_wait before it touches global memory, so
// its launch and prologue may overlap the tail of the stream's previous kernel.
template <bool CTA2, typename Kernel, typename Maps>
cudaError_t launch_kernel(Kernel kernel, int threads, int smem, bool* attr_set, const Maps* maps, const GemmParams* p,
                          int grid_x, int nvr, bool cooperative, bool programmatic, cudaStream_t stream, int* query) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 16 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[3];
  cfg.attrs = attr;
  cfg.numAttrs = 0;
  if (CTA2) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = 2;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  if (query != nullptr) {
    int sm_count = 0;  // one attribute: all of cudaGetDeviceProperties takes milliseconds
    cudaError_t e = cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    if (!CTA2) {
      *query = sm_count;  // shared memory admits exactly one CTA per SM
      return cudaSuccess;
    }
    cfg.gridDim = dim3(sm_count & ~1, 1, 1);
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
    if (e != cudaSuccess) return e;
    *query = 2 * clusters;
    return cudaSuccess;
  }
  if (CTA2) grid_x &= ~1;
  if (grid_x < (CTA2 ? 2 : 1)) grid_x = CTA2 ? 2 : 1;
  cfg.gridDim = dim3(grid_x, nvr, 1);
  if (cooperative) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeCooperative;
    attr[cfg.numAttrs].val.cooperative = 1;
    ++cfg.numAttrs;
  }
  if (programmatic) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  return cudaLaunchKernelEx(&cfg, kernel, *maps, *p);
}

// The kernels without a collective (fo_gemm_plain_launch.cu): `kidx` indexes
// gemm/fo_gemm_instances.inc, maps / p as for launch_gemm with one rank; query as above (maps and
// p may then be nullptr).
cudaError_t launch_plain_gemm(int kidx, bool bf16, const GemmTensorMaps* maps, const GemmParams* p, int grid_x,
                              cudaStream_t stream, int* query);

}  // namespace fo
