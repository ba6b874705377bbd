// Instantiations of the GEMM kernels without a collective.
#include "fo_gemm_launch.cuh"
#include "fo_gemm_plain_sm100.cuh"

namespace fo {

namespace {

template <int BN, int STAGES, bool BF16, bool CTA2, int MT, int EPI>
cudaError_t launch_plain_one(const PlainTensorMaps* maps, const GemmParams* p, int grid_x, cudaStream_t stream,
                             int* query) {
  constexpr int smem = PlainSmem<BN, STAGES, CTA2, MT>::kTotalBytes;
  static_assert(smem <= 227 * 1024, "shared memory of this configuration exceeds 227 KB");
  static bool attr_set[16] = {};
  return launch_kernel<CTA2>(fo_gemm_plain_kernel<BN, STAGES, BF16, CTA2, MT, EPI>, kPlainThreads, smem, attr_set, maps, p,
                             grid_x, 1, false, true, stream, query);
}

template <bool BF16, int EPI>
cudaError_t launch_plain(int kidx, const PlainTensorMaps* maps, const GemmParams* p, int grid_x, cudaStream_t s,
                         int* query) {
  switch (kidx) {
#define FO_GEMM_KERNEL(idx, bn, stages, cta2, mt, stages_epi4) \
  case idx: return launch_plain_one<bn, stages, BF16, cta2, mt, EPI>(maps, p, grid_x, s, query);
#include "fo_gemm_instances.inc"
#undef FO_GEMM_KERNEL
    default: return cudaErrorInvalidValue;
  }
}

// The SwiGLU epilogue exists for the kernels whose CTA pairs split a 256-wide B tile.
template <bool BF16, int BN, int STAGES, bool CTA2, int MT>
cudaError_t launch_swiglu_one(const PlainTensorMaps* maps, const GemmParams* p, int grid_x, cudaStream_t s) {
  if constexpr (CTA2 && MT == 1 && BN == 256) {
    return launch_plain_one<BN, STAGES, BF16, CTA2, MT, kEpiSwiGLU>(maps, p, grid_x, s, nullptr);
  } else {
    return cudaErrorInvalidValue;
  }
}

template <bool BF16>
cudaError_t launch_swiglu(int kidx, const PlainTensorMaps* maps, const GemmParams* p, int grid_x, cudaStream_t s) {
  switch (kidx) {
#define FO_GEMM_KERNEL(idx, bn, stages, cta2, mt, stages_epi4) \
  case idx: return launch_swiglu_one<BF16, bn, stages, cta2, mt>(maps, p, grid_x, s);
#include "fo_gemm_instances.inc"
#undef FO_GEMM_KERNEL
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t launch_plain_gemm(int kidx, bool bf16, const GemmTensorMaps* maps, const GemmParams* p, int grid_x,
                              cudaStream_t stream, int* query) {
  PlainTensorMaps pm;  // only one rank's maps travel
  if (maps != nullptr) {
    pm.a = maps->a[0];
    pm.b = maps->b[0];
    pm.st = maps->st[0];
    pm.b_half = maps->b[1];
  }
  switch (p != nullptr ? p->epilogue : kEpiStore) {
    case kEpiStore:
      return bf16 ? launch_plain<true, kEpiStore>(kidx, &pm, p, grid_x, stream, query)
                  : launch_plain<false, kEpiStore>(kidx, &pm, p, grid_x, stream, query);
    case kEpiResidual:
      return bf16 ? launch_plain<true, kEpiResidual>(kidx, &pm, p, grid_x, stream, query)
                  : launch_plain<false, kEpiResidual>(kidx, &pm, p, grid_x, stream, query);
    case kEpiSwiGLU:
      return bf16 ? launch_swiglu<true>(kidx, &pm, p, grid_x, stream) : launch_swiglu<false>(kidx, &pm, p, grid_x, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fo
