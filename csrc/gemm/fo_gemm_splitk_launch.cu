// Instantiations of the split-K GEMM and the choice of the kernel of a GEMM without a collective.
#include "fo_gemm.h"
#include "fo_gemm_splitk_sm100.cuh"

#include <algorithm>

namespace fo {

namespace {

template <bool BF16, int S>
cudaError_t launch_one(const SplitTensorMaps& maps, const GemmParams* p, cudaStream_t stream, int* query) {
  constexpr int smem = SplitSmem<S>::kTotalBytes;
  static_assert(smem <= 227 * 1024, "shared memory of this configuration exceeds 227 KB");
  static bool attr_set[16] = {};
  auto kernel = fo_gemm_splitk_kernel<BF16, S>;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16 || !attr_set[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 16) attr_set[dev] = true;
  }
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kSplitThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (query != nullptr) {
    cfg.gridDim = dim3(S, 1, 1);
    return cudaOccupancyMaxActiveClusters(query, kernel, &cfg);
  }
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  cfg.gridDim = dim3(p->tiles_m * p->tiles_n * S, 1, 1);
  return cudaLaunchKernelEx(&cfg, kernel, maps, *p);
}

cudaError_t dispatch(int split, bool bf16, const SplitTensorMaps& maps, const GemmParams* p, cudaStream_t s, int* query) {
  switch (split) {
    case 2: return bf16 ? launch_one<true, 2>(maps, p, s, query) : launch_one<false, 2>(maps, p, s, query);
    case 4: return bf16 ? launch_one<true, 4>(maps, p, s, query) : launch_one<false, 4>(maps, p, s, query);
    case 8: return bf16 ? launch_one<true, 8>(maps, p, s, query) : launch_one<false, 8>(maps, p, s, query);
    default: return cudaErrorInvalidValue;
  }
}

// Clusters of `split` CTAs that fit the current device at once (cached per device; 0 when the query fails).
int max_clusters(int split, bool bf16) {
  static int cache[16][9][2] = {};  // 0: not asked yet, else the count + 1
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16) return 0;
  int& slot = cache[dev][split][bf16 ? 1 : 0];
  if (slot == 0) {
    int n = 0;
    const SplitTensorMaps none = {};
    if (dispatch(split, bf16, none, nullptr, nullptr, &n) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    slot = n + 1;
  }
  return slot - 1;
}

// ---------------------------------------------------------------------------- choice of a kernel
//
// A model of the time of one call, in us, with what was measured on a B200 (1,590 TFLOP/s bf16, 6.5 TB/s):
//  * a tile's main loop takes, per 64-wide k-block, 0.386 us for CTA pairs on 256 x 256 (the tensor
//    rate), 0.247 us on 256 x 128 and 0.44 / 0.27 us for a CTA by itself on 128 x 256 / 128 (the L2's
//    rate), 0.77 us for pairs on 512 x 256, whose epilogue (1.5 us) nothing hides;
//  * tiles beyond one per CTA or pair take further waves;
//  * a split's CTAs take in operands at 140 KB/us each, and 6,500 KB/us together; the two cluster
//    barriers take 0.7 us and the exchange 26 KB/us per CTA.
struct KernelCost {
  double per_kb, epilogue;
};
KernelCost kernel_cost(const AlgoConfig& c) {
  if (c.mt == 2) return {0.77, 1.5};
  if (c.cta2) return c.bn == 256 ? KernelCost{0.386, 0.0} : KernelCost{0.247, 0.0};
  return c.bn == 256 ? KernelCost{0.44, 0.0} : KernelCost{0.27, 0.0};
}

double plain_time(const GemmParams& p, int algo, bool bf16, int num_kb) {
  const AlgoConfig c = algo_config(algo);
  const int units = plain_units(p, algo);
  const int slots = std::max(1, gemm_max_resident_ctas(algo, bf16, false) / (c.cta2 ? 2 : 1));
  const KernelCost k = kernel_cost(c);
  if (c.cta2 && c.mt == 1 && c.bn == 256 && plain_tail(units, slots) > 0) {
    return num_kb * (units / slots * k.per_kb + 0.247);  // the last wave in halves
  }
  return (units + slots - 1) / slots * (num_kb * k.per_kb + k.epilogue);
}

int algo_of(int bn, bool cta2, int raster_sw) {
  for (int a = 0; a < kNumAlgos; ++a) {
    const AlgoConfig t = algo_config(a);
    if (t.bn == bn && (t.cta2 != 0) == cta2 && t.mt == 1 && t.raster_sw == raster_sw) return a;
  }
  return -1;
}

}  // namespace

PlainPlan choose_plain(const GemmParams& p, int algo, bool bf16, int split, bool exact) {
  PlainPlan plan{algo, 0};
  const bool reorder = p.out_mode == kOutReorder;
  if (p.signal != 0 || p.monitor != 0 || (!reorder && p.out_mode != kOutNatural) || exact) return plan;
  const AlgoConfig own = algo_config(algo);
  const int num_kb = (p.K + kBK - 1) / kBK;
  double best = plain_time(p, algo, bf16, num_kb);
  // The Algo's own kernel unless another is expected to save 7 %: the model is no better than that.
  double bound = 0.93 * best;
  for (int bn : {256, 128}) {
    // tiles of the tile-contiguous layout may be computed in parts, not together
    if (p.N % bn != 0 || (reorder && bn > own.bn)) continue;
    for (bool cta2 : {true, false}) {
      if (cta2 && p.tiles_m < 2) continue;
      const int a = algo_of(bn, cta2, own.raster_sw);
      if (a < 0 || a == algo) continue;
      const double t = plain_time(p, a, bf16, num_kb);
      if (t < bound) {
        plan.algo = a;
        best = bound = t;
      }
    }
  }
  if (split == 0 || p.N % kSplitBN != 0) return plan;
  const int tiles = p.tiles_m * (p.N / kSplitBN);
  const double unique_us = 2e-3 * p.K * (static_cast<double>(p.M) + p.N) / 6500.0;
  for (int s : {2, 4, 8}) {
    if (split > 0 && s != split) continue;
    if (num_kb < s || tiles > max_clusters(s, bf16)) continue;
    const double operands_us = (num_kb + s - 1) / s * 32.0 / 140.0;
    const double exchange_us = 0.7 + 64.0 * (s - 1) / s / 26.0;
    const double t = std::max(operands_us, unique_us) + exchange_us;
    if (split > 0 || t < 0.93 * std::max(best, unique_us)) {
      plan.split = s;
      best = t;
      if (split > 0) break;
    }
  }
  return plan;
}

cudaError_t launch_splitk_gemm(int split, bool bf16, const CUtensorMap& a, const CUtensorMap& b, const GemmParams& p,
                               cudaStream_t stream) {
  SplitTensorMaps maps;
  maps.a = a;
  maps.b = b;
  return dispatch(split, bf16, maps, &p, stream, nullptr);
}

}  // namespace fo
