// Instantiations of the split-K GEMM and the rule that chooses a split.
#include "fo_gemm.h"
#include "fo_gemm_splitk_sm100.cuh"

namespace fo {

namespace {

template <int BN, int STAGES, bool BF16, int S>
cudaError_t launch_one(const SplitTensorMaps& maps, const GemmParams* p, cudaStream_t stream, int* query) {
  constexpr int smem = SplitSmem<BN, STAGES>::kTotalBytes;
  static_assert(smem <= 227 * 1024, "shared memory of this configuration exceeds 227 KB");
  static bool attr_set[16] = {};
  auto kernel = fo_gemm_splitk_kernel<BN, STAGES, BF16, S>;
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
  cfg.gridDim = dim3(p->num_tiles * S, 1, 1);
  return cudaLaunchKernelEx(&cfg, kernel, maps, *p);
}

template <bool BF16>
cudaError_t dispatch(int bn, int split, const SplitTensorMaps& maps, const GemmParams* p, cudaStream_t s, int* query) {
  if (bn == 256) {
    if (split == 2) return launch_one<256, 4, BF16, 2>(maps, p, s, query);
    if (split == 4) return launch_one<256, 4, BF16, 4>(maps, p, s, query);
    if (split == 8) return launch_one<256, 4, BF16, 8>(maps, p, s, query);
  } else if (bn == 128) {
    if (split == 2) return launch_one<128, 6, BF16, 2>(maps, p, s, query);
    if (split == 4) return launch_one<128, 6, BF16, 4>(maps, p, s, query);
    if (split == 8) return launch_one<128, 6, BF16, 8>(maps, p, s, query);
  }
  return cudaErrorInvalidValue;
}

constexpr int kSplits[] = {2, 4, 8};

// Clusters of a kernel that fit the device at once (cached per device; 0 when the query fails).
int max_clusters(int bn, int si, bool bf16) {
  static int cache[16][2][3][2] = {};  // 0: not asked yet, else the count + 1
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16) return 0;
  int& slot = cache[dev][bn == 256][si][bf16];
  if (slot == 0) {
    int n = 0;
    const SplitTensorMaps none = {};
    const cudaError_t e = bf16 ? dispatch<true>(bn, kSplits[si], none, nullptr, nullptr, &n)
                               : dispatch<false>(bn, kSplits[si], none, nullptr, nullptr, &n);
    if (e != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    slot = n + 1;
  }
  return slot - 1;
}

}  // namespace

SplitChoice choose_split(const GemmParams& p, int bn, bool bf16, int forced) {
  SplitChoice best{0, 0};
  if (p.signal != 0 || p.monitor != 0 || forced == 0) return best;
  const bool natural = p.out_mode == kOutNatural;
  if (!natural && p.out_mode != kOutReorder) return best;
  const int num_kb = (p.K + kBK - 1) / kBK;
  int best_cost = 0;
  for (int b : {256, 128}) {
    if (p.N % b != 0 || (!natural && b != bn)) continue;
    const int tiles = p.tiles_m * (p.N / b);
    for (int si = 0; si < 3; ++si) {
      const int s = kSplits[si];
      if (forced > 0 && s != forced) continue;
      if (num_kb < s * (forced > 0 ? 1 : kMinSplitBlocks)) continue;
      if (tiles > max_clusters(b, si, bf16)) continue;
      const int cost = ((num_kb + s - 1) / s) * (kBM + b);  // operand bytes one CTA takes in
      if (best.split == 0 || cost < best_cost) {
        best = {b, s};
        best_cost = cost;
      }
    }
  }
  return best;
}

cudaError_t launch_splitk_gemm(SplitChoice c, bool bf16, const CUtensorMap& a, const CUtensorMap& b,
                               const GemmParams& p, cudaStream_t stream) {
  SplitTensorMaps maps;
  maps.a = a;
  maps.b = b;
  return bf16 ? dispatch<true>(c.bn, c.split, maps, &p, stream, nullptr)
              : dispatch<false>(c.bn, c.split, maps, &p, stream, nullptr);
}

}  // namespace fo
