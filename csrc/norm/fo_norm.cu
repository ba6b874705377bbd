// Memory-bound row kernels: RMSNorm, residual add + RMSNorm, fused tile-un-reorder + RMSNorm, and the standalone
// row-major <-> tile-contiguous reorder.  Counterparts of the reference's
// reorder_rmsnorm_kernel / rmsnorm_kernel (src/rmsnorm/rmsnorm.cuh:14-117); the standalone
// reorder has no counterpart there (its layout change only ever happens inside the GEMM
// epilogue and the norm kernel).
//
// Differences from the reference kernels, on purpose: eps is an argument (it is hard-coded
// to 1e-5 at src/rmsnorm/rmsnorm.cuh:102), launches take a stream (the reference launches
// on the legacy default stream, src/rmsnorm/rmsnorm.cu:23), bf16 as well as fp16, and each
// thread keeps several 16-byte vectors in flight so that a B200 SM can cover HBM3e latency.
#include "fo_norm.h"

#include <cstdint>

#include "../common/fo_pack16.cuh"
#include "../common/fo_ptx.cuh"

namespace fo {

namespace {

constexpr int kNormThreads = 256;

// y = round16(round16(x * scale) * w): the normalised value is rounded to the storage type
// before the weight multiply, as in the reference (src/rmsnorm/rmsnorm.cuh:108-113) and in
// the usual `norm(x.float()).type_as(x) * weight` module.
template <bool BF16>
__device__ __forceinline__ uint32_t scale_mul2(uint32_t x, uint32_t w, float scale) {
  const float2 xf = unpack2<BF16>(x);
  if constexpr (BF16) {
    __nv_bfloat162 n = __floats2bfloat162_rn(xf.x * scale, xf.y * scale);
    __nv_bfloat162 r = __hmul2(n, *reinterpret_cast<__nv_bfloat162*>(&w));
    return *reinterpret_cast<uint32_t*>(&r);
  } else {
    __half2 n = __floats2half2_rn(xf.x * scale, xf.y * scale);
    __half2 r = __hmul2(n, *reinterpret_cast<__half2*>(&w));
    return *reinterpret_cast<uint32_t*>(&r);
  }
}

__device__ __forceinline__ float block_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();  // protects `red` against the previous row's readers
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < kNormThreads / 32) ? red[lane] : 0.f;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return __shfl_sync(0xffffffffu, t, 0);
}

// Element offset, in the tile-contiguous buffer, of logical (row b, column col).
__device__ __forceinline__ size_t reordered_offset(int b, int col, int dim, int BM, int BN,
                                                   int rldn, const int* __restrict__ RA) {
  const int t = (b / BM) * (dim / BN) + col / BN;
  const int r = RA[t];
  const size_t ld = static_cast<size_t>(rldn) * BN;
  return (static_cast<size_t>(r / rldn) * BM + (b % BM)) * ld + static_cast<size_t>(r % rldn) * BN +
         (col % BN);
}

// CTAs per SM of the build without prefetch (a full set of warps for rows of up to 4096 elements, but the
// carve-out that leaves the most L1 holds the reserved shared memory of seven).
constexpr int norm_ctas_per_sm(int vpt) { return vpt <= 2 ? 7 : (vpt <= 4 ? 6 : 3); }

// Each CTA takes a contiguous block of rows; each thread owns VPT 16-byte vectors of a row
// (VPT * 256 * 8 >= dim).  Bound by memory.  PREFETCH: the weights stay in registers and the next row's
// vectors are requested before the current row is reduced (register double buffer).  Without: a
// tile-contiguous CTA's first loads wait for the look-ups of its tiles through RA, which more CTAs per
// SM hide better than a row of prefetch in each (six of 40 registers a thread instead of four of 64);
// the look-up is done only when the block of rows crosses into another row panel, not per row.
// 16384 x 8192 in tiles of 64 x 256: 93.4 -> 88.6 us, 4096 x 4096: 17.9 -> 14.6 us, 8192 x 16384: 106.8 -> 98.7 us.
// Few rows fit the machine at once either way, and there the weights' latency behind the reduction
// is what the second build adds: 64 x 8192 3.6 against 4.3 us, 2048 x 8192 15.7 against 17.4 us.
template <bool BF16, bool REORDER, int VPT, bool PREFETCH>
__global__ void __launch_bounds__(kNormThreads, !PREFETCH ? (VPT <= 2 ? 8 : norm_ctas_per_sm(VPT))
                                                          : (VPT <= 2 ? 6 : (VPT <= 4 ? 4 : 2)))
    rmsnorm_kernel(const uint16_t* __restrict__ X, uint16_t* __restrict__ Y,
                   const uint16_t* __restrict__ W, int rows, int dim, int BM, int BN, int rldn,
                   const int* __restrict__ RA, float eps) {
  __shared__ float red[kNormThreads / 32];
  const int nvec = dim / 8;
  const int per_cta = (rows + gridDim.x - 1) / gridDim.x;
  const int row_begin = blockIdx.x * per_cta;
  const int row_end = min(rows, row_begin + per_cta);
  ptx::grid_launch_dependents();
  ptx::grid_wait();
  if (row_begin >= row_end) return;

  // Without PREFETCH the weights are re-read from L1 per row.
  [[maybe_unused]] uint4 wv[VPT];
  if constexpr (PREFETCH) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int j = threadIdx.x + i * kNormThreads;
      if (j < nvec) wv[i] = *reinterpret_cast<const uint4*>(W + static_cast<size_t>(j) * 8);
    }
  }

  // Offset, in 16-byte vectors, of (row 0 of the current panel, this thread's column) per vector;
  // 32 bits cover 64 GiB of 16-bit elements.
  uint32_t panel_off[VPT];
  int panel = -1;
  const size_t ld = REORDER ? static_cast<size_t>(rldn) * BN : static_cast<size_t>(dim);
  auto load_row = [&](int b, uint4 (&dst)[VPT]) {
    if constexpr (REORDER) {
      const int pb = b / BM;
      if (pb != panel) {
        panel = pb;
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
          const int j = threadIdx.x + i * kNormThreads;
          if (j < nvec)
            panel_off[i] = static_cast<uint32_t>(reordered_offset(pb * BM, j * 8, dim, BM, BN, rldn, RA) >> 3);
        }
      }
      const uint4* row = reinterpret_cast<const uint4*>(X + static_cast<size_t>(b - pb * BM) * ld);
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int j = threadIdx.x + i * kNormThreads;
        if (j < nvec) dst[i] = __ldcs(row + panel_off[i]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int j = threadIdx.x + i * kNormThreads;
        if (j < nvec)
          dst[i] = __ldcs(reinterpret_cast<const uint4*>(X + static_cast<size_t>(b) * dim +
                                                         static_cast<size_t>(j) * 8));
      }
    }
  };

  uint4 cur[VPT];
  [[maybe_unused]] uint4 nxt[VPT];
  if constexpr (PREFETCH) load_row(row_begin, cur);
  for (int b = row_begin; b < row_end; ++b) {
    if constexpr (PREFETCH) {
      if (b + 1 < row_end) load_row(b + 1, nxt);
    } else {
      load_row(b, cur);
    }
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int j = threadIdx.x + i * kNormThreads;
      if (j < nvec) {
        const uint32_t* u = reinterpret_cast<const uint32_t*>(&cur[i]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 f = unpack2<BF16>(u[k]);
          ss += f.x * f.x + f.y * f.y;
        }
      }
    }
    ss = block_sum(ss, red);
    const float scale = rsqrtf(ss / static_cast<float>(dim) + eps);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int j = threadIdx.x + i * kNormThreads;
      if (j < nvec) {
        uint4 w;
        if constexpr (PREFETCH) {
          w = wv[i];
        } else {
          w = __ldg(reinterpret_cast<const uint4*>(W + static_cast<size_t>(j) * 8));
        }
        uint4 y;
        y.x = scale_mul2<BF16>(cur[i].x, w.x, scale);
        y.y = scale_mul2<BF16>(cur[i].y, w.y, scale);
        y.z = scale_mul2<BF16>(cur[i].z, w.z, scale);
        y.w = scale_mul2<BF16>(cur[i].w, w.w, scale);
        __stcs(reinterpret_cast<uint4*>(Y + static_cast<size_t>(b) * dim + static_cast<size_t>(j) * 8), y);
      }
    }
    if constexpr (PREFETCH) {
#pragma unroll
      for (int i = 0; i < VPT; ++i) cur[i] = nxt[i];
    }
  }
}

// H = round16(X + T), Y = rmsnorm(H) * W: the residual add in front of a norm, in the norm's pass over
// the rows (an add of its own reads two matrices and writes one, and the norm reads that again:
// 55 us for the two at 4096 x 8192, 46 us here for 268 MB, 5.8 TB/s).
// H may be X (the residual stream is updated in place) and Y may be X or H, so no pointer is
// restrict-qualified: a row is read into registers, a whole row ahead, before it is stored, and a
// thread stores H before Y.  Threads, rows per CTA and prefetch as in rmsnorm_kernel; the weights
// are re-read from L1 per row, their registers hold the second operand.
template <bool BF16, int VPT>
__global__ void __launch_bounds__(kNormThreads, (VPT <= 2 ? 4 : 2))
    add_rmsnorm_kernel(const uint16_t* X, const uint16_t* T, uint16_t* H, uint16_t* Y, const uint16_t* W, int rows,
                       int dim, float eps) {
  __shared__ float red[kNormThreads / 32];
  const int nvec = dim / 8;
  const int per_cta = (rows + gridDim.x - 1) / gridDim.x;
  const int row_begin = blockIdx.x * per_cta;
  const int row_end = min(rows, row_begin + per_cta);
  ptx::grid_launch_dependents();
  ptx::grid_wait();
  if (row_begin >= row_end) return;
  auto load_row = [&](int b, uint4 (&x)[VPT], uint4 (&t)[VPT]) {
    const size_t base = static_cast<size_t>(b) * dim;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int j = threadIdx.x + i * kNormThreads;
      if (j < nvec) {
        x[i] = __ldcs(reinterpret_cast<const uint4*>(X + base + static_cast<size_t>(j) * 8));
        t[i] = __ldcs(reinterpret_cast<const uint4*>(T + base + static_cast<size_t>(j) * 8));
      }
    }
  };
  uint4 x[VPT], t[VPT], h[VPT];
  load_row(row_begin, x, t);
  for (int b = row_begin; b < row_end; ++b) {
    const size_t base = static_cast<size_t>(b) * dim;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int j = threadIdx.x + i * kNormThreads;
      if (j < nvec) {
        h[i] = make_uint4(add2<BF16>(x[i].x, t[i].x), add2<BF16>(x[i].y, t[i].y),
                          add2<BF16>(x[i].z, t[i].z), add2<BF16>(x[i].w, t[i].w));
        const uint32_t* u = reinterpret_cast<const uint32_t*>(&h[i]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 f = unpack2<BF16>(u[k]);
          ss += f.x * f.x + f.y * f.y;
        }
      }
    }
    if (b + 1 < row_end) load_row(b + 1, x, t);
    ss = block_sum(ss, red);
    const float scale = rsqrtf(ss / static_cast<float>(dim) + eps);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int j = threadIdx.x + i * kNormThreads;
      if (j < nvec) {
        const uint4 w = __ldg(reinterpret_cast<const uint4*>(W + static_cast<size_t>(j) * 8));
        uint4 y;
        y.x = scale_mul2<BF16>(h[i].x, w.x, scale);
        y.y = scale_mul2<BF16>(h[i].y, w.y, scale);
        y.z = scale_mul2<BF16>(h[i].z, w.z, scale);
        y.w = scale_mul2<BF16>(h[i].w, w.w, scale);
        __stcs(reinterpret_cast<uint4*>(H + base + static_cast<size_t>(j) * 8), h[i]);
        __stcs(reinterpret_cast<uint4*>(Y + base + static_cast<size_t>(j) * 8), y);
      }
    }
  }
}

// TO_REORDERED: Y[reordered] = X[natural]; otherwise Y[natural] = X[reordered].
// Same shape as the norm kernel: each CTA takes a contiguous block of rows, each thread owns VPT
// 16-byte vectors of a row, the tile look-up through RA is done only when the block of rows
// crosses into another row panel, and two rows (2 * VPT vectors per thread) are in flight.
// (The first version walked the vectors with a grid stride and paid a 64-bit division and a
// dependent RA load per vector: 0.66 of the measured copy bandwidth.)
template <bool TO_REORDERED, int VPT>
__global__ void __launch_bounds__(kNormThreads, (VPT <= 2 ? 6 : (VPT <= 4 ? 4 : 2)))
    reorder_kernel(const uint16_t* __restrict__ X, uint16_t* __restrict__ Y, int rows, int dim,
                   int BM, int BN, int rldn, const int* __restrict__ RA) {
  const int nvec = dim / 8;
  const int per_cta = (rows + gridDim.x - 1) / gridDim.x;
  const int row_begin = blockIdx.x * per_cta;
  const int row_end = min(rows, row_begin + per_cta);
  ptx::grid_launch_dependents();
  ptx::grid_wait();
  if (row_begin >= row_end) return;
  const uint4* __restrict__ x = reinterpret_cast<const uint4*>(X);
  uint4* __restrict__ y = reinterpret_cast<uint4*>(Y);
  const size_t ldv = static_cast<size_t>(rldn) * BN / 8;  // row pitch of the reordered view, in vectors

  uint32_t panel_off[VPT];  // vector offset of (row 0 of the current panel, this thread's columns)
  int panel = -1;
  auto offsets = [&](int b, size_t (&nat)[VPT], size_t (&reo)[VPT]) {
    const int pb = b / BM;
    if (pb != panel) {
      panel = pb;
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int j = threadIdx.x + i * kNormThreads;
        if (j < nvec) panel_off[i] = static_cast<uint32_t>(reordered_offset(pb * BM, j * 8, dim, BM, BN, rldn, RA) >> 3);
      }
    }
    const size_t row_reo = static_cast<size_t>(b - pb * BM) * ldv;
    const size_t row_nat = static_cast<size_t>(b) * nvec;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      nat[i] = row_nat + threadIdx.x + i * kNormThreads;
      reo[i] = row_reo + panel_off[i];
    }
  };

  for (int b = row_begin; b < row_end; b += 2) {
    size_t nat0[VPT], reo0[VPT], nat1[VPT], reo1[VPT];
    uint4 v0[VPT], v1[VPT];
    const bool two = b + 1 < row_end;
    offsets(b, nat0, reo0);
    if (two) offsets(b + 1, nat1, reo1);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      if (threadIdx.x + i * kNormThreads < nvec) {
        v0[i] = __ldcs(x + (TO_REORDERED ? nat0[i] : reo0[i]));
        if (two) v1[i] = __ldcs(x + (TO_REORDERED ? nat1[i] : reo1[i]));
      }
    }
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      if (threadIdx.x + i * kNormThreads < nvec) {
        __stcs(y + (TO_REORDERED ? reo0[i] : nat0[i]), v0[i]);
        if (two) __stcs(y + (TO_REORDERED ? reo1[i] : nat1[i]), v1[i]);
      }
    }
  }
}

// Launch whose prologue may overlap the tail of the stream's previous kernel (the kernels call
// ptx::grid_wait before they touch memory): 49.3 -> 45.9 us for a reorder and its inverse over
// 4096 x 8192, 51.5 -> 50.2 us for the norm of 8192 x 8192.  A CTA that starts while its SM is still set up for a
// GEMM's 227 KB of shared memory finds 28 KB of L1 for its loads in flight (16384 x 8192 after a GEMM:
// 328 us the two, 321 us with the carve-out asked for here, 319 us without the early launch).
template <auto kernel, typename... Args>
cudaError_t launch_rows(int grid, cudaStream_t stream, Args... args) {
  // (per kernel and device, and the same whoever sets it)
  static bool carved[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 16 && !carved[dev]) {
    const cudaError_t e =
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxL1);
    if (e != cudaSuccess) return e;
    carved[dev] = true;
  }
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(kNormThreads, 1, 1);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  if (e != cudaSuccess) cudaGetLastError();  // reported to the caller, not left for the next one
  return e;
}

// Contiguous row blocks: enough CTAs to fill the machine several times over, yet a few rows per CTA
// so that the prefetch and the cached tile look-ups pay off.
int row_grid(int rows, int sm_count) {
  int grid = rows < sm_count * 8 ? rows : sm_count * 8;
  if (rows >= sm_count * 32) grid = (rows + 3) / 4 < sm_count * 16 ? (rows + 3) / 4 : sm_count * 16;
  return grid < 1 ? 1 : grid;
}

// The same with `per` rows per CTA (down to one while that leaves the machine short of CTAs).
int row_grid(int rows, int sm_count, int per) { return rows <= sm_count * 8 ? rows : (rows + per - 1) / per; }

// Blocks of rows for the norm without prefetch, whose CTAs take about as long as they have rows: the
// number of rows that leaves the least of the last wave idle (`resident` CTAs run at once).
// 11248 x 1024: 5 -> 21.9, 6 -> 19.7, 8 -> 22.6, 10 -> 26.2 us; 6784 x 640: 6 -> 15.8, 7 -> 11.6; 2608 x 16384: 1 -> 46, 5 -> 44,
// 6 -> 35, 8 -> 37.  Up to 8 rows (ten where a CTA has an SM's third); five at most for rows of
// 4097..8192 elements, four if that is as good (16384 x 8192: 4 -> 87, 5 -> 89, 8 -> 92).  One wave of
// up to 16 narrow rows if it is nearly full (16384 x 256: 8 -> 21.5, 16 -> 20.5; not so 13568 x 768: 7 -> 21.8, 14 -> 22.4).
int whole_wave_grid(int rows, int resident, int vpt, int dim) {
  const int single = (rows + resident - 1) / resident;
  if (dim <= 1024 && single > 8 && single <= 16 && rows >= 0.97 * single * resident) return (rows + single - 1) / single;
  const bool wide = vpt > 2 && vpt <= 4;
  // candidates, the preferred of equals first
  static constexpr int kWide[] = {4, 5, 3};
  const int first = vpt <= 2 ? 8 : 10, count = wide ? 3 : first;
  int best = 1;
  int64_t least = INT64_MAX;
  for (int i = 0; i < count; ++i) {
    const int per = wide ? kWide[i] : first - i;
    const int64_t ctas = (rows + per - 1) / per;
    const int64_t cost = (ctas + resident - 1) / resident * (wide ? per : per + 1);  // + 1: a wave's start
    if (cost < least) {
      least = cost;
      best = per;
    }
  }
  return (rows + best - 1) / best;
}

template <bool BF16>
cudaError_t launch_add_norm(const void* X, const void* T, void* H, void* Y, const void* W, int rows, int dim,
                            float eps, int sm_count, cudaStream_t stream) {
  const int vpt = (dim / 8 + kNormThreads - 1) / kNormThreads;
  const int grid = row_grid(rows, sm_count);
  const uint16_t* x = static_cast<const uint16_t*>(X);
  const uint16_t* t = static_cast<const uint16_t*>(T);
  uint16_t* h = static_cast<uint16_t*>(H);
  uint16_t* y = static_cast<uint16_t*>(Y);
  const uint16_t* w = static_cast<const uint16_t*>(W);
  if (vpt <= 1) {
    return launch_rows<add_rmsnorm_kernel<BF16, 1>>(grid, stream, x, t, h, y, w, rows, dim, eps);
  } else if (vpt <= 2) {
    return launch_rows<add_rmsnorm_kernel<BF16, 2>>(grid, stream, x, t, h, y, w, rows, dim, eps);
  } else if (vpt <= 4) {
    return launch_rows<add_rmsnorm_kernel<BF16, 4>>(grid, stream, x, t, h, y, w, rows, dim, eps);
  } else if (vpt <= 8) {
    return launch_rows<add_rmsnorm_kernel<BF16, 8>>(grid, stream, x, t, h, y, w, rows, dim, eps);
  }
  return cudaErrorInvalidValue;  // dim > 16384
}

template <bool BF16, bool REORDER>
cudaError_t launch_norm(const void* X, void* Y, const void* W, int rows, int dim, int BM, int BN,
                        int rldn, const int* RA, float eps, int sm_count, cudaStream_t stream) {
  const int nvec = dim / 8;
  const int vpt = (nvec + kNormThreads - 1) / kNormThreads;
  // Measured (us, rows per CTA -> time).  Row-major, 8192 x 8192: 2 -> 42.9, 4 -> 45.9, 8 -> 47.6, and the
  // same order at 4096 x 4096 and 8192 x 16384; rows of up to 2048 elements want more (16384 x 2048:
  // 2 -> 29.3, 7 -> 27.6).
  // Tile-contiguous: the build with prefetch up to where the other one has gained on it in every place
  // measured (cold, behind the input's producer, before the output's consumer): 20 rows per SM, 17
  // for rows over 4096 elements (2048 x 8192: 15.7 against 17.4 us; 2608 x 8192: 21.1 against 19.1 us),
  // 2 over 8192 (400 x 16384: 12.7 against 9.8 us).  Of fewer, narrow rows that nearly fill their last
  // wave are the other one's too (1008 x 1024: 3.5 against 3.0 us; 1408 x 1024, 0.68 of two waves: 3.8 against 4.1 us).
  const int wave = sm_count * norm_ctas_per_sm(vpt);
  bool prefetch = !REORDER || rows < sm_count * (vpt <= 2 ? 20 : (vpt <= 4 ? 17 : 2));
  if (REORDER && vpt <= 2 && rows >= 0.86 * wave * ((rows + wave - 1) / wave)) prefetch = false;
  int grid = row_grid(rows, sm_count);
  if (!prefetch) {
    grid = whole_wave_grid(rows, wave, vpt, dim);
  } else if (REORDER) {
    // two rows each as soon as one each takes more than a wave (1008 x 4608: 8.2 -> 6.9 us)
    const int resident = sm_count * (vpt <= 2 ? 6 : (vpt <= 4 ? 4 : 2));
    if (grid == rows && rows > resident) grid = (rows + 1) / 2;
  } else if (vpt > 1) {
    grid = row_grid(rows, sm_count, 2);
  }
  const uint16_t* x = static_cast<const uint16_t*>(X);
  uint16_t* y = static_cast<uint16_t*>(Y);
  const uint16_t* w = static_cast<const uint16_t*>(W);
#define FO_LAUNCH_NORM(V)                                                                                          \
  do {                                                                                                             \
    if constexpr (REORDER) {                                                                                       \
      if (!prefetch)                                                                                               \
        return launch_rows<rmsnorm_kernel<BF16, true, V, false>>(grid, stream, x, y, w, rows, dim, BM, BN, rldn, RA, eps); \
    }                                                                                                              \
    return launch_rows<rmsnorm_kernel<BF16, REORDER, V, true>>(grid, stream, x, y, w, rows, dim, BM, BN, rldn, RA, eps); \
  } while (0)
  if (vpt <= 1) {
    FO_LAUNCH_NORM(1);
  } else if (vpt <= 2) {
    FO_LAUNCH_NORM(2);
  } else if (vpt <= 4) {
    FO_LAUNCH_NORM(4);
  } else if (vpt <= 8) {
    FO_LAUNCH_NORM(8);
  }
#undef FO_LAUNCH_NORM
  return cudaErrorInvalidValue;  // dim > 16384
}

}  // namespace

// Every tensor here is read and written 16 bytes at a time.
template <typename... P>
static bool unaligned(P... p) {
  return ((reinterpret_cast<uintptr_t>(p) | ...) & 15) != 0;
}

cudaError_t rmsnorm_launch(const void* X, void* Y, const void* W, int rows, int dim, float eps,
                           bool bf16, int sm_count, cudaStream_t stream) {
  if (dim % 8 != 0 || (rows > 0 && unaligned(X, Y, W))) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  return bf16 ? launch_norm<true, false>(X, Y, W, rows, dim, 1, 1, 1, nullptr, eps, sm_count, stream)
              : launch_norm<false, false>(X, Y, W, rows, dim, 1, 1, 1, nullptr, eps, sm_count, stream);
}

cudaError_t add_rmsnorm_launch(const void* X, const void* T, void* H, void* Y, const void* W, int rows, int dim,
                               float eps, bool bf16, int sm_count, cudaStream_t stream) {
  if (dim % 8 != 0 || (rows > 0 && unaligned(X, T, H, Y, W))) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  return bf16 ? launch_add_norm<true>(X, T, H, Y, W, rows, dim, eps, sm_count, stream)
              : launch_add_norm<false>(X, T, H, Y, W, rows, dim, eps, sm_count, stream);
}

cudaError_t reorder_rmsnorm_launch(const void* X, void* Y, const void* W, int rows, int dim, int BM,
                                   int BN, int rldn, const int* RA, float eps, bool bf16,
                                   int sm_count, cudaStream_t stream) {
  if (dim % 8 != 0 || BN % 8 != 0 || dim % BN != 0 || rows % BM != 0 || rldn < 1 ||
      (rows > 0 && unaligned(X, Y, W)))
    return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  return bf16 ? launch_norm<true, true>(X, Y, W, rows, dim, BM, BN, rldn, RA, eps, sm_count, stream)
              : launch_norm<false, true>(X, Y, W, rows, dim, BM, BN, rldn, RA, eps, sm_count, stream);
}

cudaError_t reorder_launch(const void* X, void* Y, int rows, int dim, int BM, int BN, int rldn,
                           const int* RA, bool to_reordered, int sm_count, cudaStream_t stream) {
  if (dim % 8 != 0 || BN % 8 != 0 || dim % BN != 0 || rows % BM != 0 || rldn < 1 ||
      (rows > 0 && unaligned(X, Y)))
    return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  const int nvec = dim / 8;
  const int vpt = (nvec + kNormThreads - 1) / kNormThreads;
  // Four rows per CTA, two (what a thread has in flight) for fewer than 24 rows per SM of 2049..8192 elements:
  // cold, two would be better for any number of those (8192 x 4096: 2 -> 22.1, 4 -> 23.2 us), but not where a
  // kernel has just written the input and part of it is in the L2 (the two kernels: 2 -> 39.6, 4 -> 37.2 us;
  // 4096 x 8192: 42.2 and 40.5; 2608 x 8192: 28.7 and 28.1).  Narrow rows and rows that fill the registers want four
  // either way (16384 x 512: 2 -> 15.6, 4 -> 13.2; 8192 x 16384: 106 and 93.4).
  const int grid = row_grid(rows, sm_count, vpt == 1 || vpt > 4 || rows >= sm_count * 24 ? 4 : 2);
  const uint16_t* x = static_cast<const uint16_t*>(X);
  uint16_t* y = static_cast<uint16_t*>(Y);
#define FO_LAUNCH_REORDER(V)                                                                              \
  do {                                                                                                    \
    if (to_reordered) {                                                                                   \
      return launch_rows<reorder_kernel<true, V>>(grid, stream, x, y, rows, dim, BM, BN, rldn, RA);           \
    } else {                                                                                              \
      return launch_rows<reorder_kernel<false, V>>(grid, stream, x, y, rows, dim, BM, BN, rldn, RA);          \
    }                                                                                                     \
  } while (0)
  if (vpt <= 1) {
    FO_LAUNCH_REORDER(1);
  } else if (vpt <= 2) {
    FO_LAUNCH_REORDER(2);
  } else if (vpt <= 4) {
    FO_LAUNCH_REORDER(4);
  } else if (vpt <= 8) {
    FO_LAUNCH_REORDER(8);
  }
#undef FO_LAUNCH_REORDER
  return cudaErrorInvalidValue;  // dim > 16384
}

}  // namespace fo
