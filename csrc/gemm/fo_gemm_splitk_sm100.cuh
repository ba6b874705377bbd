// tcgen05 GEMM of few output tiles for B200 (sm_100a), split over K inside a cluster:
// C = A * B^T written row-major or tile-contiguous, without a collective, counters or monitoring.
//
// With one CTA per 128 x BN tile a decode batch (M = 128) or a narrow projection leaves most SMs
// idle: 128 x 8192 x 3584 is 32 tiles of 128 x 256 on 148 SMs, and one SM takes in 100 - 140 GB/s of
// operands, so reading 59 MB of weights took 23 us.  Here the S CTAs of a cluster share one 128 x 128
// tile: CTA s multiplies k-blocks [s * kb / S, (s + 1) * kb / S), sends its fp32 partial sums of the
// columns that CTA d finishes, [d * 128 / S, (d + 1) * 128 / S), straight from TMEM into d's shared memory,
// and after a cluster barrier adds up the S partials of its own columns.  The sums are fp32 and are
// added in the order of the ranks, so results do not depend on timing; no workspace, no second
// launch.
//
// The exchange is what a split costs: distributed shared memory moves about 14 bytes a cycle and SM,
// so 32 KB (S = 2) take 2,300 cycles and the 96 KB of 128 x 256 tiles split in four took 7,600.  Hence
// narrow tiles, small splits, a receive buffer of its own (sends need not wait for the receiver's
// ring) and stores rather than loads.  128 x 8192 x 3584: 25.2 us on 128 x 256 tiles, 16.6 us on 128 x 128
// tiles, 14.4 us with those split in two (16.5 us in four where that needs two waves of clusters), of
// which the weights' way through HBM takes 9 us; 128 x 1024 x 28672: 153 us, 19.4 us split in eight.
//
// Roles as in fo_gemm_plain_sm100.cuh (warp 0 TMA producer, warp 1 MMA issuer, warps 2-9
// epilogue); one tile per cluster, so nothing is persistent and TMEM holds one accumulator.
#pragma once
#include "fo_gemm.h"
#include "fo_gemm_device.cuh"

namespace fo {

constexpr int kSplitThreads = 64 + 256;

struct SplitTensorMaps {
  CUtensorMap a, b;
};

constexpr int kSplitStages = 5;

template <int S>
struct SplitSmem {
  static constexpr int kABytes = kBM * kBK * 2;
  static constexpr int kBBytes = kSplitBN * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  // Partial sums from the other CTAs: [S - 1 senders][own columns / 4][128 rows] x 16 bytes;
  // consecutive lanes (rows) take consecutive vectors.
  static constexpr int kRecvOffset = kSplitStages * kStageBytes;
  static constexpr int kOwnCols = kSplitBN / S;
  static constexpr int kSlotBytes = kOwnCols * kBM * 4;
  static constexpr int kBarOffset = kRecvOffset + (S - 1) * kSlotBytes;
  static constexpr int kNumBars = 2 * kSplitStages + 1;
  static constexpr int kMiscOffset = kBarOffset + kNumBars * 8;
  static constexpr int kTotalBytes = kMiscOffset + 16 + 1024;
};

template <bool BF16, int S>
__global__ void __launch_bounds__(kSplitThreads, 1)
    fo_gemm_splitk_kernel(const __grid_constant__ SplitTensorMaps maps, const __grid_constant__ GemmParams p) {
  using L = SplitSmem<S>;
  constexpr int BN = kSplitBN, STAGES = kSplitStages;
  constexpr int kOwnCols = L::kOwnCols;  // columns whose sum this CTA finishes
  // columns of one warpgroup: half of them, or all (the other idles) when half is below 16
  constexpr int kWgCols = kOwnCols >= 32 ? kOwnCols / 2 : kOwnCols;
  static_assert(kOwnCols % 16 == 0, "columns are summed 16 at a time");
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = ptx::smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kBarOffset);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full_bar = full_bar + 2 * STAGES;
  uint32_t* misc = reinterpret_cast<uint32_t*>(smem + L::kMiscOffset);
  uint32_t* s_tmem_base = misc;
  volatile int* s_abort = reinterpret_cast<volatile int*>(misc + 1);
  volatile uint32_t* s_peer_failed = misc + 2;  // set by a CTA of the cluster that sent nothing

  const int warp_idx = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(ptx::cluster_ctarank());
  const int pos = static_cast<int>(blockIdx.x) / S;
  const TileCoord tc = tile_of_position(pos, p.tiles_m, p.tiles_n, p.raster_sw);
  const int num_kb = (p.K + kBK - 1) / kBK;
  const int kb_begin = num_kb * rank / S;
  const int kb_end = num_kb * (rank + 1) / S;
  int32_t* status = p.status[0];
  const uint64_t pipe_timeout = 4ull * p.timeout_ns + 1000000000ull;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) {
      ptx::mbar_init(&full_bar[i], 1);
      ptx::mbar_init(&empty_bar[i], 1);
    }
    ptx::mbar_init(tmem_full_bar, 1);
    *s_abort = 0;
    *s_peer_failed = 0;
    ptx::mbar_fence_init();
  }
  if (warp_idx == 0 && lane == 0) {
    ptx::prefetch_tmap(&maps.a);
    ptx::prefetch_tmap(&maps.b);
  }
  if (warp_idx == 1) {
    ptx::tmem_alloc(s_tmem_base, BN);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  // First phase of the cluster barrier: every CTA runs and has cleared its failure word before
  // anybody stores into its shared memory.  The epilogue waits for it ahead of its sends.
  ptx::cluster_arrive_release();
  const uint32_t tmem_base = *s_tmem_base;
  ptx::grid_launch_dependents();
  ptx::grid_wait();

  const int ew = warp_idx - 2;
  const int wg = ew >> 2;
  const int quad = warp_idx & 3;  // TMEM lane quadrant this warp may read
  const int row = quad * 32 + lane;
  const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);

  if (warp_idx == 0) {
    // ------------------------------------------------------------------ TMA producer
    const bool elected = ptx::elect_one();
    int stage = 0;
    uint32_t phase = 0;
    uint32_t issued = 0;
    for (int kb = kb_begin; kb < kb_end; ++kb) {
      if (!ptx::mbar_wait_bounded(&empty_bar[stage], phase ^ 1u, s_abort, pipe_timeout, p.wait_sleep_ns)) {
        if (elected) ptx::report_status(status, kStatusTimeoutSmemEmpty, pos, kb, stage);
        *s_abort = 1;
        break;
      }
      if (elected) {
        uint8_t* sa = smem + stage * L::kStageBytes;
        ptx::mbar_arrive_expect_tx(&full_bar[stage], L::kStageBytes);
        ptx::tma_load_2d(sa + L::kABytes, &maps.b, &full_bar[stage], kb * kBK, tc.n * BN, p.l2_hint_b);
        ptx::tma_load_2d(sa, &maps.a, &full_bar[stage], kb * kBK, tc.m * kBM, p.l2_hint_a);
      }
      __syncwarp();
      ++issued;
      if (++stage == STAGES) {
        stage = 0;
        phase ^= 1u;
      }
    }
    // Drain: no bulk copy may still write this CTA's shared memory when it leaves (bounded).
    for (int s = 0; elected && s < STAGES; ++s) {
      if (issued <= static_cast<uint32_t>(s)) continue;
      const uint32_t par = ((issued - 1 - s) / STAGES) & 1u;
      for (uint32_t it = 0; it < ptx::kMbarDrainPolls; ++it) {
        if (ptx::mbar_try_wait(&full_bar[s], par)) break;
      }
    }
    __syncwarp();
  } else if (warp_idx == 1) {
    // ------------------------------------------------------------------ MMA issuer
    const bool elected = ptx::elect_one();
    constexpr uint32_t idesc = ptx::make_idesc_f16(BF16, kBM, BN);
    int stage = 0;
    uint32_t phase = 0;
    bool go = true;
    for (int kb = kb_begin; kb < kb_end; ++kb) {
      if (!ptx::mbar_wait_bounded(&full_bar[stage], phase, s_abort, pipe_timeout, p.wait_sleep_ns)) {
        if (elected) ptx::report_status(status, kStatusTimeoutSmemFull, pos, kb, stage);
        *s_abort = 1;
        go = false;
        break;
      }
      ptx::tc_fence_after_sync();
      const uint32_t sa = ptx::smem_u32(smem + stage * L::kStageBytes);
      const uint64_t da = ptx::make_smem_desc_sw128_kmajor(sa);
      const uint64_t db = ptx::make_smem_desc_sw128_kmajor(sa + L::kABytes);
      if (elected) {
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k) {
          ptx::umma_f16_ss(tmem_base, da + static_cast<uint64_t>(2 * k), db + static_cast<uint64_t>(2 * k), idesc,
                           (kb > kb_begin || k > 0) ? 1u : 0u);
        }
        ptx::umma_commit(&empty_bar[stage]);
      }
      __syncwarp();
      if (++stage == STAGES) {
        stage = 0;
        phase ^= 1u;
      }
    }
    if (go && elected) ptx::umma_commit(tmem_full_bar);
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue, first half
    const bool ok = __all_sync(0xffffffffu, ptx::mbar_wait_bounded(tmem_full_bar, 0, s_abort, pipe_timeout,
                                                                   4u * p.wait_sleep_ns));
    if (!ok && lane == 0) {
      ptx::report_status(status, kStatusTimeoutTmemFull, pos, 0, 0);
      *s_abort = 1;
    }
    __syncwarp();  // the barrier's aligned form takes whole warps
    ptx::tc_fence_after_sync();
    ptx::cluster_wait_acquire();
    if (ok) {
      // Columns that other CTAs finish go to their receive buffers.
#pragma unroll
      for (int c = wg * 32; c < BN; c += 64) {
        uint32_t v[32];
        ptx::tmem_ld_32x32b_x32(t_row + c, v);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c0 = c + 16 * h;
          const int d = c0 / kOwnCols;  // CTA that finishes these columns
          if (d == rank) continue;
          const int slot = rank < d ? rank : rank - 1;
          const uint32_t dst = ptx::mapa_shared(ptx::smem_u32(smem + L::kRecvOffset), d) +
                               ((slot * kOwnCols + c0 - d * kOwnCols) / 4 * kBM + row) * 16;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int b = 16 * h + 4 * j;
            ptx::st_shared_cluster_v4(dst + j * kBM * 16, v[b], v[b + 1], v[b + 2], v[b + 3]);
          }
        }
      }
    } else if (lane < S) {
      ptx::st_shared_cluster_u32(ptx::mapa_shared(ptx::smem_u32(misc + 2), lane), 1u);
    }
  }
  __syncwarp();
  if (warp_idx < 2) ptx::cluster_wait_acquire();

  // Every CTA's partial sums have arrived (release / acquire at cluster scope).
  ptx::cluster_arrive_release();
  ptx::cluster_wait_acquire();

  if (warp_idx >= 2) {
    // ------------------------------------------------------------------ epilogue, second half
    // (A CTA that gave up sent nothing: nobody in the cluster stores, the status says why.)
    if (*s_peer_failed == 0 && (kOwnCols >= 32 || wg == 0)) {
      const int n0 = tc.n * BN;
      size_t off;  // element offset of (this row, tile column 0)
      if (p.out_mode == kOutNatural) {
        off = (static_cast<size_t>(tc.m) * kBM + row) * p.N + n0;
      } else {
        const int r = tile_position(p, tc.m * (p.N / p.out_bn) + n0 / p.out_bn, status);
        const size_t ld = static_cast<size_t>(p.rldn) * p.out_bn;
        off = (static_cast<size_t>(r / p.rldn) * kBM + row) * ld + static_cast<size_t>(r % p.rldn) * p.out_bn +
              n0 % p.out_bn;
      }
      uint8_t* out = reinterpret_cast<uint8_t*>(p.out[0]);
#pragma unroll
      for (int i = 0; i < kWgCols; i += 16) {
        const int oc = (kOwnCols >= 32 ? wg * kWgCols : 0) + i;  // among the own columns
        const int c = rank * kOwnCols + oc;                      // in the tile
        uint32_t own[16];
        ptx::tmem_ld_32x32b_x16(t_row + c, own);
        ptx::tmem_ld_wait();
        float a[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) a[j] = 0.f;
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const int slot = s < rank ? s : s - 1;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float4 x;
            if (s == rank) {
              x = make_float4(__uint_as_float(own[4 * j]), __uint_as_float(own[4 * j + 1]),
                              __uint_as_float(own[4 * j + 2]), __uint_as_float(own[4 * j + 3]));
            } else {
              x = *reinterpret_cast<const float4*>(smem + L::kRecvOffset +
                                                   (((slot * kOwnCols + oc) / 4 + j) * kBM + row) * 16);
            }
            a[4 * j + 0] += x.x;
            a[4 * j + 1] += x.y;
            a[4 * j + 2] += x.z;
            a[4 * j + 3] += x.w;
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint4 w;
          w.x = pack2<BF16>(a[8 * h + 0], a[8 * h + 1]);
          w.y = pack2<BF16>(a[8 * h + 2], a[8 * h + 3]);
          w.z = pack2<BF16>(a[8 * h + 4], a[8 * h + 5]);
          w.w = pack2<BF16>(a[8 * h + 6], a[8 * h + 7]);
          if (p.res != nullptr) {  // residual, laid out like the row-major output (which it may be)
            const uint4 r = ptx::ld_cg_v4(reinterpret_cast<const uint8_t*>(p.res) + (off + c + 8 * h) * 2);
            w = make_uint4(add2<BF16>(w.x, r.x), add2<BF16>(w.y, r.y), add2<BF16>(w.z, r.z), add2<BF16>(w.w, r.w));
          }
          ptx::st_v4(out + (off + c + 8 * h) * 2, w);
        }
      }
    }
  }

  // Nobody stores into another CTA's shared memory after the barrier: each leaves by itself.
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp_idx == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, BN);
  }
}

}  // namespace fo
