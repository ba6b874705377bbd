// Persistent, warp-specialised tcgen05 GEMM for B200 (sm_100a) without a collective inside:
// C = A * B^T written row-major, tile-contiguous ("reordered") or row-scattered, optionally
// announcing finished tiles (the producer half of the counter-gated NCCL path, reference:
// src/overlap/gemm_with_signal.h:210-256, :338-361) and recording their completion order.
// The fused GEMM + collective kernels live in fo_gemm_sm100.cuh.
//
// Roles inside a CTA (one CTA per SM, 128 x BN output tiles, BK = 64):
//   warp 0      TMA producer: 2-D tiled loads (128-byte swizzle, one CTA per copy) into a
//               STAGES-deep shared-memory ring, completion counted on mbarriers;
//   warp 1      MMA issuer: tcgen05.mma.kind::f16 (fp32 accumulate in TMEM), tcgen05.commit
//               releases ring slots and publishes finished accumulators; owns the TMEM allocation;
//   warps 2-9   epilogue: tcgen05.ld -> convert -> swizzled shared memory -> TMA tensor store (or
//               128-byte coalesced stores).
// Warps 0 and 1 walk their loops with all lanes and a lane chosen by elect.sync issues, so that
// counters, addresses and descriptors stay in uniform registers.
//
// CTA2: two CTAs of a cluster share one 256-row tile through tcgen05.mma.cta_group::2, each
// loading its own 128 rows of A and its own half of the B tile.  MT = 2 (with CTA2): each CTA owns
// two 128-row halves that share its B tile (512 x 256 per pair); the two accumulators fill TMEM,
// so a tile's epilogue is not hidden behind the next main loop.
//
// Epilogue.  Eight warps, each on its own: a warp owns 32 rows (its TMEM lane quadrant) of every
// second 64-column chunk of the tile (MT = 2: of every chunk of one half), and a 4 KB buffer that
// it transposes through and stores from with a 32 x 64 tensor store of its own.  No barrier spans
// warps, so a warp that waits for its buffer's previous store does not hold the others up.  Four
// warps that handed 128 x 64 chunks over at CTA barriers took 4,100 cycles for a 128 x 256 tile by
// itself and 5,700-7,000 under a running main loop; now 2,800 from the complete accumulator to the
// last store landed, and the hand-back of the accumulator no longer waits for global stores.
// Launches of one 128 x 256 tile per SM (1024 x 4096 x 1024): 10.9 -> 10.0 us, CTA pairs
// 11.5 -> 10.2 us; 256 x 256 per CTA, whose epilogue is exposed at every tile: 17.4 -> 15.3 us, and
// 229 -> 200 us at 16384 x 8192 x 1024.
//
// Last wave.  With CTA pairs on 256-wide tiles the tiles left over after the last full wave are computed
// as 256 x 128 halves when those fit one wave (tail_start): the wave then takes 0.64 of a full one.
// 1920 x 5376 x 1000 (168 units on 74 pairs): 26.2 -> 24.2 us; projection + residual + norm of
// 2048 x 8192 x 1792 (256 units): 76.7 -> 75.1 us a call.
//
// Every wait is bounded: on expiry the role records a status code, raises a CTA-wide abort
// flag, the producer drains its TMA loads in flight, TMEM is freed and the kernel returns.
#pragma once
#include "fo_gemm_device.cuh"

namespace fo {

constexpr int kPlainEpilogueWarps = 8;
constexpr int kPlainThreads = 64 + 32 * kPlainEpilogueWarps;

// The tensor maps of one launch: operands, and the output when it can be described as a 2-D
// tensor (GemmParams::tma_out), box 32 x 64.
struct PlainTensorMaps {
  CUtensorMap a, b, st;
  CUtensorMap b_half;  // half-width tiles of the last wave (GemmParams::tail_start): boxes of half of b's rows
};

template <int BN, int STAGES, bool CTA2 = false, int MT = 1>
struct PlainSmem {
  static constexpr int kAHalfBytes = kBM * kBK * 2;
  static constexpr int kABytes = MT * kAHalfBytes;
  static constexpr int kBRows = CTA2 ? BN / 2 : BN;  // B rows this CTA loads per k-block
  static constexpr int kBBytes = kBRows * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kWarpBufBytes = 32 * 128;  // 32 rows x 64 16-bit columns
  static constexpr int kEpiOffset = STAGES * kStageBytes;
  static constexpr int kBarOffset = kEpiOffset + kPlainEpilogueWarps * kWarpBufBytes;
  static constexpr int kNumBars = 2 * STAGES + 4;
  static constexpr int kMiscOffset = kBarOffset + kNumBars * 8;
  // +1024: the ring is aligned up to 1024 B at run time (128-byte swizzle atom).
  static constexpr int kTotalBytes = kMiscOffset + 16 + 1024;
};

template <bool BF16>
__device__ __forceinline__ uint4 add8(const uint4& a, const uint4& b) {
  return make_uint4(add2<BF16>(a.x, b.x), add2<BF16>(a.y, b.y), add2<BF16>(a.z, b.z), add2<BF16>(a.w, b.w));
}

// On the fp32 accumulators: nothing is rounded before the product is (the element-wise kernel, which reads
// gate and up in 16 bits, also rounds silu, as two operators in a row do).
__device__ __forceinline__ float silu_mul(uint32_t g, uint32_t u) {
  return silu(__uint_as_float(g)) * __uint_as_float(u);
}

template <int BN, int STAGES, bool BF16, bool CTA2, int MT, int EPI>
__global__ void __launch_bounds__(kPlainThreads, 1)
    fo_gemm_plain_kernel(const __grid_constant__ PlainTensorMaps maps, const __grid_constant__ GemmParams p) {
  static_assert(MT == 1 || (MT == 2 && CTA2 && BN == 256), "two row halves need CTA pairs and BN = 256");
  static_assert(EPI != kEpiSwiGLU || (CTA2 && MT == 1 && BN == 256), "the two CTAs of a pair load the two halves of B");
  using L = PlainSmem<BN, STAGES, CTA2, MT>;
  constexpr int kOutCols = EPI == kEpiSwiGLU ? BN / 2 : BN;  // output columns of a tile
  // Accumulator slots in TMEM: two tiles in flight (MT = 1) or the two halves of one (MT = 2).
  constexpr int kAccStages = MT == 2 ? 1 : 2;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = ptx::smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);

  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kBarOffset);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full_bar = full_bar + 2 * STAGES;
  uint64_t* tmem_empty_bar = full_bar + 2 * STAGES + 2;
  uint32_t* misc = reinterpret_cast<uint32_t*>(smem + L::kMiscOffset);
  uint32_t* s_tmem_base = misc;  // written by tcgen05.alloc
  volatile int* s_abort = reinterpret_cast<volatile int*>(misc + 1);

  // broadcast from lane 0: tells the compiler that the role index is warp-uniform
  const int warp_idx = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int num_kb = (p.K + kBK - 1) / kBK;
  constexpr uint32_t kTmemCols = 2 * BN;
  // Scheduling unit: a CTA (128-row tiles) or a CTA pair (256 or 512 rows, this CTA's part).
  const uint32_t cta_rank = CTA2 ? ptx::cluster_ctarank() : 0u;
  const bool leader = cta_rank == 0u;
  const int unit = CTA2 ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
  const int num_units = CTA2 ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);
  constexpr int kRowsPerUnit = (CTA2 ? 2 : 1) * MT;  // 128-row tiles of one scheduling unit
  // A launch may have fewer row tiles than its units cover (an odd tiles_m under CTA pairs): the TMA
  // loads of the missing rows return zeros and their tiles are not stored.
  const int sched_tiles_m = (p.tiles_m + kRowsPerUnit - 1) / kRowsPerUnit;
  const int sched_tiles = sched_tiles_m * p.tiles_n;
  // Positions from tail_start on are two half-width tiles each, side by side in the schedule.
  constexpr bool kHalves = CTA2 && MT == 1 && BN == 256;
  const int sched_len = kHalves ? 2 * sched_tiles - p.tail_start : sched_tiles;
  struct Work {
    TileCoord tc;
    bool narrow;  // BN / 2 columns from n0
    int n0;       // first output column
  };
  auto my_tile = [&](int i) {
    Work w;
    w.narrow = kHalves && i >= p.tail_start;
    const int pos = w.narrow ? p.tail_start + (i - p.tail_start) / 2 : i;
    w.tc = tile_of_position(pos, sched_tiles_m, p.tiles_n, p.raster_sw);
    w.tc.m = kRowsPerUnit * w.tc.m + MT * static_cast<int>(cta_rank);  // first half; halves follow
    w.n0 = w.tc.n * kOutCols + (w.narrow ? ((i - p.tail_start) & 1) * (kOutCols / 2) : 0);
    return w;
  };
  int32_t* status = p.status[0];
  const uint64_t pipe_timeout = 4ull * p.timeout_ns + 1000000000ull;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) {
      ptx::mbar_init(&full_bar[i], 1);
      ptx::mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&tmem_full_bar[i], 1);
      // one arrival per epilogue warp, from both CTAs of a pair
      ptx::mbar_init(&tmem_empty_bar[i], (CTA2 ? 2 : 1) * kPlainEpilogueWarps);
    }
    *s_abort = 0;
    ptx::mbar_fence_init();
  }
  if (warp_idx == 0 && lane == 0) {
    ptx::prefetch_tmap(&maps.a);
    ptx::prefetch_tmap(&maps.b);
  }
  if (warp_idx == 2 && lane == 0 && p.tma_out != 0) ptx::prefetch_tmap(&maps.st);
  if (warp_idx == 1) {
    if constexpr (CTA2) {
      ptx::tmem_alloc_pair(s_tmem_base, kTmemCols);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(s_tmem_base, kTmemCols);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before_sync();
  if constexpr (CTA2) {
    // Both CTAs' barriers must be initialised before either receives a remote signal.  The release
    // form, since this is also what hands s_tmem_base and s_abort to the other warps (no store is in
    // flight yet that it would wait for).
    ptx::cluster_arrive_release();
    ptx::cluster_wait_acquire();
  } else {
    __syncthreads();
  }
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *s_tmem_base;
  ptx::grid_launch_dependents();
  ptx::grid_wait();

  if (warp_idx == 0) {
    // ------------------------------------------------------------------ TMA producer
    const bool elected = ptx::elect_one();
    int stage = 0;
    uint32_t phase = 0;
    uint32_t issued = 0;
    bool ok = true;
    for (int pos = unit; ok && pos < sched_len; pos += num_units) {
      const Work work = my_tile(pos);
      const TileCoord tc = work.tc;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!ptx::mbar_wait_bounded(&empty_bar[stage], phase ^ 1u, s_abort, pipe_timeout, p.wait_sleep_ns)) {
          if (elected) ptx::report_status(status, kStatusTimeoutSmemEmpty, pos, kb, stage);
          *s_abort = 1;
          ok = false;
          break;
        }
        uint8_t* sa = smem + stage * L::kStageBytes;
        uint8_t* sb = sa + L::kABytes;
        if (elected) {
          if constexpr (CTA2) {
            // The leader's barrier collects the bytes of both CTAs.
            if (leader) {
              ptx::mbar_arrive_expect_tx(&full_bar[stage],
                                         2 * (work.narrow ? L::kStageBytes - L::kBBytes / 2 : L::kStageBytes));
            }
#pragma unroll
            for (int h = 0; h < MT; ++h) {
              ptx::tma_load_2d_pair(sa + h * L::kAHalfBytes, &maps.a, &full_bar[stage], kb * kBK, (tc.m + h) * kBM,
                                    p.l2_hint_a);
            }
            // SwiGLU: the leader loads 128 rows of G, the follower the same rows of U, and so the tile's
            // accumulators hold the 128 gate columns and then the 128 up columns.
            const int rank = static_cast<int>(cta_rank);
            if (kHalves && work.narrow) {
              const int b_row = EPI == kEpiSwiGLU ? rank * p.N + work.n0 : work.n0 + rank * (L::kBRows / 2);
              ptx::tma_load_2d_pair(sb, &maps.b_half, &full_bar[stage], kb * kBK, b_row, p.l2_hint_b);
            } else {
              const int b_row = EPI == kEpiSwiGLU ? rank * p.N + work.n0 : work.n0 + rank * L::kBRows;
              ptx::tma_load_2d_pair(sb, &maps.b, &full_bar[stage], kb * kBK, b_row, p.l2_hint_b);
            }
          } else {
            ptx::mbar_arrive_expect_tx(&full_bar[stage], L::kStageBytes);
            ptx::tma_load_2d(sa, &maps.a, &full_bar[stage], kb * kBK, tc.m * kBM, p.l2_hint_a);
            ptx::tma_load_2d(sb, &maps.b, &full_bar[stage], kb * kBK, tc.n * BN, p.l2_hint_b);
          }
        }
        __syncwarp();
        ++issued;
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    // Drain: do not leave the CTA while a bulk copy may still write its shared memory.
    // For each ring slot wait (bounded) for the last load issued into it.
    // (In a pair the follower's loads are counted on the leader's barriers, which the
    // follower cannot poll; it relies on the cluster-wide barrier at the end instead: the
    // leader reaches it only after draining the barriers that count both CTAs' bytes.)
    for (int s = 0; elected && s < STAGES && (!CTA2 || leader); ++s) {
      if (issued <= static_cast<uint32_t>(s)) continue;
      const uint32_t last = ((issued - 1 - s) / STAGES) * STAGES + s;  // last issue index on slot s
      const uint32_t par = (last / STAGES) & 1u;
      for (uint32_t it = 0; it < ptx::kMbarDrainPolls; ++it) {
        if (ptx::mbar_try_wait(&full_bar[s], par)) break;
      }
    }
  } else if (warp_idx == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (leader) {
      const bool elected = ptx::elect_one();
      constexpr uint32_t idesc_full = ptx::make_idesc_f16(BF16, CTA2 ? 2 * kBM : kBM, BN);
      constexpr uint32_t idesc_half = ptx::make_idesc_f16(BF16, CTA2 ? 2 * kBM : kBM, BN / 2);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int pos = unit; ok && pos < sched_len; pos += num_units) {
        if (!ptx::mbar_wait_bounded(&tmem_empty_bar[acc], acc_phase ^ 1u, s_abort, pipe_timeout, p.wait_sleep_ns)) {
          if (elected) ptx::report_status(status, kStatusTimeoutTmemEmpty, pos, acc, 0);
          *s_abort = 1;
          break;
        }
        ptx::tc_fence_after_sync();
        const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(acc * BN);
        const uint32_t idesc = kHalves && pos >= p.tail_start ? idesc_half : idesc_full;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!ptx::mbar_wait_bounded(&full_bar[stage], phase, s_abort, pipe_timeout, p.wait_sleep_ns)) {
            if (elected) ptx::report_status(status, kStatusTimeoutSmemFull, pos, kb, stage);
            *s_abort = 1;
            ok = false;
            break;
          }
          ptx::tc_fence_after_sync();
          const uint32_t sa = ptx::smem_u32(smem + stage * L::kStageBytes);
          const uint64_t da = ptx::make_smem_desc_sw128_kmajor(sa);
          const uint64_t db = ptx::make_smem_desc_sw128_kmajor(sa + L::kABytes);
          if (elected) {
            // advance 16 elements (32 B) along K inside the swizzle atom: +2 in 16-byte units
            if constexpr (CTA2) {
#pragma unroll
              for (int h = 0; h < MT; ++h) {
                // half h: its A rows sit h * 16 KB further in the stage, its accumulator BN
                // columns further in TMEM; both halves multiply the same B tile.  The four MMAs
                // of a half are issued back to back so that consecutive instructions accumulate
                // into the same TMEM columns.
#pragma unroll
                for (int k = 0; k < kBK / 16; ++k) {
                  ptx::umma_f16_ss_pair(tmem_d + static_cast<uint32_t>(h * BN),
                                        da + static_cast<uint64_t>(h * (L::kAHalfBytes >> 4) + 2 * k),
                                        db + static_cast<uint64_t>(2 * k), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                }
              }
              ptx::umma_commit_pair(&empty_bar[stage], 3);  // slot reusable in both CTAs
            } else {
#pragma unroll
              for (int k = 0; k < kBK / 16; ++k) {
                ptx::umma_f16_ss(tmem_d, da + static_cast<uint64_t>(2 * k), db + static_cast<uint64_t>(2 * k), idesc,
                                 (kb > 0 || k > 0) ? 1u : 0u);
              }
              ptx::umma_commit(&empty_bar[stage]);
            }
          }
          __syncwarp();
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) break;
        if (elected) {
          if constexpr (CTA2) {
            ptx::umma_commit_pair(&tmem_full_bar[acc], 3);  // accumulators complete in both CTAs
          } else {
            ptx::umma_commit(&tmem_full_bar[acc]);
          }
        }
        __syncwarp();
        if (++acc == kAccStages) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int ew = warp_idx - 2;
    const int wg = ew >> 2;         // warpgroup: every second chunk (MT = 1) or one half (MT = 2)
    const int quad = warp_idx & 3;  // TMEM lane quadrant this warp may read
    uint8_t* buf = smem + L::kEpiOffset + ew * L::kWarpBufBytes;
    // Threads that together finish a 128-row tile: both warpgroups, or one per half.
    constexpr uint32_t kTileThreads = MT == 2 ? 128 : 256;
    const uint32_t tile_bar = MT == 2 ? 1u + wg : 1u;
    const bool first = MT == 2 ? (ew & 3) == 0 : ew == 0;  // warp that announces a finished tile
    const bool use_tma = p.tma_out != 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    // tmem_empty lives in the leader CTA of a pair
    const uint32_t tmem_empty_addr0 =
        CTA2 ? ptx::mapa_shared(ptx::smem_u32(&tmem_empty_bar[0]), 0u) : ptx::smem_u32(&tmem_empty_bar[0]);

    for (int pos = unit; pos < sched_len; pos += num_units) {
      const Work work = my_tile(pos);
      TileCoord tc = work.tc;
      if constexpr (MT == 2) tc.m += wg;
      const bool exists = tc.m < p.tiles_m;
      // tile of the layout that holds this one: the same, or (out_bn > BN) a wider one
      const int n0 = work.n0;
      const int out_cols = kHalves && work.narrow ? kOutCols / 2 : kOutCols;
      const int chunks = out_cols / 64;
      const int t = tc.m * (p.N / p.out_bn) + n0 / p.out_bn;
      const int r = exists ? tile_position(p, t, status) : 0;

      // Where the tile goes.  TMA stores: coordinates of the warp's first chunk in the output's 2-D
      // view.  Per-thread stores: lane l stores the 16-byte piece (l & 7) of the warp's rows
      // (l >> 3) + 4 * i, i = 0..7.
      int tma_x0 = 0, tma_y0 = 0;
      uint8_t* row_ptr[8];
      uint32_t row_valid = 0xffu;  // bit i clear: row i has no destination
      if (!exists) {
        row_valid = 0;
      } else if (use_tma) {
        if (p.out_mode == kOutNatural) {
          tma_x0 = n0;
          tma_y0 = tc.m * kBM + quad * 32;
        } else {  // tile-contiguous: [M * N / (rldn * out_bn)] rows of rldn * out_bn elements
          tma_x0 = (r % p.rldn) * p.out_bn + n0 % p.out_bn;
          tma_y0 = (r / p.rldn) * kBM + quad * 32;
        }
      } else {
        uint8_t* base = reinterpret_cast<uint8_t*>(p.out[0]) + (lane & 7) * 16;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int lr = quad * 32 + (lane >> 3) + 4 * i;
          size_t off = 0;  // element offset of (row lr, tile column 0)
          if (p.out_mode == kOutNatural) {
            off = (static_cast<size_t>(tc.m) * kBM + lr) * p.N + n0;
          } else if (p.out_mode == kOutReorder) {
            const size_t ld = static_cast<size_t>(p.rldn) * p.out_bn;
            off = (static_cast<size_t>(r / p.rldn) * kBM + lr) * ld + static_cast<size_t>(r % p.rldn) * p.out_bn +
                  n0 % p.out_bn;
          } else {  // kOutScatterRows: rows of the [M*N/BN, BN] view are remapped through RE
            const size_t row_id = static_cast<size_t>(r) * kBM + lr;
            const int re = p.RE[row_id];
            if (static_cast<unsigned>(re) >= static_cast<unsigned>(p.M) * static_cast<unsigned>(p.tiles_n)) {
              // a row index outside the buffer: report it and drop the row
              ptx::report_status(status, kStatusBadArgument, 2, static_cast<int32_t>(row_id), re);
              row_valid &= ~(1u << i);
            } else {
              off = static_cast<size_t>(re) * BN;
            }
          }
          row_ptr[i] = base + off * 2;
        }
      }

      // Residual: the warp's 32 rows x 64 columns of a chunk, a chunk ahead, 8 lanes to a row.
      [[maybe_unused]] uint4 res[8];
      [[maybe_unused]] auto load_residual = [&](int c) {
        const uint8_t* src = reinterpret_cast<const uint8_t*>(p.res) +
                             ((static_cast<size_t>(tc.m) * kBM + quad * 32 + (lane >> 3)) * p.N + n0 + c * 64) * 2 +
                             (lane & 7) * 16;
#pragma unroll
        for (int i = 0; i < 8; ++i) res[i] = ptx::ld_cg_v4(src + static_cast<size_t>(4 * i) * p.N * 2);
      };
      if constexpr (EPI == kEpiResidual) {
        if (exists) load_residual(MT == 2 ? 0 : wg);
      }

      // A warp that gives up goes on through the loop without touching data: the others may be
      // waiting for it at the tile barrier below.
      if (ok) {
        ok = __all_sync(0xffffffffu, ptx::mbar_wait_bounded(&tmem_full_bar[acc], acc_phase, s_abort, pipe_timeout,
                                                            4u * p.wait_sleep_ns));
        if (!ok && lane == 0) {
          ptx::report_status(status, kStatusTimeoutTmemFull, pos, acc, 0);
          *s_abort = 1;
        }
      }
      ptx::tc_fence_after_sync();

      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) +
                             static_cast<uint32_t>((MT == 2 ? wg : acc) * BN);
      constexpr int kChunkStep = MT == 2 ? 1 : 2;
      static_assert(kPlainEpilogueWarps * (kOutCols / 64) * L::kWarpBufBytes <= L::kEpiOffset, "the ring must hold a tile");
      const bool last_tile = pos + num_units >= sched_len;
      if (EPI == kEpiSwiGLU && ok && wg >= chunks && lane == 0) {
        // a half-width SwiGLU tile has one chunk: nothing for this warp to read before the hand-back
        ptx::mbar_arrive_cluster_tmem(tmem_empty_addr0 + static_cast<uint32_t>(acc) * 8u);
      }
#pragma unroll 1
      for (int c = MT == 2 ? 0 : wg; ok && c < chunks; c += kChunkStep) {
        uint32_t v0[32], v1[32];
        ptx::tmem_ld_32x32b_x32(t_row + c * 64, v0);
        ptx::tmem_ld_32x32b_x32(t_row + c * 64 + 32, v1);
        if constexpr (EPI == kEpiSwiGLU) {
          uint32_t u0[32], u1[32];
          ptx::tmem_ld_32x32b_x32(t_row + out_cols + c * 64, u0);
          ptx::tmem_ld_32x32b_x32(t_row + out_cols + c * 64 + 32, u1);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            v0[i] = __float_as_uint(silu_mul(v0[i], u0[i]));
            v1[i] = __float_as_uint(silu_mul(v1[i], u1[i]));
          }
        } else {
          ptx::tmem_ld_wait();
        }
        if (c + kChunkStep >= chunks) {
          // Accumulator fully read by this warp: hand it back to the (leader's) MMA warp.
          ptx::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_cluster_tmem(tmem_empty_addr0 + static_cast<uint32_t>(acc) * 8u);
        }
        if (!exists) continue;
        // The buffer is free once the previous store has read it: about 600 cycles after its issue,
        // 900 for a CTA's first store.  On the CTA's last tile nothing hides that and the operand
        // ring is idle (the accumulator is complete, so every load has landed and been multiplied):
        // the later chunks go through it instead.
        uint8_t* cbuf = buf;
        if (use_tma) {
          if (last_tile && c >= kChunkStep) {
            cbuf = smem + (ew * (kOutCols / 64) + c) * L::kWarpBufBytes;
          } else {
            if (lane == 0) ptx::bulk_wait_group_read<0>();
            __syncwarp();
          }
        }
        if constexpr (EPI == kEpiResidual) {
          // to the layout of the accumulators (a row per lane), through the buffer
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int lr = (lane >> 3) + 4 * i;
            *reinterpret_cast<uint4*>(cbuf + lr * 128 + (((lane & 7) ^ (lr & 7)) * 16)) = res[i];
          }
          __syncwarp();
          if (c + kChunkStep < chunks) load_residual(c + kChunkStep);
        }
        // Row `lane` of the warp's slice, 16-byte pieces swizzled as the tensor store expects.
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t(&v)[32] = j < 4 ? v0 : v1;
          const int b = 8 * (j & 3);
          uint4 w;
          w.x = pack2<BF16>(__uint_as_float(v[b + 0]), __uint_as_float(v[b + 1]));
          w.y = pack2<BF16>(__uint_as_float(v[b + 2]), __uint_as_float(v[b + 3]));
          w.z = pack2<BF16>(__uint_as_float(v[b + 4]), __uint_as_float(v[b + 5]));
          w.w = pack2<BF16>(__uint_as_float(v[b + 6]), __uint_as_float(v[b + 7]));
          uint4* piece = reinterpret_cast<uint4*>(cbuf + lane * 128 + ((j ^ (lane & 7)) * 16));
          if constexpr (EPI == kEpiResidual) w = add8<BF16>(w, *piece);
          *piece = w;
        }
        if (use_tma) {
          ptx::fence_proxy_async_smem();  // generic-proxy writes before the async-proxy read
          __syncwarp();
          if (lane == 0) {
            ptx::tma_store_2d(&maps.st, cbuf, tma_x0 + c * 64, tma_y0);
            ptx::bulk_commit_group();
          }
        } else {
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int lr = (lane >> 3) + 4 * i;
            const uint4 w = *reinterpret_cast<const uint4*>(buf + lr * 128 + (((lane & 7) ^ (lr & 7)) * 16));
            if ((row_valid >> i) & 1u) ptx::st_v4(row_ptr[i] + c * 128, w);
          }
          __syncwarp();  // everybody has read the buffer before it is written again
        }
      }

      if (exists && (p.signal | p.monitor) != 0 && p.MM[0] != nullptr) {
        // The tile may be announced only once all its stores have been written.
        if (use_tma && lane == 0) {
          ptx::bulk_wait_group<0>();
          ptx::fence_proxy_async_all();
        }
        ptx::named_bar_sync(tile_bar, kTileThreads);
        if (first && lane == 0 && *s_abort == 0) {
          int* mm = p.MM[0];
          if (p.signal) {
            int g, need;
            group_of_position(p, r, &g, &need);
            ptx::fence_acq_rel_gpu();
            ptx::red_release_gpu_add(reinterpret_cast<uint32_t*>(mm + g), 1u);
          }
          if (p.monitor) {
            const int order = atomicAdd(mm + p.mm_stride - 1, 1);
            mm[p.mm_stride + r] = order;
          }
        }
      }
      if (++acc == kAccStages) {
        acc = 0;
        acc_phase ^= 1u;
      }
    }
    // No tensor store may still read this CTA's shared memory when the CTA exits.
    if (use_tma && lane == 0) ptx::bulk_wait_group<0>();
  }

  __syncwarp();  // lanes that drained join theirs: the barriers' aligned forms take whole warps
  ptx::tc_fence_before_sync();
  if constexpr (CTA2) {
    // Neither CTA may free TMEM or leave while the other can still signal its barriers or
    // its MMAs read this CTA's shared memory.  Execution order only: no data crosses here (the
    // release form waited for the output stores to reach L2, 1,700 cycles at the end of a launch).
    ptx::cluster_arrive_relaxed();
    ptx::cluster_wait_acquire();
    if (warp_idx == 1) {
      ptx::tc_fence_after_sync();
      ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
    }
  } else {
    __syncthreads();
    if (warp_idx == 1) {
      ptx::tc_fence_after_sync();
      ptx::tmem_dealloc(tmem_base, kTmemCols);
    }
  }
}

}  // namespace fo
