// Error-corrected tensor-core GEMM, persistent CTA-pair variant (tcgen05 cta_group::2).
//
// Same arithmetic, panels and barrier protocol as tcec_gemm.cu (which replaces the
// reference's src/cumpsgemm_kernel.cuh:468-585); what changes is the tile and the schedule.
// A cluster of two CTAs owns 256 x 256 tiles of C: each CTA loads its own 128 rows of A
// (hi, lo) and its own 128-row half of the B tile (hi, lo), the even CTA issues every
// tcgen05.mma for the pair, and each CTA's TMEM receives its own 128 x 256 part of the
// accumulators, which its own epilogue warps drain.  Per SM and k-stage this moves 64 KiB from
// L2 instead of 96 KiB and leaves room for three stages instead of two.
//
// The kernel is persistent: the grid holds at most one cluster per SM pair and every cluster
// walks the tiles  t = cluster, cluster + #clusters, ...  The producer and the MMA issuer run
// ahead into the next tile while the epilogue warps still write the previous one: the next
// tile's operands are loaded and its hi*hi products start as soon as the last drain of D0 is
// done; its correction products wait until the epilogue gives D1 back, which is after the stores:
// the finished sums are kept in the D1 columns and stored from there (epilogue.cuh).
// Two schedule details came out of measurements and are explained where they are coded:
// clusters announce every tile start on a device counter and wait for their wave (keeps
// clusters that share panel rows at the same k, so the rows are fetched from DRAM once per
// wave); with beta != 0 the C tile is prefetched into L2 and read in groups of columns.
//
// Barriers (one set per CTA at identical shared-memory offsets; "leader" = cluster rank 0):
//   full[s]   leader's only: 1 arrival (leader's producer, expect_tx of both CTAs' bytes);
//             both CTAs' TMA loads complete on it (cta_group::2 loads, no multicast)
//   empty[s]  in both CTAs: 1 arrival, tcgen05.commit multicast from the leader
//   d0_full   in both CTAs: commit multicast after the hi*hi products of a chunk of stages
//   d0_empty  leader's only: 16 arrivals = 8 drain warps of each CTA (remote mbarrier arrive)
//   d1_full   in both CTAs: commit multicast after the last stage of a tile
//   d1_empty  leader's only: 16 arrivals, after the epilogue warps have stored the tile from D1
// Every wait is bounded; no TMA multicast is used.
#include "epilogue.cuh"
#include "gemm_common.cuh"
#include "ptx.cuh"
#include "work_list.cuh"

#include <mutex>

namespace cumpsgemm_b200 {
namespace {

constexpr int BM_CTA = 128;  // rows of C per CTA
constexpr int BN_PAIR = 256; // columns of C per pair (each CTA stores 128 rows of B)
constexpr int ROW_BYTES = kGemmRowBytes;
constexpr int NUM_THREADS = 384;
constexpr int NUM_EPI_WARPS = 8;
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t D1_COL = 256;
constexpr int TILE_BYTES = 128 * ROW_BYTES; // every sub-tile is 128 rows
constexpr int STAGE_BYTES = 4 * TILE_BYTES; // A_hi, A_lo, B_hi, B_lo
constexpr int STAGES = 3;
constexpr uint32_t kPaceMinStages = 32; // shortest K loop (in stages) that is paced
constexpr uint32_t C_PREFETCH_LEAD = 8; // drain chunks between the L2 prefetch of C and its use
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;

template <int KIND>
__device__ __forceinline__ void mma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t acc) {
  if constexpr (KIND == 0) {
    ptx::mma_f16_ss_pair(d, a, b, idesc, acc);
  } else {
    ptx::mma_tf32_ss_pair(d, a, b, idesc, acc);
  }
}

struct TileCoord {
  uint32_t batch;
  int m0; // first row of this CTA's 128 rows
  int n0; // first column of the pair's 256 columns
};

__device__ __forceinline__ TileCoord tile_coord(uint32_t tile, const GemmKernelParams &p,
                                                uint32_t rank) {
  const TilePos t = tile_raster(tile, p.tiles_m, p.tiles_n);
  TileCoord c;
  c.batch = t.batch;
  c.m0 = static_cast<int>(t.tm * 2 * BM_CTA + rank * BM_CTA);
  c.n0 = static_cast<int>(t.tn * BN_PAIR);
  return c;
}

// Tiles left over from the whole waves are cut along K (work_list.cuh) when that shortens the
// launch: m=n=k=4096 has 256 tiles on 74 clusters = 3.46 waves, the last 34 tiles are cut in two
// and the launch takes 3.5 tile times instead of 4.  Every piece parks its plain FP32 partial
// sums in scratch memory; piece_fixup.cu adds them.
struct PairPlan {
  float *partial; // [cluster][2][CTA rank][256 columns][128 rows]
  WorkPlan w;
};

// Where a CTA's stages, barriers and flags are in shared memory.
struct SharedLayout {
  uint8_t *smem;
  uint64_t *full_bar, *empty_bar, *d0_full, *d0_empty, *d1_full, *d1_empty;
  uint32_t *tmem_base_ptr;
  volatile int *abort_flag;
  __device__ __forceinline__ SharedLayout() {
    extern __shared__ uint8_t smem_raw[];
    smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                       ~static_cast<uintptr_t>(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + STAGES * STAGE_BYTES);
    full_bar = bars;
    empty_bar = bars + STAGES;
    d0_full = bars + 2 * STAGES;
    d0_empty = bars + 2 * STAGES + 1;
    d1_full = bars + 2 * STAGES + 2;
    d1_empty = bars + 2 * STAGES + 3;
    tmem_base_ptr = reinterpret_cast<uint32_t *>(bars + 2 * STAGES + 4);
    abort_flag = reinterpret_cast<volatile int *>(tmem_base_ptr + 1);
  }
};

// Barriers, TMEM, tensor maps, and the peer's: what a CTA does before it needs anything of an earlier
// kernel, the same for both kinds.  Returns the TMEM address.
__device__ __forceinline__ uint32_t set_up(const CUtensorMap &map_a, const CUtensorMap &map_b) {
  const SharedLayout sm;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(ptx::smem_u32(&sm.full_bar[s]), 1);
      ptx::mbar_init(ptx::smem_u32(&sm.empty_bar[s]), 1);
    }
    ptx::mbar_init(ptx::smem_u32(sm.d0_full), 1);
    ptx::mbar_init(ptx::smem_u32(sm.d0_empty), 2 * NUM_EPI_WARPS);
    ptx::mbar_init(ptx::smem_u32(sm.d1_full), 1);
    ptx::mbar_init(ptx::smem_u32(sm.d1_empty), 2 * NUM_EPI_WARPS);
    *sm.abort_flag = 0;
    ptx::mbar_init_fence();
    ptx::prefetch_tensormap(&map_a);
    ptx::prefetch_tensormap(&map_b);
  }
  if ((threadIdx.x >> 5) == 1) {
    ptx::tmem_alloc_pair(ptx::smem_u32(sm.tmem_base_ptr), TMEM_COLS);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before();
  __syncthreads();
  // both CTAs' barriers must exist before any remote arrive / remote TMA completion
  ptx::cluster_arrive();
  ptx::cluster_wait();
  ptx::tc_fence_after();
  return *sm.tmem_base_ptr;
}

// SET_UP = false: the caller has called set_up.
template <int KIND, bool SET_UP = true>
__device__ __forceinline__ void pair_body(const CUtensorMap &map_a, const CUtensorMap &map_b,
                                          const GemmKernelParams &p, const PairPlan &plan) {
  constexpr int K_STEPS = ROW_BYTES / 32;
  constexpr uint32_t STAGES_PER_UNIT = (KIND == 0) ? 1 : 2; // a unit is 64 k values
  constexpr int MY_MODE = (KIND == 0) ? CUMPSGEMM_FP16TCEC : CUMPSGEMM_TF32TCEC;
  constexpr uint32_t IDESC = ptx::make_idesc(KIND == 0 ? 0 : 2, 2 * BM_CTA, BN_PAIR);
  constexpr int CPT = BN_PAIR / 2;

  const SharedLayout sm;
  uint8_t *smem = sm.smem;
  uint64_t *full_bar = sm.full_bar, *empty_bar = sm.empty_bar;
  uint64_t *d0_full = sm.d0_full, *d0_empty = sm.d0_empty;
  uint64_t *d1_full = sm.d1_full, *d1_empty = sm.d1_empty;
  volatile int *abort_flag = sm.abort_flag;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();
  const bool leader = (rank == 0);
  const uint32_t cluster_id = blockIdx.x >> 1;
  const uint32_t num_clusters = gridDim.x >> 1;

  const uint32_t tmem_base = SET_UP ? set_up(map_a, map_b) : *sm.tmem_base_ptr;
  const uint32_t k_blocks = p.k_blocks;
  const bool dbg = (p.debug != nullptr);
  unsigned long long dbg_wait = 0, dbg_wait2 = 0;

  // Gated launch: nothing to do when the device-side decision picked the other kind (uniform
  // over the grid).  The decision is written by a kernel in front of the split pass.  That the
  // split pass has waited for it says that the write is done; that this grid sees it, the wait
  // here says.
  bool mine = true;
  if (p.dyn != nullptr) {
    ptx::griddep_wait();
    mine = p.dyn->gemm_mode == MY_MODE;
  }

  if (!mine) {
    // straight to the teardown
  } else if (warp == 0) {
    // ================================================================ TMA producer (both CTAs)
    if (ptx::elect_one()) {
      // launched with programmatic serialization behind the split pass, which also zeroes the
      // wave counter: both are complete after this
      ptx::griddep_wait();
      uint32_t it = 0; // stage uses since kernel start, across tiles
      bool ok = true;
      bool pace = leader && p.wave_counter != nullptr && plan.w.whole_tiles > num_clusters;
      uint32_t wave = 0;
      WorkList list(plan.w, cluster_id, num_clusters);
      WorkItem x;
      while (ok && list.next(plan.w, x)) {
        const TileCoord tc = tile_coord(x.tile, p, rank);
        const int za = static_cast<int>(tc.batch * 2u);
        const int nb0 = tc.n0 + static_cast<int>(rank) * 128; // this CTA's rows of the B tile
        if (pace && x.tile < plan.w.whole_tiles) {
          // Keep the clusters in step.  Clusters that run at the same time share panel rows
          // through L2 only while they are at about the same k; left alone they drift apart
          // by about 2 % per tile and, once the drift exceeds what L2 retains, most loads go
          // to DRAM (measured at m=n=k=16384: 88 GB read per launch against 4 GB of panels
          // and C).  So every cluster announces each tile start and waits until all clusters
          // of the wave have.  The wait is only a pacing aid: it gives up after 100 us, and
          // then this cluster stops pacing for the rest of the launch, so clusters that are
          // not resident at the same time cost one time-out and never a wrong result.
          atomicAdd(p.wave_counter, 1u);
          const uint32_t target = min(plan.w.whole_tiles, (++wave) * num_clusters);
          const uint64_t t0 = ptx::globaltimer_ns();
          while (*reinterpret_cast<volatile unsigned int *>(p.wave_counter) < target) {
            if (ptx::globaltimer_ns() - t0 > 100000ull) {
              pace = false;
              break;
            }
            __nanosleep(64);
          }
        }
        const uint32_t kb0 = x.u0 * STAGES_PER_UNIT, kbn = x.un * STAGES_PER_UNIT;
        for (uint32_t kb = 0; kb < kbn; ++kb, ++it) {
          const uint32_t s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1u;
          ok = ptx::mbar_wait_timed(ptx::smem_u32(&empty_bar[s]), ph ^ 1u, abort_flag, p.status,
                                    ptx::kErrWaitEmpty, dbg, &dbg_wait);
          if (!ok) break;
          const uint32_t fb_local = ptx::smem_u32(&full_bar[s]);
          if (leader) ptx::mbar_arrive_expect_tx(fb_local, 2 * STAGE_BYTES);
          const uint32_t fb = ptx::map_to_cta(fb_local, 0); // the leader's barrier
          const uint32_t st = ptx::smem_u32(smem + s * STAGE_BYTES);
          // coordinates: (element in the K block, row, plane * k_blocks + K block); each box
          // is one contiguous 16 KiB run of the K-blocked panel
          const int zh = static_cast<int>(static_cast<uint32_t>(za) * k_blocks + kb0 + kb);
          const int zl = zh + static_cast<int>(k_blocks);
          ptx::tma_load_3d_pair(st, &map_a, fb, 0, tc.m0, zh);
          ptx::tma_load_3d_pair(st + TILE_BYTES, &map_a, fb, 0, tc.m0, zl);
          ptx::tma_load_3d_pair(st + 2 * TILE_BYTES, &map_b, fb, 0, nb0, zh);
          ptx::tma_load_3d_pair(st + 3 * TILE_BYTES, &map_b, fb, 0, nb0, zl);
        }
      }
      if (dbg) atomicAdd(p.debug + 2, dbg_wait);
    }
  } else if (warp == 1) {
    // ================================================================ MMA issuer (leader only)
    if (leader && ptx::elect_one()) {
      const uint32_t d0 = tmem_base;
      const uint32_t d1 = tmem_base + D1_COL;
      constexpr uint16_t BOTH = 0x3;
      bool ok = true;
      const long long dbg_t0 = clock64();
      const uint32_t chunk = p.drain_chunk, first = p.first_chunk;
      const uint64_t desc0 = ptx::make_kmajor_desc<ROW_BYTES>(ptx::smem_u32(smem));
      constexpr uint64_t kStage = STAGE_BYTES >> 4, kTile = TILE_BYTES >> 4;
      uint32_t s = 0, ph = 0, d0_ph = 1, d1_ph = 1;
      WorkList list(plan.w, cluster_id, num_clusters);
      WorkItem x;
      while (ok && list.next(plan.w, x)) {
        const uint32_t kbn = x.un * STAGES_PER_UNIT;
        uint32_t chunk_end = 0; // first stage after the current chunk
        for (uint32_t kb = 0; kb < kbn; ++kb) {
          const bool first_in_chunk = (kb == chunk_end);
          if (first_in_chunk) chunk_end = min(kb + (kb == 0 ? first : chunk), kbn);
          ok = ptx::mbar_wait_timed(ptx::smem_u32(&full_bar[s]), ph, abort_flag, p.status,
                                    ptx::kErrWaitFull, dbg, &dbg_wait);
          if (!ok) break;
          ptx::tc_fence_after();
          const uint64_t a_hi = desc0 + s * kStage;
          const uint64_t a_lo = a_hi + kTile, b_hi = a_hi + 2 * kTile, b_lo = a_hi + 3 * kTile;
          auto corrections = [&](uint32_t acc_first) {
#pragma unroll
            for (int ks = 0; ks < K_STEPS; ++ks)
              mma_pair<KIND>(d1, a_lo + 2 * ks, b_hi + 2 * ks, IDESC, ks > 0 ? 1u : acc_first);
#pragma unroll
            for (int ks = 0; ks < K_STEPS; ++ks)
              mma_pair<KIND>(d1, a_hi + 2 * ks, b_lo + 2 * ks, IDESC, 1u);
          };
          // The corrections of a chunk's first stage come before its hi*hi products, those of
          // its last stage after them: the drain of D0 in between has two stages' corrections
          // to hide behind (one with single-stage chunks).  In the first stage of an item they
          // come after, because they have to wait until the epilogue has given D1 back.
          const bool corrections_first = first_in_chunk && kb > 0;
          if (corrections_first) corrections(1u);
          if (first_in_chunk) {
            // D0 of the previous chunk must have been drained before it is overwritten.
            ok = ptx::mbar_wait_timed(ptx::smem_u32(d0_empty), d0_ph, abort_flag, p.status,
                                      ptx::kErrWaitD0Empty, dbg, &dbg_wait2);
            if (!ok) break;
            d0_ph ^= 1u;
            ptx::tc_fence_after();
          }
#pragma unroll
          for (int ks = 0; ks < K_STEPS; ++ks)
            mma_pair<KIND>(d0, a_hi + 2 * ks, b_hi + 2 * ks, IDESC,
                           (!first_in_chunk || ks > 0) ? 1u : 0u);
          if (kb + 1 == chunk_end) ptx::tc_commit_pair(ptx::smem_u32(d0_full), BOTH);
          if (!corrections_first) {
            if (kb == 0) {
              ok = ptx::mbar_wait_timed(ptx::smem_u32(d1_empty), d1_ph, abort_flag, p.status,
                                        ptx::kErrWaitD1Empty, dbg, &dbg_wait2);
              if (!ok) break;
              d1_ph ^= 1u;
              ptx::tc_fence_after();
            }
            corrections(kb > 0 ? 1u : 0u);
          }
          ptx::tc_commit_pair(ptx::smem_u32(&empty_bar[s]), BOTH);
          if (++s == STAGES) {
            s = 0;
            ph ^= 1u;
          }
        }
        if (ok) ptx::tc_commit_pair(ptx::smem_u32(d1_full), BOTH);
      }
      if (dbg) {
        atomicAdd(p.debug + 0, dbg_wait);
        atomicAdd(p.debug + 1, dbg_wait2);
        atomicAdd(p.debug + 4, static_cast<unsigned long long>(clock64() - dbg_t0));
        atomicAdd(p.debug + 5, 1ull);
      }
    }
  } else if (warp >= 4) {
    // ================================================================ drain + epilogue (both CTAs)
    const uint32_t t_base = tmem_base + ((static_cast<uint32_t>(warp & 3) * 32u) << 16) +
                            static_cast<uint32_t>((warp - 4) >> 2) * CPT;
    const uint32_t d0_empty_leader = ptx::map_to_cta(ptx::smem_u32(d0_empty), 0);

    // the split pass has read its sources and zeroed nothing these warps touch before the first
    // finished chunk, but the wait keeps every global access of this kernel behind it
    ptx::griddep_wait();
    uint32_t d0_ph = 0, d1_ph = 0;
    bool ok = true;
    WorkList list(plan.w, cluster_id, num_clusters);
    WorkItem x;
    while (ok && list.next(plan.w, x)) {
      const uint32_t stages = x.un * STAGES_PER_UNIT;
      const uint32_t n_chunks =
          1u + (stages > p.first_chunk
                    ? (stages - p.first_chunk + p.drain_chunk - 1u) / p.drain_chunk
                    : 0u);
      const uint32_t prefetch_at =
          ((p.beta_r == 0.f && p.beta_i == 0.f) || x.un != plan.w.units) ? n_chunks
          : (n_chunks > C_PREFETCH_LEAD) ? n_chunks - C_PREFETCH_LEAD
                                         : 0u;
      float acc[CPT];
#pragma unroll
      for (int i = 0; i < CPT; ++i) acc[i] = 0.f;

#pragma unroll 1
      for (uint32_t c = 0; c < n_chunks; ++c) {
        if (c == prefetch_at) {
          // beta != 0: pull this warp's part of the C tile into L2 a few chunks before the
          // epilogue reads it (lane l fetches the line of columns l, l+32, ...)
          const TileCoord tc = tile_coord(opaque(x.tile), p, rank);
          const uint32_t row = static_cast<uint32_t>(tc.m0) + static_cast<uint32_t>(warp & 3) * 32u;
          const float *cp =
              ((p.c_array != nullptr) ? p.c_array[tc.batch]
                                      : p.c + static_cast<uint64_t>(tc.batch) * p.stride_c) + row;
#pragma unroll 1
          for (int q = 0; q < CPT / 32; ++q) {
            const uint32_t col = static_cast<uint32_t>(tc.n0) +
                                 static_cast<uint32_t>(((warp - 4) >> 2) * CPT + q * 32 + lane);
            if (col < p.n && row < p.m) ptx::prefetch_l2(cp + static_cast<uint64_t>(col) * p.ldc);
          }
        }
        ok = ptx::warp_agrees(ptx::mbar_wait(ptx::smem_u32(d0_full), d0_ph, abort_flag, p.status,
                                             ptx::kErrWaitD0Full));
        if (!ok) break;
        d0_ph ^= 1u;
        ptx::tc_fence_after();
        drain_sums<CPT>(t_base, acc);
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_cluster(d0_empty_leader);
      }
      if (!ok) break;

      ok = ptx::warp_agrees(ptx::mbar_wait(ptx::smem_u32(d1_full), d1_ph, abort_flag, p.status,
                                           ptx::kErrWaitD1Full));
      if (!ok) break;
      d1_ph ^= 1u;
      ptx::tc_fence_after();
      // the finished sums stay in the D1 columns; from here on they are read from there, and what
      // the epilogue needs to know of the tile is worked out only now (epilogue.cuh)
      const uint32_t t_sums = t_base + D1_COL;
      add_corrections_in_tmem<CPT>(t_sums, acc, p.lo_scale_inv);
      const bool part = x.un != plan.w.units; // this item is a piece of a tile
      const TileCoord tc = tile_coord(opaque(x.tile), p, rank);
      const uint32_t quarter = static_cast<uint32_t>(warp & 3);
      const uint32_t col_base = static_cast<uint32_t>((warp - 4) >> 2) * CPT;
      const uint32_t d1_empty_leader = ptx::map_to_cta(ptx::smem_u32(d1_empty), 0);
      // D1 is no longer needed: the issuer may start the next tile's correction products
      auto release_d1 = [&]() {
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_cluster(d1_empty_leader);
      };

      if (part) {
        // a piece of a tile: park the partial sums for the kernel that adds the pieces
        constexpr uint32_t HALF = BN_PAIR * BM_CTA; // floats of one CTA's 128 x 256 half
        const uint32_t lane_off = col_base * BM_CTA + quarter * 32u + static_cast<uint32_t>(lane);
        float *mine = plan.partial +
                      static_cast<uint64_t>((cluster_id * 2u + x.slot) * 2u + rank) * HALF + lane_off;
#pragma unroll 1
        for (int c = 0; c < CPT; c += kEpiGroup) {
          uint32_t v[kEpiGroup];
          ptx::tmem_ld_32x32b_x16(t_sums + c, v);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < kEpiGroup; ++i)
            __stcg(mine + (c + i) * BM_CTA, __uint_as_float(v[i]));
        }
        release_d1();
        continue;
      }

      // C(row, col): lanes hold consecutive rows of the column-major C, so each warp access
      // covers 128 contiguous bytes of one column.
      const uint32_t row =
          static_cast<uint32_t>(tc.m0) + quarter * 32u + static_cast<uint32_t>(lane);
      float *cbase = ((p.c_array != nullptr) ? p.c_array[tc.batch]
                                              : p.c + static_cast<uint64_t>(tc.batch) * p.stride_c) +
                     row;
      const float unscale = (p.dyn != nullptr) ? p.dyn->unscale_c : 1.f;
      store_tile<CPT>(t_sums, cbase, p.ldc, static_cast<uint32_t>(tc.n0) + col_base, p.n, row < p.m,
                      p.alpha_r * unscale, p.alpha_i * unscale, p.beta_r, p.beta_i,
                      p.is_complex != 0);
      release_d1();
    }
  }

  // ---------------------------------------------------------------- teardown
  // The peer's shared memory and TMEM are in use by the leader's MMAs until the last d1_full
  // has fired in both CTAs; the cluster barrier below keeps either CTA from leaving before
  // the other has finished its last epilogue.
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_arrive();
  ptx::cluster_wait();
  if (*abort_flag) {
    const uint64_t t0 = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

template <int KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
    tcec_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a,
                          const __grid_constant__ CUtensorMap map_b, const GemmKernelParams p,
                          const PairPlan plan) {
  pair_body<KIND>(map_a, map_b, p, plan);
}

// AUTO: both kinds' tensor maps and parameters travel with the launch; the device-side
// decision picks the pipeline (uniform over the grid).  The reference launches the kernels of
// both kinds and lets the deselected one exit at once (src/cumpsgemm_kernel.cuh:478-489).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
    tcec_gemm_pair_auto_kernel(const __grid_constant__ CUtensorMap map_a16,
                               const __grid_constant__ CUtensorMap map_b16,
                               const GemmKernelParams p16,
                               const __grid_constant__ CUtensorMap map_a32,
                               const __grid_constant__ CUtensorMap map_b32,
                               const GemmKernelParams p32, const PairPlan plan) {
  set_up(map_a16, map_b16);
  ptx::griddep_wait(); // the decision is written by an earlier kernel of the call
  if (p16.dyn->gemm_mode == CUMPSGEMM_TF32TCEC) {
    pair_body<1, false>(map_a32, map_b32, p32, plan);
  } else {
    pair_body<0, false>(map_a16, map_b16, p16, plan);
  }
}

// Per device and kernel, once (any thread): shared-memory attribute and the number of
// clusters the device can keep resident.  TAG tells the kernels apart (two of them have the
// same function type, which alone would make them share the statics below).
template <int TAG, class Kernel> cudaError_t pair_setup(Kernel kernel, int *clusters_out) {
  static std::once_flag once[64];
  static cudaError_t setup_error[64];
  static int max_clusters[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::call_once(once[dev], [&]() {
    setup_error[dev] =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // one cluster per SM pair; if the device can co-schedule fewer, use what it reports
    int clusters = sms / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(2 * clusters));
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    int active = 0;
    if (setup_error[dev] == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&active, kernel, &cfg) == cudaSuccess) {
      if (active > 0 && active < clusters) clusters = active;
    } else {
      cudaGetLastError();
    }
    max_clusters[dev] = clusters > 0 ? clusters : 1;
  });
  *clusters_out = max_clusters[dev];
  return setup_error[dev];
}

// Tensor maps and kernel parameters of one kind.  Returns false on invalid sizes.
bool pair_prepare(const TcecGemmArgs &a, SplitKind kind, int max_clusters, CUtensorMap *map_a,
                  CUtensorMap *map_b, GemmKernelParams *pp) {
  const uint32_t planes = a.batch * 2u;
  if (!make_panel_map(map_a, kind, a.panel_a, a.k_pad, a.rows_pad_a, planes, 128) ||
      !make_panel_map(map_b, kind, a.panel_b, a.k_pad, a.rows_pad_b, planes, 128)) {
    return false;
  }
  GemmKernelParams &p = *pp;
  p.c = a.c;
  p.c_array = a.c_array;
  p.ldc = a.ldc;
  p.stride_c = a.stride_c;
  p.m = a.m;
  p.n = a.n;
  const uint32_t es = (kind == SplitKind::fp16) ? 2u : 4u;
  p.k_blocks = a.k_pad / (ROW_BYTES / es);
  p.tiles_m = (a.m + 2 * BM_CTA - 1) / (2 * BM_CTA);
  p.tiles_n = (a.n + BN_PAIR - 1) / BN_PAIR;
  p.alpha_r = a.alpha_r;
  p.alpha_i = a.alpha_i;
  p.beta_r = a.beta_r;
  p.beta_i = a.beta_i;
  p.lo_scale_inv = (kind == SplitKind::fp16) ? (1.f / 2048.f) : 1.f;
  p.is_complex = a.is_complex ? 1 : 0;
  p.dyn = a.dyn;
  p.status = a.dev_status;
  p.debug = a.debug;
  {
    const int v = a.tuning.drain_chunk;
    // Two stages (128 FP16 / 64 TF32 k values) per drain.  Measured at m=n=k=16384, uniform(-1,1):
    // residual 3.1e-7 / 2.8e-7 / 3.7e-7 / 6.5e-7 / 2.5e-6 / 1.9e-5 for 1 / 2 / 4 / 8 / 32 / 256
    // stages per drain (FP32 cuBLAS SGEMM on the same inputs: 2.3e-6).  One stage where there is at
    // most one wave of tiles, as in the single-CTA kernel that shares those sizes (m=n=k=2048:
    // 1.7e-7 instead of 2.3e-7 for 3 % of the time).
    const uint32_t pairs = static_cast<uint32_t>(max_clusters);
    const uint32_t dflt = (static_cast<uint64_t>(p.tiles_m) * p.tiles_n * a.batch > pairs) ? 2 : 1;
    p.drain_chunk = static_cast<uint16_t>((v >= 1) ? (v > 0xffff ? 0xffff : v) : dflt);
    // The first chunk of a tile may be longer (the epilogue warps are still storing the previous
    // tile then).  By default it is not: accuracy falls with the length of a chunk, and time hardly
    // does (4096^3, beta = 0.5, us per call with a first chunk of 2 / 4 / 8 stages: 336 / 337 / 328).
    const int fv = a.tuning.first_chunk;
    p.first_chunk = static_cast<uint16_t>((fv >= 1) ? (fv > 0xffff ? 0xffff : fv) : p.drain_chunk);
    if (p.first_chunk < p.drain_chunk) p.first_chunk = p.drain_chunk;
  }
  const uint64_t total = static_cast<uint64_t>(p.tiles_m) * p.tiles_n * a.batch;
  if (total == 0 || total > 0x7fffffffull) return false;
  if (a.rows_pad_a < p.tiles_m * 2 * BM_CTA || a.rows_pad_b < p.tiles_n * BN_PAIR) return false;
  p.total_tiles = static_cast<uint32_t>(total);
  p.wave_counter = nullptr;
  return true;
}

} // namespace

// Plan of a launch on at most `max_clusters` clusters: how the tiles left over from the whole
// waves are cut along K.
//   At most half a wave of them: every tile in equal slices, one cluster each.  A slice keeps at
//   least 1024 k values, so that its prologue and drain stay amortised.
//   More than half a wave: their k range laid end to end and shared by all clusters.
// Either way only if the launch gets shorter by more than the pieces cost: parking and adding
// them takes about 0.35 us per left-over tile, a unit of 64 k values 0.9 us (FP16) or 1.8 (TF32).
WorkPlan plan_pair(const Tuning &tuning, bool tf32, bool can_cut, uint32_t total_tiles,
                   uint32_t units, uint32_t max_clusters) {
  WorkPlan t;
  t.total_tiles = total_tiles;
  t.whole_tiles = total_tiles;
  t.units = units;
  t.slice_units = 0;
  t.piece_clusters = 0;
  t.slices = 0;
  const uint32_t rem = max_clusters > 0 ? total_tiles % max_clusters : 0;
  if (!can_cut || tuning.tail_split == 0 || rem == 0 || max_clusters > 0xffffu) return t;
  const uint32_t min_saved = 2 + (tf32 ? rem / 5 : 2 * rem / 5);
  if (2 * rem <= max_clusters) {
    uint32_t slices = max_clusters / rem;
    if (slices > units / 16u) slices = units / 16u;
    if (slices > 8u) slices = 8u;
    if (tuning.tail_split > 1 && slices > static_cast<uint32_t>(tuning.tail_split))
      slices = static_cast<uint32_t>(tuning.tail_split);
    if (slices < 2u) return t;
    const uint32_t per = (units + slices - 1) / slices;
    slices = (units + per - 1) / per; // no empty slice
    if (slices < 2u || per + min_saved > units) return t;
    t.whole_tiles = total_tiles - rem;
    t.slices = static_cast<uint16_t>(slices);
    t.slice_units = per;
    t.piece_clusters = static_cast<uint16_t>(rem * slices);
    return t;
  }
  const uint64_t left = static_cast<uint64_t>(rem) * units;
  const uint32_t per = static_cast<uint32_t>((left + max_clusters - 1) / max_clusters);
  if (tuning.tail_split > 1 || per + min_saved > units || left > 0x7fffffffull) return t;
  t.whole_tiles = total_tiles - rem;
  t.piece_clusters = static_cast<uint16_t>(max_clusters);
  return t;
}

namespace {

// Pacing pays when tiles are long (the drift it removes is 2 % of a tile) and clusters share
// panel rows; for short tiles a barrier per tile costs more than it saves.
bool wants_pacing(const TcecGemmArgs &a, uint32_t clusters, const GemmKernelParams &p,
                  const WorkPlan &w) {
  return a.wave_counter != nullptr && w.whole_tiles > clusters && p.k_blocks >= kPaceMinStages &&
         a.tuning.pace != 0;
}

// Grid and plan of a launch, in units of 64 k values.
PairPlan make_plan(const TcecGemmArgs &a, bool tf32, uint32_t total_tiles, int max_clusters,
                   uint32_t *clusters) {
  PairPlan plan;
  plan.partial = a.tail_partial;
  plan.w = plan_pair(a.tuning, tf32, a.tail_partial != nullptr, total_tiles,
                     a.k_pad / 64, static_cast<uint32_t>(max_clusters));
  *clusters = plan.w.whole_tiles > plan.w.piece_clusters ? plan.w.whole_tiles
                                                          : plan.w.piece_clusters;
  if (*clusters > static_cast<uint32_t>(max_clusters)) *clusters = static_cast<uint32_t>(max_clusters);
  return plan;
}

// The kernel that adds the pieces, if the plan cut any tile.
cudaError_t fix_up(const TcecGemmArgs &a, const GemmKernelParams &p, const PairPlan &plan,
                   cudaStream_t stream) {
  if (plan.w.piece_clusters == 0) return cudaSuccess;
  const PieceFixupArgs f = {plan.partial, a.c,       a.c_array, a.dyn,     a.ldc,
                            a.stride_c,   a.m,       a.n,       p.tiles_m, p.tiles_n,
                            BN_PAIR,      a.alpha_r, a.alpha_i, a.beta_r,  a.beta_i,
                            a.is_complex};
  return launch_piece_fixup(f, plan.w, stream);
}

template <int KIND> cudaError_t launch_pair(const TcecGemmArgs &a, cudaStream_t stream) {
  int max_clusters = 1;
  const cudaError_t se = pair_setup<KIND>(tcec_gemm_pair_kernel<KIND>, &max_clusters);
  if (se != cudaSuccess) return se;
  constexpr SplitKind kind = KIND == 0 ? SplitKind::fp16 : SplitKind::tf32;
  CUtensorMap map_a, map_b;
  GemmKernelParams p;
  if (!pair_prepare(a, kind, max_clusters, &map_a, &map_b, &p)) return cudaErrorInvalidValue;
  uint32_t clusters = 0;
  const PairPlan plan = make_plan(a, KIND == 1, p.total_tiles, max_clusters, &clusters);
  if (wants_pacing(a, clusters, p, plan.w)) p.wave_counter = a.wave_counter;
  const cudaError_t e = launch_chained(tcec_gemm_pair_kernel<KIND>, 2 * clusters, NUM_THREADS,
                                       SMEM_BYTES, stream, map_a, map_b, p, plan);
  return e != cudaSuccess ? e : fix_up(a, p, plan, stream);
}

} // namespace

cudaError_t pair_max_clusters(StreamKind kind, int *clusters) {
  switch (kind) {
  case StreamKind::fp16:
    return pair_setup<0>(tcec_gemm_pair_kernel<0>, clusters);
  case StreamKind::tf32:
    return pair_setup<1>(tcec_gemm_pair_kernel<1>, clusters);
  default:
    return pair_setup<2>(tcec_gemm_pair_auto_kernel, clusters);
  }
}

cudaError_t launch_tcec_gemm_pair(const TcecGemmArgs &a, cudaStream_t stream) {
  if (!a.error_correction) return cudaErrorInvalidValue;
  return (a.kind == SplitKind::fp16) ? launch_pair<0>(a, stream) : launch_pair<1>(a, stream);
}

cudaError_t launch_tcec_gemm_pair_auto(const TcecGemmArgs &a, cudaStream_t stream) {
  if (!a.error_correction || a.dyn == nullptr) return cudaErrorInvalidValue;
  int max_clusters = 1;
  const cudaError_t se = pair_setup<2>(tcec_gemm_pair_auto_kernel, &max_clusters);
  if (se != cudaSuccess) return se;
  CUtensorMap a16, b16, a32, b32;
  GemmKernelParams p16, p32;
  if (!pair_prepare(a, SplitKind::fp16, max_clusters, &a16, &b16, &p16) ||
      !pair_prepare(a, SplitKind::tf32, max_clusters, &a32, &b32, &p32))
    return cudaErrorInvalidValue;
  uint32_t clusters = 0;
  // (one plan for whichever kind runs)
  const PairPlan plan = make_plan(a, false, p16.total_tiles, max_clusters, &clusters);
  // pacing depends on the K loop length, which differs by kind: one counter serves whichever runs
  if (wants_pacing(a, clusters, p16, plan.w)) p16.wave_counter = a.wave_counter;
  if (wants_pacing(a, clusters, p32, plan.w)) p32.wave_counter = a.wave_counter;
  const cudaError_t e = launch_chained(tcec_gemm_pair_auto_kernel, 2 * clusters, NUM_THREADS,
                                       SMEM_BYTES, stream, a16, b16, p16, a32, b32, p32, plan);
  return e != cudaSuccess ? e : fix_up(a, p16, plan, stream);
}

} // namespace cumpsgemm_b200

extern "C" int cuMpSGEMM_plan_pair_tail(unsigned total_tiles, unsigned clusters, unsigned k_pad,
                                        int tf32, unsigned *split_begin, unsigned *slices,
                                        unsigned *slice_k, unsigned *work_items) {
  using namespace cumpsgemm_b200;
  if (total_tiles == 0 || clusters == 0 || k_pad == 0 || k_pad % 64 != 0 ||
      split_begin == nullptr || slices == nullptr || slice_k == nullptr || work_items == nullptr)
    return 1;
  const WorkPlan t = plan_pair(Tuning{}, tf32 != 0, true, total_tiles, k_pad / 64, clusters);
  const bool sliced = t.slice_units != 0;
  *split_begin = sliced ? t.whole_tiles : total_tiles;
  *slices = sliced ? t.slices : 1;
  *slice_k = sliced ? t.slice_units * 64 : k_pad;
  *work_items = sliced ? t.whole_tiles + t.piece_clusters : total_tiles;
  return 0;
}

extern "C" int cuMpSGEMM_plan_pair(unsigned total_tiles, unsigned clusters, unsigned k_pad, int tf32,
                                   unsigned *units, unsigned *whole_tiles, unsigned *piece_clusters,
                                   unsigned *slices, unsigned *slice_units) {
  using namespace cumpsgemm_b200;
  if (total_tiles == 0 || clusters == 0 || k_pad == 0 || k_pad % 64 != 0 || units == nullptr ||
      whole_tiles == nullptr || piece_clusters == nullptr || slices == nullptr ||
      slice_units == nullptr)
    return 1;
  const WorkPlan t = plan_pair(Tuning{}, tf32 != 0, true, total_tiles, k_pad / 64, clusters);
  *units = t.units;
  *whole_tiles = t.whole_tiles;
  *piece_clusters = t.piece_clusters;
  *slices = t.slices;
  *slice_units = t.slice_units;
  return 0;
}
