// Error-corrected tensor-core GEMM on CTA pairs that splits its FP32 operands on the way from
// TMA to the tensor core: no split pass, no operand workspace, one launch.
//
// The reference splits every FP32 value at fragment load, inside the GEMM kernel
// (src/device_tcec_wrapper.hpp:72-80 called from src/cumpsgemm_kernel.cuh:58-100).  Here a
// cluster of two CTAs owns a 256 x BN tile of C (BN = 256 or 128; for batches of matrices with at most 128
// rows a single CTA a 128 x 128 one, with the same body); each CTA
//   * fetches its own 128 rows of op(A) and its own BN / 2 rows of op(B) as plain FP32 through TMA
//     into a ring of raw slots (32 k values each; edges are zero filled by TMA, so no thread
//     tests bounds),
//   * has sixteen converter warps, which split the raw values into hi / lo (same bits as
//     split_kernels.cu) and write them as 128-byte-swizzled K-major tiles in shared memory, with 128
//     columns A's to tensor memory instead, lane = row,
//   * and holds its 128 rows of the accumulators in tensor memory: those of hi*hi, one per half of the
//     tile's columns, which its eight epilogue warps drain after every stage (64 FP16 / 32 TF32 values
//     of k) into FP32 running sums in registers, and those of the corrections lo*hi + hi*lo, which are
//     read once, at the end of the tile.
// The even CTA's single issuing thread drives the tensor cores of both SMs (cta_group::2).
//
// The corrections have accumulators of their own because the tensor core truncates what it adds, and
// aligns the products of FP16 numbers below 2^-14 as if they were larger.  Added to hi*hi there (scaled by
// 2^-11 on the way, which would leave room for A in tensor memory with 256 columns too) they
// cost 2 to 6 % less time and lost bits wherever few products make up a sum: with one non-zero per row of
// A the mean of the relative errors was -3.5e-8 instead of 0, and with small elements in B
// the largest one 4e-6 instead of 4.5e-7.  (Draining both kinds every stage instead takes 1.5 times as long.)
// The issue order hides the drain of one stage behind the corrections of the next; a finished tile's
// corrections are given back before its stores.
//
// What bounds it: with 256 columns shared memory.  Per stage of 64 k values it takes 64 KiB from TMA,
// gives 64 KiB to the converters, takes 64 KiB of hi / lo tiles back and feeds 112 KiB to the tensor
// core (A_hi once more for either half): 2432 cycles at 128 bytes a cycle, for 1536 of tensor-core work;
// 2335 were measured at 2048^3, so not all of the tensor core's reads cost what this counts.
// With 128 columns the instructions of the converters and the epilogue (with A in tensor memory the port
// has 1088 cycles to do, and the tensor core 768).  Two rules of the code below matter as much:
// sums are added two at a time (packed), and whatever is live in the loop over the stages besides the 128
// sums is little; a variant that kept all sums in registers up to the end of the tile spilled some
// of them and took 81 us for 2048^3 instead of 53.  Measured per call (us, 256 columns / 128): 2048^3
// 52.8 / 61.0, 2048 x 1024 x 2048 40.9 / 34.1, complex 1280 x 960 x 1500 57.8 / 63.1, 512 x complex 256^3
// 234 / 339 (beta = 0.5 309 / 420), 512 x 256^3 83 / 105, TF32TCEC 107 / 147, 256 x 256 x 65536 51 / 49.
// One team of eight converter warps, A in shared memory and sums added one by one took 53.3 and
// 47.8 us for the first two in their better width.
//
// Work distribution: work_list.cuh.  What is left over from whole waves (total mod clusters, or
// everything when there are fewer tiles than clusters) can be cut along K; piece_fixup.cu then
// adds the pieces and runs their epilogue.
//
// Threads: 896 = warp 0 TMA producer, warp 1 TMEM allocation + MMA issue (even CTA), warps 2-3
// idle, warps 4-11 drain / epilogue, warps 12-27 converters.  Launched with 72 registers per
// thread = 64512, which setmaxnreg deals out again (StreamCfg); the sum is the same, so the increase
// can always be served.
//
// Barriers (per CTA, same shared-memory offsets; "leader" = even CTA):
//   raw_full[r]    1 arrival (producer, expect_tx) + TMA bytes      own CTA
//   raw_empty[r]   8 or 16 arrivals, the slot's converter warps    own CTA
//   full[s]        leader's only: the converter warps of both CTAs
//   empty[s]       tcgen05.commit multicast from the leader         both CTAs
//   d_full[b]      the same, after hi*hi of one half of the columns
//   d_empty[b]     leader's only: 8 arrivals, the epilogue warps of that half in both CTAs
//   d1_empty       leader's only: 16 arrivals, the epilogue warps of both CTAs
// A wait tells phases apart by one bit, so whoever waits on a barrier looks at each of its phases, and
// before the next one can end: one that passed over a phase could take the phase before it for the one
// it wants, and nothing says that arrivals on different barriers are seen in the order they were sent.
// So the numbers of stages and accumulators are even (each belongs to one team, one half of the columns),
// and where the number of raw slots is not, every converter warp has a share of each slot.  Every
// wait is bounded; no TMA multicast is used.
#include "epilogue.cuh"
#include "gemm_common.cuh"
#include "ptx.cuh"
#include "split_math.cuh"
#include "work_list.cuh"

#include <mutex>

namespace cumpsgemm_b200 {
namespace {

constexpr int BM_CTA = 128;
constexpr int ROW_BYTES = kGemmRowBytes;
constexpr int SLOT_K = 32; // k values of a raw slot (128 bytes of FP32)
constexpr int NUM_THREADS = 896;
constexpr int FIRST_EPI_WARP = 4, NUM_EPI_WARPS = 8;
constexpr int FIRST_CVT_WARP = 12, CVT_TEAMS = 2, TEAM_WARPS = 8;
constexpr int LAUNCH_REGS = 72;
constexpr uint32_t C_PREFETCH_LEAD = 8; // stages between the L2 prefetch of C and its use

// Raw layouts a converter can read (values of StreamGemmArgs::layout_a / layout_b).
enum RawLayout : int {
  kRawK = 0,    // element (r, k) at [r * ld + k]: K contiguous, 128-byte rows, 128-byte swizzle
  kRawR = 1,    // element (r, k) at [k * ld + r]: rows contiguous
  kRawCplxAR = 2, // complex A, op N: rows contiguous
  kRawCplxAK = 3, // complex A, op T / C: K contiguous, swizzled
  kRawCplxBR = 4  // complex B, op T / C: rows contiguous   (complex B, op N is kRawK)
};

struct StreamParams {
  float *c;
  const DynParams *dyn;
  int *status;
  float *partial; // [cluster][2][CTA rank][BN columns][128 rows]
  unsigned long long *debug;
  uint64_t ldc, stride_c;
  uint32_t m, n;
  uint32_t tiles_m, tiles_n;
  float alpha_r, alpha_i, beta_r, beta_i;
  WorkPlan w;
  uint8_t layout_a, layout_b;
  uint8_t flags; // k* below
};
static_assert(sizeof(StreamParams) <= 128, "kernel parameter structs stay within 128 bytes");
constexpr uint32_t kIsComplex = 1, kConjA = 2, kConjB = 4, kBatchA = 8, kBatchB = 16,
                   kDirectStores = 32;

// CG: CTAs of a cluster, 2 (a pair shares a 256-row tile) or 1 (128 rows).
template <int BN, int CG> struct StreamCfg {
  static constexpr int B_ROWS = BN / CG;         // rows of op(B) per CTA: two blocks of HALF_ROWS,
  static constexpr int HALF_ROWS = BN / 2 / CG;  // one for each half of the tile's columns
  // 128 columns: A in tensor memory.  256: the accumulators take all of it, and A is in shared memory.
  static constexpr bool A_IN_TMEM = BN == 128;
  static constexpr int A_TILE = BM_CTA * ROW_BYTES, B_TILE = B_ROWS * ROW_BYTES;
  static constexpr int A_BYTES = A_IN_TMEM ? 0 : 2 * A_TILE; // of a stage: hi, lo; those of B behind it
  static constexpr int STAGE_BYTES = A_BYTES + 2 * B_TILE;
  static constexpr int STAGES = 2;
  static constexpr int RAW_A = BM_CTA * SLOT_K * 4;
  static constexpr int RAW_HALF_B = HALF_ROWS * SLOT_K * 4;
  static constexpr int RAW_BYTES = RAW_A + 2 * RAW_HALF_B;
  static constexpr int RAW_SLOTS = (BN == 256) ? 3 : (CG == 1) ? 4 : 6;
  // An even number of slots: the two converter teams take them in turn; otherwise every warp has a
  // share of each.
  static constexpr int SLOT_TEAMS = (RAW_SLOTS % 2 == 0) ? 2 : 1;
  static constexpr int SLOT_WARPS = CVT_TEAMS / SLOT_TEAMS * TEAM_WARPS;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + RAW_SLOTS * RAW_BYTES + 1024 + 256;
  // Tensor memory: accumulators for hi*hi of half a tile's columns each, the corrections of the whole
  // tile, then A, 64 columns per stage (hi, lo)
  static constexpr uint32_t D_BUFS = (BN == 256) ? 2 : 4;
  static constexpr uint32_t D1_COL = D_BUFS * (BN / 2), A_COL = D1_COL + BN;
  static constexpr int REGS_EPI = (BN == 256) ? 152 : 112;
  static constexpr int REGS_CVT = (BN == 256) ? 40 : 48;
  static constexpr int REGS_REST = (BN == 256) ? 40 : 72;
  static_assert(256 * REGS_EPI + 512 * REGS_CVT + 128 * REGS_REST <= NUM_THREADS * LAUNCH_REGS,
                "register re-allocation must fit what the CTA was launched with");
  static_assert(REGS_EPI >= LAUNCH_REGS && REGS_CVT <= LAUNCH_REGS && REGS_REST <= LAUNCH_REGS,
                "setmaxnreg.inc goes up, setmaxnreg.dec down: anything else is an illegal instruction");
  // Barriers behind the raw slots, as byte offsets: eight bytes each
  static constexpr uint32_t RAW_FULL = 0, RAW_EMPTY = 8 * RAW_SLOTS, FULL = RAW_EMPTY + 8 * RAW_SLOTS,
                            EMPTY = FULL + 8 * STAGES, D_FULL = EMPTY + 8 * STAGES,
                            D_EMPTY = D_FULL + 8 * D_BUFS, D1_EMPTY = D_EMPTY + 8 * D_BUFS,
                            TMEM_PTR = D1_EMPTY + 8, ABORT = TMEM_PTR + 4;
  static_assert(ABORT + 4 <= 256, "barriers");
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
  static_assert(STAGES % 2 == 0 && D_BUFS % 2 == 0, "a stage belongs to one team, a buffer to one half");
  static_assert(A_COL + (A_IN_TMEM ? STAGES * 64 : 0) <= 512, "tensor memory");
};
constexpr uint32_t A_STAGE_COLS = 64, A_LO_COLS = 32, TMEM_COLS = 512;

struct TileCoord {
  uint32_t batch;
  int m0; // first row of this CTA's 128 rows
  int n0; // first column of the pair's BN columns
};

template <int BN, int CG>
__device__ __forceinline__ TileCoord tile_coord(uint32_t tile, const StreamParams &p,
                                                uint32_t rank) {
  const TilePos t = tile_raster(tile, p.tiles_m, p.tiles_n);
  TileCoord c;
  c.batch = t.batch;
  c.m0 = static_cast<int>((t.tm * CG + rank) * BM_CTA);
  c.n0 = static_cast<int>(t.tn * BN);
  return c;
}

// One product over 32 bytes of K: step ks of the 128 bytes that `a` and `b` begin (a: a tensor-memory
// address or, like b, a descriptor).
template <int KIND, int CG, typename A>
__device__ __forceinline__ void mma(uint32_t d, A a, uint64_t b, int ks, uint32_t idesc, uint32_t acc) {
  if constexpr (sizeof(A) == 4) {
    if constexpr (KIND == 0) ptx::mma_f16_ts<CG>(d, a + 8 * ks, b + 2 * ks, idesc, acc);
    else ptx::mma_tf32_ts<CG>(d, a + 8 * ks, b + 2 * ks, idesc, acc);
  } else {
    static_assert(CG == 2, "A in shared memory: pairs only");
    if constexpr (KIND == 0) ptx::mma_f16_ss_pair(d, a + 2 * ks, b + 2 * ks, idesc, acc);
    else ptx::mma_tf32_ss_pair(d, a + 2 * ks, b + 2 * ks, idesc, acc);
  }
}
template <int CG> __device__ __forceinline__ void commit(uint32_t bar) {
  if constexpr (CG == 2) ptx::tc_commit_pair(bar, 0x3);
  else ptx::tc_commit(bar);
}

// ---------------------------------------------------------------- converters
// One warp converts 32 rows (lane = row) of one operand: of every raw slot JOBS groups of eight
// consecutive k values, of which a slot has four.  Each layout has a loop of its own: a warp runs
// one of them, so the code it cycles through stays small (a first version chose the layout per
// group inside one unrolled loop: 5,000 cycles per stage, most of them instruction fetches and
// spills).  Shared-memory accesses are free of bank conflicts: K-contiguous tiles are swizzled by
// TMA (eight lanes of a 16-byte access hit eight different 16-byte positions), row-contiguous
// ones are read 4 or 8 bytes per lane along the row.  Row r's 16-byte chunk q of a swizzled
// tile is at r * 128 + ((q ^ (r & 7)) << 4), i.e. at (r * 128 + ((r & 7) << 4)) ^ (q << 4).
struct ConverterState {
  uint32_t bars;        // shared address of this CTA's barriers
  uint32_t bars_leader; // shared::cluster address of the leader's
  uint32_t raw;         // shared address of slot 0's raw tile
  uint32_t row;         // this lane's row of the raw tile
  uint32_t dst;         // stage 0's hi values of the lane's row: shared address of the (swizzled) row,
                        // or the warp's tensor-memory address
  uint32_t team;
  uint32_t group0;      // first of the warp's 8-k groups in a slot
  float scale;
  uint32_t conj_mask;   // sign bit if the operand is conjugated, else 0
  int *status;
};

__device__ __forceinline__ float flip_sign(float x, uint32_t mask) {
  return __uint_as_float(__float_as_uint(x) ^ mask);
}

// Eight consecutive expanded k values (group g of the slot) of the lane's row; `raw` is the slot's
// tile, lane_addr the lane's precomputed address inside it.
// Complex A expands to rows (2i, 2i+1) x columns (2l, 2l+1) = [[re, -im], [im, re]].
template <int LAYOUT, int ROWS>
__device__ __forceinline__ void load_raw8(uint32_t lane_addr, uint32_t g, const ConverterState &st,
                                          float (&v)[8]) {
  if constexpr (LAYOUT == kRawK) {
    const float4 x = ld_shared_f4(lane_addr ^ ((2u * g) << 4));
    const float4 y = ld_shared_f4(lane_addr ^ ((2u * g + 1u) << 4));
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
    v[4] = y.x, v[5] = y.y, v[6] = y.z, v[7] = y.w;
  } else if constexpr (LAYOUT == kRawR) {
#pragma unroll
    for (uint32_t e = 0; e < 8; ++e) v[e] = ld_shared_f1(lane_addr + (8u * g + e) * ROWS * 4u);
  } else if constexpr (LAYOUT == kRawCplxBR) {
#pragma unroll
    for (uint32_t e = 0; e < 4; ++e) {
      const float2 x = ld_shared_f2(lane_addr + (4u * g + e) * ROWS * 8u);
      v[2 * e] = x.x;
      v[2 * e + 1] = flip_sign(x.y, st.conj_mask);
    }
  } else {
    float2 x[4];
    if constexpr (LAYOUT == kRawCplxAR) {
#pragma unroll
      for (uint32_t e = 0; e < 4; ++e) x[e] = ld_shared_f2(lane_addr + (4u * g + e) * ROWS * 4u);
    } else {
#pragma unroll
      for (uint32_t h = 0; h < 2; ++h) {
        const float4 y = ld_shared_f4(lane_addr ^ ((2u * g + h) << 4));
        x[2 * h] = make_float2(y.x, flip_sign(y.y, st.conj_mask));
        x[2 * h + 1] = make_float2(y.z, flip_sign(y.w, st.conj_mask));
      }
    }
    const bool im_row = (st.row & 1u) != 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[2 * e] = im_row ? x[e].y : x[e].x;
      v[2 * e + 1] = im_row ? x[e].x : -x[e].y;
    }
  }
}

// Splits eight consecutive k values and stores them at 8-k group kc of the stage: A in tensor
// memory where it goes there, else in shared memory.
template <int KIND, int LO_DELTA, bool TO_TMEM>
__device__ __forceinline__ void split_store8(const float (&v)[8], uint32_t dst, uint32_t kc) {
  if constexpr (TO_TMEM && KIND == 1) {
    uint32_t h[8], l[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) split_tf32(v[t], h[t], l[t]);
    ptx::tmem_st_32x32b_x8(dst + 8u * kc, h);
    ptx::tmem_st_32x32b_x8(dst + A_LO_COLS + 8u * kc, l);
    return;
  }
  constexpr int VECS = (KIND == 0) ? 1 : 2; // vectors of four 32-bit words
#pragma unroll
  for (uint32_t g = 0; g < VECS; ++g) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      if constexpr (KIND == 0) split2_mixed(v[2 * t], v[2 * t + 1], h[t], l[t]);
      else split_tf32(v[4 * g + t], h[t], l[t]);
    }
    const uint32_t q = VECS * kc + g;
    if constexpr (TO_TMEM) {
      ptx::tmem_st_32x32b_x4(dst + 4u * q, h);
      ptx::tmem_st_32x32b_x4(dst + A_LO_COLS + 4u * q, l);
    } else {
      const uint32_t addr = dst ^ (q << 4);
      st_shared_v4(addr, h[0], h[1], h[2], h[3]);
      st_shared_v4(addr + LO_DELTA, l[0], l[1], l[2], l[3]);
    }
  }
}

template <int KIND, int BN, int CG, int LAYOUT, int ROWS, int JOBS, bool IS_A>
__device__ __forceinline__ void convert_loop(uint32_t total_stages, ConverterState &st) {
  using Cfg = StreamCfg<BN, CG>;
  constexpr uint32_t SLOTS_PER_STAGE = (KIND == 0) ? 2 : 1;
  constexpr bool TO_TMEM = IS_A && Cfg::A_IN_TMEM;
  constexpr bool IN_TURN = Cfg::SLOT_TEAMS == 2;
  // stages from a warp's slot to its next one (in turn: a team's); a stage of two slots is passed in two
  constexpr uint32_t STAGE_STEP = IN_TURN ? 2 / SLOTS_PER_STAGE : 1;
  const uint32_t r = st.row;
  const int lane = static_cast<int>(threadIdx.x & 31);
  uint32_t lane_raw;
  if constexpr (LAYOUT == kRawK) lane_raw = st.raw + r * 128u + ((r & 7u) << 4);
  else if constexpr (LAYOUT == kRawR) lane_raw = st.raw + r * 4u;
  else if constexpr (LAYOUT == kRawCplxBR) lane_raw = st.raw + r * 8u;
  else if constexpr (LAYOUT == kRawCplxAR) lane_raw = st.raw + (r >> 1) * 8u;
  else lane_raw = st.raw + (r >> 1) * 128u + (((r >> 1) & 7u) << 4);
  const bool scaled = st.scale != 1.f;
  uint32_t rs = IN_TURN ? st.team : 0u, rph = 0;
  // index in the stream of stages; the stage, and parity of the release of its previous use
  uint32_t i = (KIND == 1 && IN_TURN) ? st.team : 0u;
  uint32_t s = i, e_ph = 1;
  auto next = [&]() {
    i += STAGE_STEP;
    s += STAGE_STEP;
    if (s >= Cfg::STAGES) {
      s -= Cfg::STAGES;
      e_ph ^= 1u;
    }
  };
  uint32_t second = (KIND == 0 && IN_TURN) ? st.team : 0u; // the slot is the second of its stage
#pragma unroll 1
  while (i < total_stages) {
    if (!ptx::warp_agrees(ptx::mbar_wait_s(st.bars + Cfg::RAW_FULL + 8u * rs, rph,
                                           st.bars + Cfg::ABORT, st.status, ptx::kErrWaitFull) &&
                          ptx::mbar_wait_s(st.bars + Cfg::EMPTY + 8u * s, e_ph, st.bars + Cfg::ABORT,
                                           st.status, ptx::kErrWaitEmpty)))
      return;
    if constexpr (TO_TMEM) ptx::tc_fence_after();
    const uint32_t raw_addr = lane_raw + rs * Cfg::RAW_BYTES;
    const uint32_t dst = st.dst + s * (TO_TMEM ? A_STAGE_COLS : static_cast<uint32_t>(Cfg::STAGE_BYTES));
#pragma unroll
    for (int j = 0; j < JOBS; ++j) {
      float v[8];
      load_raw8<LAYOUT, ROWS>(raw_addr, st.group0 + j, st, v);
      if (scaled) {
#pragma unroll
        for (int t = 0; t < 8; ++t) v[t] *= st.scale;
      }
      split_store8<KIND, IS_A ? Cfg::A_TILE : Cfg::B_TILE, TO_TMEM>(v, dst, 4u * second + st.group0 + j);
    }
    if constexpr (TO_TMEM) {
      ptx::tmem_st_wait();
      ptx::tc_fence_before();
    } else {
      fence_proxy_async_shared();
    }
    // every value of the slot has been read: it may be refilled
    __syncwarp();
    if (lane == 0) {
      ptx::mbar_arrive(st.bars + Cfg::RAW_EMPTY + 8u * rs);
      ptx::mbar_arrive_cluster(st.bars_leader + Cfg::FULL + 8u * s);
    }
    rs += Cfg::SLOT_TEAMS;
    if (rs >= Cfg::RAW_SLOTS) {
      rs -= Cfg::RAW_SLOTS;
      rph ^= 1u;
    }
    if (KIND == 0 && !IN_TURN) {
      second ^= 1u;
      if (second != 0) continue;
    }
    next();
  }
  // the issuer's last commits arrive on this CTA's barriers: it must not be gone by then (TF32TCEC:
  // each team waits for those that it would go on with)
  for (; i < total_stages + Cfg::STAGES; next()) {
    if (i < Cfg::STAGES) continue; // (nothing was in it)
    if (!ptx::mbar_wait_s(st.bars + Cfg::EMPTY + 8u * s, e_ph, st.bars + Cfg::ABORT, st.status,
                          ptx::kErrWaitEmpty))
      return;
  }
}

template <int KIND, int BN, int CG>
__device__ __forceinline__ void stream_body(const CUtensorMap &map_a, const CUtensorMap &map_b,
                                            const StreamParams &p) {
  using Cfg = StreamCfg<BN, CG>;
  constexpr int STAGES = Cfg::STAGES, RAW_SLOTS = Cfg::RAW_SLOTS;
  constexpr int K_STEPS = ROW_BYTES / 32;
  constexpr uint32_t SLOTS_PER_STAGE = (KIND == 0) ? 2 : 1;
  constexpr uint32_t STAGES_PER_UNIT = (KIND == 0) ? 1 : 2;
  constexpr uint32_t IDESC = ptx::make_idesc(KIND == 0 ? 0 : 2, CG * BM_CTA, BN),
                     IDESC_HALF = ptx::make_idesc(KIND == 0 ? 0 : 2, CG * BM_CTA, BN / 2);
  constexpr float LO_SCALE_INV = (KIND == 0) ? (1.f / 2048.f) : 1.f;
  constexpr int CPT = BN / 2; // accumulator columns per epilogue thread

  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t *raw_smem = smem + STAGES * Cfg::STAGE_BYTES;
  const uint32_t bars = ptx::smem_u32(raw_smem + RAW_SLOTS * Cfg::RAW_BYTES);
  const uint32_t abort_flag = bars + Cfg::ABORT;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = (CG == 2) ? ptx::cluster_ctarank() : 0u;
  const bool leader = (rank == 0);
  const uint32_t cluster_id = blockIdx.x / CG;
  const uint32_t num_clusters = gridDim.x / CG;

  if (threadIdx.x == 0) {
    for (uint32_t r = 0; r < RAW_SLOTS; ++r) {
      ptx::mbar_init(bars + Cfg::RAW_FULL + 8u * r, 1);
      ptx::mbar_init(bars + Cfg::RAW_EMPTY + 8u * r, Cfg::SLOT_WARPS);
    }
    for (uint32_t s = 0; s < STAGES; ++s) {
      ptx::mbar_init(bars + Cfg::FULL + 8u * s, CG * SLOTS_PER_STAGE * Cfg::SLOT_WARPS);
      ptx::mbar_init(bars + Cfg::EMPTY + 8u * s, 1);
    }
    for (uint32_t b = 0; b < Cfg::D_BUFS; ++b) {
      ptx::mbar_init(bars + Cfg::D_FULL + 8u * b, 1);
      ptx::mbar_init(bars + Cfg::D_EMPTY + 8u * b, CG * NUM_EPI_WARPS / 2);
    }
    ptx::mbar_init(bars + Cfg::D1_EMPTY, CG * NUM_EPI_WARPS);
    st_shared_u32(abort_flag, 0u);
    ptx::mbar_init_fence();
    ptx::prefetch_tensormap(&map_a);
    ptx::prefetch_tensormap(&map_b);
  }
  if (warp == 1) {
    if constexpr (CG == 2) {
      ptx::tmem_alloc_pair(bars + Cfg::TMEM_PTR, TMEM_COLS);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(bars + Cfg::TMEM_PTR, TMEM_COLS);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if constexpr (CG == 2) { // both CTAs' barriers must exist before any remote arrive
    ptx::cluster_arrive();
    ptx::cluster_wait();
  }
  ptx::tc_fence_after();
  constexpr uint32_t tmem_base = 0; // all of tensor memory
  // launched behind the previous kernel of the stream (programmatic serialization): from here
  // on global memory is read and written
  ptx::griddep_wait();
  const bool dbg = (p.debug != nullptr);

  if (warp < FIRST_EPI_WARP) {
    ptx::setmaxnreg_dec<Cfg::REGS_REST>();
    if (warp == 0) {
      if (ptx::elect_one()) {
        // ============================================================== TMA producer (both CTAs)
        const bool a_k = p.layout_a == kRawK || p.layout_a == kRawCplxAK;
        const bool a_cplx = p.layout_a == kRawCplxAR || p.layout_a == kRawCplxAK;
        const bool b_k = p.layout_b == kRawK;
        const bool b_cplx = p.layout_b == kRawCplxBR;
        // coordinate steps per slot: x for K-contiguous operands, y for row-contiguous ones
        const int a_dy = a_cplx ? SLOT_K / 2 : SLOT_K;
        const int b_dy = b_cplx ? SLOT_K / 2 : SLOT_K;
        const uint32_t bytes = (a_cplx ? Cfg::RAW_A / 2 : Cfg::RAW_A) +
                               static_cast<uint32_t>(Cfg::B_ROWS * SLOT_K * 4);
        uint32_t s = 0, ph = 0;
        bool ok = true;
        WorkList list(p.w, cluster_id, num_clusters);
        WorkItem x;
        while (ok && list.next(p.w, x)) {
          const TileCoord tc = tile_coord<BN, CG>(x.tile, p, rank);
          const int b_row = tc.n0 + static_cast<int>(rank) * Cfg::HALF_ROWS;
          const int t0 = static_cast<int>(2u * x.u0);
          int ax = a_k ? t0 * SLOT_K : tc.m0;
          int ay = a_k ? (a_cplx ? tc.m0 >> 1 : tc.m0) : t0 * a_dy;
          int bx = b_k ? t0 * SLOT_K : (b_cplx ? 2 * b_row : b_row);
          int by = b_k ? b_row : t0 * b_dy;
          // the rows for the second half of the tile's columns
          const int bx2 = b_k ? 0 : (b_cplx ? BN : BN / 2), by2 = b_k ? BN / 2 : 0;
          const int az = (p.flags & kBatchA) ? static_cast<int>(tc.batch) : 0;
          const int bz = (p.flags & kBatchB) ? static_cast<int>(tc.batch) : 0;
          for (uint32_t t = 0; t < 2u * x.un; ++t) {
            ok = ptx::mbar_wait_s(bars + Cfg::RAW_EMPTY + 8u * s, ph ^ 1u, abort_flag, p.status,
                                ptx::kErrWaitEmpty);
            if (!ok) break;
            const uint32_t fb = bars + Cfg::RAW_FULL + 8u * s;
            ptx::mbar_arrive_expect_tx(fb, bytes);
            const uint32_t dst = ptx::smem_u32(raw_smem + s * Cfg::RAW_BYTES);
            ptx::tma_load_3d(dst, &map_a, fb, ax, ay, az);
            ptx::tma_load_3d(dst + Cfg::RAW_A, &map_b, fb, bx, by, bz);
            ptx::tma_load_3d(dst + Cfg::RAW_A + Cfg::RAW_HALF_B, &map_b, fb, bx + bx2,
                             by + by2, bz);
            if (a_k) ax += SLOT_K;
            else ay += a_dy;
            if (b_k) bx += SLOT_K;
            else by += b_dy;
            if (++s == RAW_SLOTS) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
      }
    } else if (warp == 1 && leader) {
      if (ptx::elect_one()) {
        // ============================================================== MMA issuer (leader only)
        const uint64_t desc0 = ptx::make_kmajor_desc<ROW_BYTES>(ptx::smem_u32(smem));
        constexpr uint64_t kStage = Cfg::STAGE_BYTES >> 4, kLo = Cfg::B_TILE >> 4,
                           kHalf = (Cfg::HALF_ROWS * ROW_BYTES) >> 4;
        uint32_t s = 0, ph = 0, b = 0, d_ph = 1, d1_ph = 1;
        bool ok = true;
        auto wait_timed = [&](uint32_t bar, uint32_t parity, int code, uint32_t &cycles) {
          const uint32_t t0 = dbg ? static_cast<uint32_t>(clock()) : 0u;
          const bool r = ptx::mbar_wait_s(bar, parity, abort_flag, p.status, code);
          if (dbg) cycles += static_cast<uint32_t>(clock()) - t0;
          return r;
        };
        uint32_t dbg_wait = 0, dbg_wait2 = 0;
        const long long dbg_t0 = dbg ? clock64() : 0;
        WorkList list(p.w, cluster_id, num_clusters);
        WorkItem x;
        while (ok && list.next(p.w, x)) {
          const uint32_t kbn = x.un * STAGES_PER_UNIT;
          for (uint32_t kb = 0; kb < kbn; ++kb) {
            ok = wait_timed(bars + Cfg::FULL + 8u * s, ph, ptx::kErrWaitFull, dbg_wait);
            if (!ok) break;
            // (the item before this one: its corrections must have been read)
            if (kb == 0)
              ok = wait_timed(bars + Cfg::D1_EMPTY, d1_ph, ptx::kErrWaitD1Empty, dbg_wait2);
            if (!ok) break;
            ptx::tc_fence_after();
            const uint64_t stage = desc0 + s * kStage;
            const uint64_t b_hi = stage + (Cfg::A_BYTES >> 4), b_lo = b_hi + kLo;
            const auto a_hi = [&]() {
              if constexpr (Cfg::A_IN_TMEM) return tmem_base + Cfg::A_COL + s * A_STAGE_COLS;
              else return stage;
            }();
            const auto a_lo = a_hi + (Cfg::A_IN_TMEM ? A_LO_COLS : Cfg::A_TILE >> 4);
            // The corrections come first: behind them the sums of the stage before are drained.
#pragma unroll
            for (int ks = 0; ks < K_STEPS; ++ks)
              mma<KIND, CG>(tmem_base + Cfg::D1_COL, a_lo, b_hi, ks, IDESC, (ks > 0 || kb > 0) ? 1u : 0u);
#pragma unroll
            for (int ks = 0; ks < K_STEPS; ++ks)
              mma<KIND, CG>(tmem_base + Cfg::D1_COL, a_hi, b_lo, ks, IDESC, 1u);
            // the previous sums of these columns must have been drained (at the end of an item:
            // stored)
            auto next_buffer = [&]() {
              ok = ok && wait_timed(bars + Cfg::D_EMPTY + 8u * b, d_ph, ptx::kErrWaitD0Empty, dbg_wait2);
              ptx::tc_fence_after();
              return tmem_base + b * CPT;
            };
            auto filled = [&]() {
              commit<CG>(bars + Cfg::D_FULL + 8u * b);
              if (++b == Cfg::D_BUFS) {
                b = 0;
                d_ph ^= 1u;
              }
            };
#pragma unroll
            for (uint32_t g = 0; g < 2; ++g) {
              const uint32_t d = next_buffer();
              if (!ok) break;
#pragma unroll
              for (int ks = 0; ks < K_STEPS; ++ks)
                mma<KIND, CG>(d, a_hi, b_hi + g * kHalf, ks, IDESC_HALF, ks > 0 ? 1u : 0u);
              filled(); // (behind an item's last products this tells of its corrections too)
            }
            if (!ok) break;
            commit<CG>(bars + Cfg::EMPTY + 8u * s);
            if (++s == STAGES) {
              s = 0;
              ph ^= 1u;
            }
          }
          d1_ph ^= 1u;
        }
        if (dbg) {
          atomicAdd(p.debug + 0, static_cast<unsigned long long>(dbg_wait));
          atomicAdd(p.debug + 1, static_cast<unsigned long long>(dbg_wait2));
          atomicAdd(p.debug + 4, static_cast<unsigned long long>(clock64() - dbg_t0));
          atomicAdd(p.debug + 5, 1ull);
        }
      }
    }
  } else if (warp >= FIRST_CVT_WARP) {
    // ================================================================ converters (both CTAs)
    ptx::setmaxnreg_dec<Cfg::REGS_CVT>();
    // Two teams of eight warps take the raw slots in turn, or (three slots) half of each slot's groups.
    // In a team warps 0-3 convert the four 32-row blocks of A, warps 4-7 those of B (64 rows: two
    // warps to each of its two blocks, half of a slot's groups each).
    constexpr int A_JOBS = (Cfg::SLOT_TEAMS == 2) ? 4 : 2;
    constexpr int B_JOBS = (Cfg::B_ROWS == 128) ? A_JOBS : 2;
    static_assert(Cfg::B_ROWS == 128 || Cfg::SLOT_TEAMS == 2, "who converts what");
    const uint32_t cw = static_cast<uint32_t>(warp - FIRST_CVT_WARP) & 7u;
    const bool for_a = cw < 4;
    // the converters see a plain stream of stages; only its length depends on the work items
    uint32_t total_stages = 0;
    {
      WorkList list(p.w, cluster_id, num_clusters);
      WorkItem x;
      while (list.next(p.w, x)) total_stages += x.un * STAGES_PER_UNIT;
    }
    ConverterState st;
    st.bars = bars;
    st.bars_leader = ptx::map_to_cta(bars, 0);
    st.team = static_cast<uint32_t>(warp - FIRST_CVT_WARP) >> 3;
    st.raw = ptx::smem_u32(raw_smem);
    if (for_a) {
      st.row = cw * 32u + lane;
      st.group0 = 0;
      if constexpr (Cfg::A_IN_TMEM) st.dst = tmem_base + Cfg::A_COL + ((cw * 32u) << 16);
      else st.dst = ptx::smem_u32(smem) + st.row * 128u + ((st.row & 7u) << 4);
    } else {
      const uint32_t half = (cw - 4u) >> 1; // of the tile's columns
      st.row = (Cfg::B_ROWS == 128 ? (cw & 1u) * 32u : 0u) + lane;
      st.group0 = (Cfg::B_ROWS == 128) ? 0u : 2u * (cw & 1u);
      st.raw += Cfg::RAW_A + half * Cfg::RAW_HALF_B;
      const uint32_t r = half * Cfg::HALF_ROWS + st.row;
      st.dst = ptx::smem_u32(smem) + Cfg::A_BYTES + r * 128u + ((r & 7u) << 4);
    }
    if (Cfg::SLOT_TEAMS == 1) st.group0 = 2u * st.team;
    st.scale = 1.f;
    if (p.dyn != nullptr) st.scale = for_a ? p.dyn->scale_a : p.dyn->scale_b;
    st.conj_mask = (p.flags & (for_a ? kConjA : kConjB)) ? 0x80000000u : 0u;
    st.status = p.status;
    if (for_a) {
      switch (p.layout_a) {
      case kRawK:
        convert_loop<KIND, BN, CG, kRawK, BM_CTA, A_JOBS, true>(total_stages, st);
        break;
      case kRawR:
        convert_loop<KIND, BN, CG, kRawR, BM_CTA, A_JOBS, true>(total_stages, st);
        break;
      case kRawCplxAR:
        convert_loop<KIND, BN, CG, kRawCplxAR, BM_CTA, A_JOBS, true>(total_stages, st);
        break;
      default:
        convert_loop<KIND, BN, CG, kRawCplxAK, BM_CTA, A_JOBS, true>(total_stages, st);
        break;
      }
    } else {
      switch (p.layout_b) {
      case kRawK:
        convert_loop<KIND, BN, CG, kRawK, Cfg::HALF_ROWS, B_JOBS, false>(total_stages, st);
        break;
      case kRawR:
        convert_loop<KIND, BN, CG, kRawR, Cfg::HALF_ROWS, B_JOBS, false>(total_stages, st);
        break;
      default:
        convert_loop<KIND, BN, CG, kRawCplxBR, Cfg::HALF_ROWS, B_JOBS, false>(total_stages, st);
        break;
      }
    }
  } else {
    // ================================================================ drain + epilogue (both CTAs)
    ptx::setmaxnreg_inc<Cfg::REGS_EPI>();
    // Few registers are left beside the running sums: what the loop over the stages keeps is little,
    // and the rest is worked out where it is needed.
    const uint32_t half = static_cast<uint32_t>((warp - FIRST_EPI_WARP) >> 2); // of the columns
    const uint32_t t_base = tmem_base + ((static_cast<uint32_t>(warp & 3) * 32u) << 16);

    uint32_t b = half, d_ph = 0; // accumulator and parity of the next stage
    auto arrive = [&](uint32_t bar) { // at the leader
      ptx::tc_fence_before();
      __syncwarp();
      if (ptx::elect_one()) ptx::mbar_arrive_cluster(ptx::map_to_cta(bars + bar, 0));
      __syncwarp();
    };
    auto give_back = [&]() {
      arrive(Cfg::D_EMPTY + 8u * b);
      b += 2u;
      if (b >= Cfg::D_BUFS) {
        b -= Cfg::D_BUFS;
        d_ph ^= 1u;
      }
    };
    // beta != 0: pull this warp's part of a C tile into L2 before the epilogue reads it
    auto prefetch_c = [&](uint32_t tile) {
      const TileCoord tc = tile_coord<BN, CG>(opaque(tile), p, rank);
      const uint32_t row = static_cast<uint32_t>(tc.m0) + static_cast<uint32_t>(warp & 3) * 32u;
      const float *cp = p.c + static_cast<uint64_t>(tc.batch) * p.stride_c + row;
#pragma unroll 1
      for (int q = 0; q < CPT / 32; ++q) {
        const uint32_t col =
            static_cast<uint32_t>(tc.n0) +
            static_cast<uint32_t>(((warp - FIRST_EPI_WARP) >> 2) * CPT + q * 32 + lane);
        if (col < p.n && row < p.m) ptx::prefetch_l2(cp + static_cast<uint64_t>(col) * p.ldc);
      }
    };
    bool ok = true;
    WorkList list(p.w, cluster_id, num_clusters);
    WorkItem x;
    while (ok && list.next(p.w, x)) {
      uint32_t left = x.un * STAGES_PER_UNIT; // stages to drain
      if (left < C_PREFETCH_LEAD && (p.beta_r != 0.f || p.beta_i != 0.f)) prefetch_c(x.tile);
      unsigned long long acc[CPT / 2];
#pragma unroll
      for (int i = 0; i < CPT / 2; ++i) acc[i] = 0ull;

#pragma unroll 1
      while (true) {
        if (left == C_PREFETCH_LEAD && (p.beta_r != 0.f || p.beta_i != 0.f)) prefetch_c(x.tile);
        ok = ptx::warp_agrees(ptx::mbar_wait_s(bars + Cfg::D_FULL + 8u * b, d_ph, abort_flag, p.status,
                                               ptx::kErrWaitD0Full));
        if (!ok) break;
        ptx::tc_fence_after();
        if (--left == 0) break; // the last ones are added below
        drain_pairs<CPT>(t_base + b * CPT, acc);
        give_back();
      }
      if (!ok) break;
      // (a pair's columns come half from one CTA's rows of op(B), half from the other's)
      const uint32_t t_cor = t_base + Cfg::D1_COL + half * Cfg::HALF_ROWS;
      const uint32_t t_sums = t_base + b * CPT;
      if (BN == 128 && (p.flags & kDirectStores)) {
        // Many short tiles per cluster, C not read: stores straight from the registers.  That is
        // long code, but it stays in the instruction cache from tile to tile, and the columns go back to
        // the issuer before the stores instead of after them.
        drain_pairs<CPT>(t_sums, acc);
        add_corrections_to_pairs<CPT, Cfg::HALF_ROWS, Cfg::B_ROWS>(t_cor, acc, LO_SCALE_INV);
        arrive(Cfg::D1_EMPTY);
        give_back();
        float sums[CPT];
#pragma unroll
        for (int i = 0; i < CPT / 2; ++i)
          asm("mov.b64 {%0, %1}, %2;" : "=f"(sums[2 * i]), "=f"(sums[2 * i + 1]) : "l"(acc[i]));
        const TileCoord tc = tile_coord<BN, CG>(opaque(x.tile), p, rank);
        const uint32_t row = static_cast<uint32_t>(tc.m0) + static_cast<uint32_t>(warp & 3) * 32u +
                             static_cast<uint32_t>(lane);
        const uint32_t col0 = static_cast<uint32_t>(tc.n0) +
                              static_cast<uint32_t>((warp - FIRST_EPI_WARP) >> 2) * CPT;
        const float unscale = (p.dyn != nullptr) ? p.dyn->unscale_c : 1.f;
        store_registers<CPT>(sums, p.c + static_cast<uint64_t>(tc.batch) * p.stride_c + row, p.ldc,
                             col0, p.n, row < p.m, p.alpha_r * unscale, p.alpha_i * unscale,
                             (p.flags & kIsComplex) != 0);
        continue;
      }
      // the finished sums go back to the columns of the last ones; from here on they are read from
      // there, and what the epilogue needs to know of the tile is worked out only now (epilogue.cuh)
      finish_pairs_in_tmem<CPT, Cfg::HALF_ROWS, Cfg::B_ROWS>(t_sums, t_cor, acc, LO_SCALE_INV);
      arrive(Cfg::D1_EMPTY);
      const bool part = x.un != p.w.units; // this item is a piece of a tile
      const TileCoord tc = tile_coord<BN, CG>(opaque(x.tile), p, rank);
      const uint32_t quarter = static_cast<uint32_t>(warp & 3);
      const uint32_t col_base = static_cast<uint32_t>((warp - FIRST_EPI_WARP) >> 2) * CPT;
      const uint32_t row =
          static_cast<uint32_t>(tc.m0) + quarter * 32u + static_cast<uint32_t>(lane);
      float *cbase = p.c + static_cast<uint64_t>(tc.batch) * p.stride_c + row;
      if (part) {
        // park the partial sums for the kernel that adds the pieces
        constexpr uint32_t HALF = BN * BM_CTA; // floats of one CTA's half of a tile
        const uint32_t lane_off = col_base * BM_CTA + quarter * 32u + static_cast<uint32_t>(lane);
        float *mine = p.partial + static_cast<uint64_t>((cluster_id * 2u + x.slot) * 2u + rank) * HALF +
                      lane_off;
#pragma unroll 1
        for (int c = 0; c < CPT; c += kEpiGroup) {
          uint32_t v[kEpiGroup];
          ptx::tmem_ld_32x32b_x16(t_sums + c, v);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < kEpiGroup; ++i)
            __stcg(mine + (c + i) * BM_CTA, __uint_as_float(v[i]));
        }
        give_back();
        continue;
      }

      const float unscale = (p.dyn != nullptr) ? p.dyn->unscale_c : 1.f;
      store_tile<CPT>(t_sums, cbase, p.ldc, static_cast<uint32_t>(tc.n0) + col_base, p.n, row < p.m,
                      p.alpha_r * unscale, p.alpha_i * unscale, p.beta_r, p.beta_i,
                      (p.flags & kIsComplex) != 0);
      give_back();
    }
  }

  // ---------------------------------------------------------------- teardown
  // neither CTA leaves while the other still uses its shared memory or TMEM
  ptx::tc_fence_before();
  __syncthreads();
  if constexpr (CG == 2) {
    ptx::cluster_arrive();
    ptx::cluster_wait();
  }
  if (*reinterpret_cast<volatile int *>(raw_smem + RAW_SLOTS * Cfg::RAW_BYTES + Cfg::ABORT)) {
    // a wait gave up: let copies and tensor-core work still in flight land
    const uint64_t t0 = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    ptx::tc_fence_after();
    if constexpr (CG == 2) ptx::tmem_dealloc_pair(tmem_base, TMEM_COLS);
    else ptx::tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// KIND: 0 = FP16, 1 = TF32, 2 = decided on the device (AUTO)
template <int KIND, int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
    tcec_gemm_stream_kernel(const __grid_constant__ CUtensorMap map_a,
                            const __grid_constant__ CUtensorMap map_b, const StreamParams p) {
  if constexpr (KIND == 2) {
    ptx::griddep_wait(); // the decision is written by an earlier kernel of the call
    if (p.dyn->gemm_mode == CUMPSGEMM_TF32TCEC)
      stream_body<1, BN, 2>(map_a, map_b, p);
    else
      stream_body<0, BN, 2>(map_a, map_b, p);
  } else {
    stream_body<KIND, BN, 2>(map_a, map_b, p);
  }
}

// The same on single CTAs, 128 x 128 tiles: batches of matrices with at most 128 rows.
template <int KIND>
__global__ void __launch_bounds__(NUM_THREADS, 1)
    tcec_gemm_stream_solo_kernel(const __grid_constant__ CUtensorMap map_a,
                                 const __grid_constant__ CUtensorMap map_b, const StreamParams p) {
  if constexpr (KIND == 2) {
    ptx::griddep_wait();
    if (p.dyn->gemm_mode == CUMPSGEMM_TF32TCEC)
      stream_body<1, 128, 1>(map_a, map_b, p);
    else
      stream_body<0, 128, 1>(map_a, map_b, p);
  } else {
    stream_body<KIND, 128, 1>(map_a, map_b, p);
  }
}

template <int KIND, int BN, int CG> constexpr auto stream_kernel() {
  if constexpr (CG == 2) return &tcec_gemm_stream_kernel<KIND, BN>;
  else return &tcec_gemm_stream_solo_kernel<KIND>;
}

// Per device and kernel, once: shared-memory attribute, register count, resident clusters.
template <int KIND, int BN, int CG> cudaError_t stream_setup(int *clusters_out) {
  static std::once_flag once[64];
  static cudaError_t setup_error[64];
  static int max_clusters[64];
  auto kernel = stream_kernel<KIND, BN, CG>();
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::call_once(once[dev], [&]() {
    constexpr int smem = StreamCfg<BN, CG>::SMEM_BYTES;
    setup_error[dev] =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    // the register re-allocation inside the kernel draws on what the CTA was launched with: an
    // increase that cannot be served would wait for ever, so refuse to launch with fewer
    cudaFuncAttributes attr;
    if (setup_error[dev] == cudaSuccess) {
      setup_error[dev] = cudaFuncGetAttributes(&attr, kernel);
      if (setup_error[dev] == cudaSuccess && attr.numRegs < LAUNCH_REGS)
        setup_error[dev] = cudaErrorLaunchOutOfResources;
    }
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int clusters = sms / CG;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(2 * clusters));
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = smem;
    int active = 0;
    if (CG == 2 && setup_error[dev] == cudaSuccess &&
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

// Tensor maps of the raw operands (see RawLayout).  Box: one slot of one CTA's rows.
bool raw_map(CUtensorMap *map, const StreamOperand &o, int layout, uint64_t rows, uint64_t k,
             uint32_t batch, uint32_t box_rows) {
  // rows, k: extents of the expanded real operand
  uint64_t d0, d1;
  uint32_t b0, b1;
  bool swizzle = false;
  switch (layout) {
  case kRawK:
    d0 = k, d1 = rows, b0 = SLOT_K, b1 = box_rows, swizzle = true;
    break;
  case kRawR:
    d0 = rows, d1 = k, b0 = box_rows, b1 = SLOT_K;
    break;
  case kRawCplxAR: // floats of a column = expanded rows
    d0 = rows, d1 = k / 2, b0 = box_rows, b1 = SLOT_K / 2;
    break;
  case kRawCplxAK: // floats of a row = expanded k
    d0 = k, d1 = rows / 2, b0 = SLOT_K, b1 = box_rows / 2, swizzle = true;
    break;
  default: // kRawCplxBR: two floats per row of B'
    d0 = 2 * rows, d1 = k / 2, b0 = 2 * box_rows, b1 = SLOT_K / 2;
    break;
  }
  const uint64_t nb = (o.stride != 0 && batch > 1) ? batch : 1;
  const uint64_t ld_bytes = o.ld * sizeof(float);
  const uint64_t stride_bytes = (nb > 1) ? o.stride * sizeof(float) : ld_bytes;
  const uint64_t dims[3] = {d0, d1, nb};
  const uint64_t strides[2] = {ld_bytes, stride_bytes};
  const uint32_t box[3] = {b0, b1, 1};
  return make_float_map(map, o.src, dims, strides, box, swizzle);
}

template <int KIND, int BN, int CG>
cudaError_t launch_variant(const StreamGemmArgs &a, cudaStream_t stream) {
  int max_clusters = 1;
  const cudaError_t se = stream_setup<KIND, BN, CG>(&max_clusters);
  if (se != cudaSuccess) return se;
  CUtensorMap map_a, map_b;
  if (!raw_map(&map_a, a.a, a.layout_a, a.m, a.k, a.batch, BM_CTA) ||
      !raw_map(&map_b, a.b, a.layout_b, a.n, a.k, a.batch, StreamCfg<BN, CG>::HALF_ROWS))
    return cudaErrorNotSupported; // an extent TMA cannot address: the caller takes another path
  StreamParams p;
  p.c = a.c;
  p.dyn = a.dyn;
  p.status = a.dev_status;
  p.partial = a.partial;
  p.debug = a.debug;
  p.ldc = a.ldc;
  p.stride_c = a.stride_c;
  p.m = a.m;
  p.n = a.n;
  p.tiles_m = (a.m + CG * BM_CTA - 1) / (CG * BM_CTA);
  p.tiles_n = (a.n + BN - 1) / BN;
  p.alpha_r = a.alpha_r;
  p.alpha_i = a.alpha_i;
  p.beta_r = a.beta_r;
  p.beta_i = a.beta_i;
  p.layout_a = static_cast<uint8_t>(a.layout_a);
  p.layout_b = static_cast<uint8_t>(a.layout_b);
  p.flags = static_cast<uint8_t>((a.is_complex ? kIsComplex : 0) | (a.conj_a ? kConjA : 0) |
                                 (a.conj_b ? kConjB : 0) |
                                 (a.batch > 1 && a.a.stride != 0 ? kBatchA : 0) |
                                 (a.batch > 1 && a.b.stride != 0 ? kBatchB : 0));
  const StreamPlan &plan = a.plan;
  if (plan.tile_n != BN || plan.tile_m != CG * BM_CTA || plan.total_tiles != p.tiles_m * p.tiles_n * a.batch ||
      plan.units != (a.k + 63) / 64)
    return cudaErrorInvalidValue;
  p.w.total_tiles = plan.total_tiles;
  p.w.whole_tiles = plan.whole_tiles;
  p.w.units = plan.units;
  p.w.slice_units = 0;
  p.w.piece_clusters = static_cast<uint16_t>(plan.piece_clusters);
  p.w.slices = static_cast<uint16_t>(plan.slices);
  // Direct stores: at least three waves of whole tiles of a short K loop, beta = 0 (with 256 columns
  // the sums leave too few registers for it).  What they save is a tile's hand-over, so the gain
  // shrinks with the K loop.  Batches of 256 x 128 x 64u, looped / direct stores, us, three and eight
  // waves (medians of runs in turn): FP16TCEC u = 1 15.6 / 15.2 and 31.9 / 31.1, u = 4 28.3 / 27.4 and
  // 59.8 / 59.4, u = 8 44.6 / 44.3 and 103.4 / 102.9; TF32TCEC u = 2 30.6 / 29.9 and 58.3 / 57.4, u = 8
  // 58.1 / 57.9.  At u = 16 and above, and at one wave, the two sides differ by less than their runs.
  if (BN == 128 && plan.piece_clusters == 0 && plan.whole_tiles >= 3u * static_cast<uint32_t>(max_clusters) &&
      plan.units <= 16 && a.beta_r == 0.f && a.beta_i == 0.f)
    p.flags |= kDirectStores;
  uint32_t clusters = plan.whole_tiles > plan.piece_clusters ? plan.whole_tiles : plan.piece_clusters;
  if (clusters > static_cast<uint32_t>(max_clusters)) clusters = static_cast<uint32_t>(max_clusters);
  if (clusters == 0 || plan.piece_clusters > clusters) return cudaErrorInvalidValue;
  const cudaError_t e = launch_chained(stream_kernel<KIND, BN, CG>(), CG * clusters, NUM_THREADS,
                                       StreamCfg<BN, CG>::SMEM_BYTES, stream, map_a, map_b, p);
  if (e != cudaSuccess || plan.piece_clusters == 0) return e;
  const PieceFixupArgs f = {a.partial,  a.c,       nullptr,   a.dyn,     a.ldc,
                            a.stride_c, a.m,       a.n,       p.tiles_m, p.tiles_n,
                            BN,         a.alpha_r, a.alpha_i, a.beta_r,  a.beta_i,
                            a.is_complex};
  return launch_piece_fixup(f, p.w, stream);
}

template <int BN, int CG> cudaError_t launch_by_kind(const StreamGemmArgs &a, cudaStream_t stream) {
  switch (a.kind) {
  case StreamKind::fp16:
    return launch_variant<0, BN, CG>(a, stream);
  case StreamKind::tf32:
    return launch_variant<1, BN, CG>(a, stream);
  default:
    return a.dyn != nullptr ? launch_variant<2, BN, CG>(a, stream) : cudaErrorInvalidValue;
  }
}

} // namespace

// Left-over tiles (total mod clusters, or all of them when there are fewer tiles than clusters)
// are cut along K where that saves more than it costs.
StreamPlan plan_stream(const Tuning &tuning, int tile_n, uint64_t m, uint64_t n, uint64_t k,
                       uint64_t batch, uint32_t clusters) {
  StreamPlan pl = {};
  pl.tile_m = 2 * BM_CTA;
  pl.tile_n = tile_n;
  const uint64_t total =
      ((m + 2 * BM_CTA - 1) / (2 * BM_CTA)) * ((n + tile_n - 1) / tile_n) * batch;
  const uint64_t units = (k + 63) / 64;
  if (total == 0 || total > 0x3fffffffull || units == 0 || units > 0x3fffffull || clusters == 0)
    return StreamPlan{};
  pl.total_tiles = static_cast<uint32_t>(total);
  pl.units = static_cast<uint32_t>(units);
  pl.whole_tiles = pl.total_tiles;
  const uint32_t rem = pl.total_tiles % clusters;
  if (rem == 0 || clusters > 0xffffu) return pl;
  constexpr uint32_t kMinSliceUnits = 3; // shortest slice / piece, in units of 64 k values
  // a cut has to save more than parking and adding the pieces costs: about 0.3 us per left-over
  // tile, at 1.45 us per unit
  const uint32_t min_saved = 2 + rem / 5;
  if (3 * pl.total_tiles <= clusters && tuning.split_k != 0) {
    // few tiles: each in the same number of slices
    uint32_t s = clusters / pl.total_tiles;
    if (s > pl.units / kMinSliceUnits) s = pl.units / kMinSliceUnits;
    if (s >= 2 && pl.units - pl.units / s >= min_saved + 2) {
      pl.whole_tiles = 0;
      pl.slices = s;
      pl.piece_clusters = s * pl.total_tiles;
    }
    return pl;
  }
  if (tuning.split_k == 0 || tuning.tail_split == 0) return pl;
  const uint64_t left = static_cast<uint64_t>(rem) * pl.units;
  uint32_t pc = clusters;
  if (left / kMinSliceUnits < pc) pc = static_cast<uint32_t>(left / kMinSliceUnits);
  if (pc <= rem) return pl;
  const uint32_t per = static_cast<uint32_t>((left + pc - 1) / pc);
  if (per + min_saved > pl.units) return pl;
  pl.whole_tiles = pl.total_tiles - rem;
  pl.piece_clusters = pc;
  return pl;
}

StreamPlan plan_stream_solo(uint64_t m, uint64_t n, uint64_t k, uint64_t batch) {
  StreamPlan pl = {};
  const uint64_t total = ((m + BM_CTA - 1) / BM_CTA) * ((n + 127) / 128) * batch;
  const uint64_t units = (k + 63) / 64;
  if (total == 0 || total > 0x3fffffffull || units == 0 || units > 0x3fffffull) return pl;
  pl.tile_m = BM_CTA;
  pl.tile_n = 128;
  pl.total_tiles = pl.whole_tiles = static_cast<uint32_t>(total);
  pl.units = static_cast<uint32_t>(units);
  return pl;
}

std::size_t stream_scratch_bytes(const StreamPlan &plan) {
  return static_cast<std::size_t>(plan.piece_clusters) * 2u * 2u * BM_CTA *
         static_cast<std::size_t>(plan.tile_n) * sizeof(float);
}

cudaError_t launch_tcec_gemm_stream(const StreamGemmArgs &a, cudaStream_t stream) {
  if (a.plan.tile_m == BM_CTA) return launch_by_kind<128, 1>(a, stream);
  if (a.plan.tile_n == 256) return launch_by_kind<256, 2>(a, stream);
  if (a.plan.tile_n == 128) return launch_by_kind<128, 2>(a, stream);
  return cudaErrorInvalidValue;
}

cudaError_t stream_max_clusters(StreamKind kind, int tile_n, int *clusters) {
  switch (kind) {
  case StreamKind::fp16:
    return tile_n == 256 ? stream_setup<0, 256, 2>(clusters) : stream_setup<0, 128, 2>(clusters);
  case StreamKind::tf32:
    return tile_n == 256 ? stream_setup<1, 256, 2>(clusters) : stream_setup<1, 128, 2>(clusters);
  default:
    return tile_n == 256 ? stream_setup<2, 256, 2>(clusters) : stream_setup<2, 128, 2>(clusters);
  }
}

} // namespace cumpsgemm_b200

extern "C" int cuMpSGEMM_plan_stream(uint64_t m, uint64_t n, uint64_t k, uint64_t batch, int tile_n,
                                     unsigned clusters, unsigned *total_tiles, unsigned *units,
                                     unsigned *whole_tiles, unsigned *piece_clusters,
                                     unsigned *slices) {
  using namespace cumpsgemm_b200;
  if (m == 0 || n == 0 || k == 0 || batch == 0 || (tile_n != 256 && tile_n != 128) ||
      clusters == 0 || total_tiles == nullptr || units == nullptr || whole_tiles == nullptr ||
      piece_clusters == nullptr || slices == nullptr)
    return 1;
  const StreamPlan pl = plan_stream(Tuning{}, tile_n, m, n, k, batch, clusters);
  if (pl.total_tiles == 0) return 1;
  *total_tiles = pl.total_tiles;
  *units = pl.units;
  *whole_tiles = pl.whole_tiles;
  *piece_clusters = pl.piece_clusters;
  *slices = pl.slices;
  return 0;
}
