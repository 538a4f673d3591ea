// Adds the K pieces of the tiles a CTA-pair GEMM launch cut (work_list.cuh) and runs their
// alpha / beta epilogue: the deterministic successor of the reference's atomic accumulation
// (src/cumpsgemm.cu:272-304, src/dmem_accessor.hpp:352-395).
//
// All pieces of a launch end at about the same time, so adding them is a job for the whole GPU:
// the scratch tiles are still in L2 and every thread has the loads of four pieces in flight.  (Done
// instead inside the GEMM kernel by whichever CTA finished a tile last, with a ticket counter per
// tile, it took 20 us for 40 tiles: a few CTAs, one L2 latency per group of columns and piece.)
//
// A block takes COLS columns x 256 rows (both CTAs' halves) of one tile; thread = row, so every
// access covers whole 128-byte lines.  With many pieces per tile GROUPS thread groups share them:
// each adds a contiguous part in ascending k, then the parts are added in order.
#include "gemm_common.cuh"
#include "work_list.cuh"

namespace cumpsgemm_b200 {
namespace {

struct FixupParams {
  const float *partial;
  float *c;
  float *const *c_array;
  const DynParams *dyn;
  uint64_t ldc, stride_c;
  uint32_t m, n, tiles_m, tiles_n, tile_n;
  float alpha_r, alpha_i, beta_r, beta_i;
  uint32_t is_complex;
  WorkPlan w;
};
static_assert(sizeof(FixupParams) <= 128, "kernel parameter structs stay within 128 bytes");

template <int COLS, int GROUPS>
__global__ void __launch_bounds__(256 * GROUPS) piece_fixup_kernel(const FixupParams p) {
  CUMPSGEMM_CHAINED_KERNEL_ENTRY(); // launched behind the GEMM kernel
  const uint32_t blocks_per_tile = p.tile_n / COLS;
  const uint32_t ti = blockIdx.x / blocks_per_tile;
  const uint32_t col_in_tile = (blockIdx.x - ti * blocks_per_tile) * COLS;
  const TilePos pos = tile_raster(p.w.whole_tiles + ti, p.tiles_m, p.tiles_n);
  const uint32_t col0 = pos.tn * p.tile_n + col_in_tile;
  const uint32_t r = threadIdx.x & 255u;
  const uint32_t row = pos.tm * 256u + r;
  if (col0 >= p.n) return; // uniform over the block
  const TilePieces tp = tile_pieces(ti, p.w);
  const uint64_t half = static_cast<uint64_t>(p.tile_n) * 128u; // one CTA's part of a scratch tile
  const float *base = p.partial + (r >> 7) * half + col_in_tile * 128u + (r & 127u);
  auto piece = [&](uint32_t cc) {
    return base + (cc * 2u + (cc == tp.c0 ? tp.slot0 : 0u)) * 2u * half;
  };
  const uint32_t pieces = tp.c1 - tp.c0 + 1u;
  const uint32_t group = threadIdx.x >> 8;
  const uint32_t first = pieces * group / GROUPS, last = pieces * (group + 1u) / GROUPS;
  const bool read_c = (p.beta_r != 0.f) || (p.beta_i != 0.f);
  const bool row_ok = row < p.m;
  float *cp = ((p.c_array != nullptr) ? p.c_array[pos.batch]
                                      : p.c + static_cast<uint64_t>(pos.batch) * p.stride_c) +
              static_cast<uint64_t>(col0) * p.ldc + row;
  float old[COLS]; // on their way while the pieces are added
#pragma unroll
  for (uint32_t j = 0; j < COLS; ++j)
    old[j] = (read_c && group == 0 && row_ok && col0 + j < p.n) ? __ldcs(cp + j * p.ldc) : 0.f;
  float sum[COLS];
#pragma unroll
  for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
#pragma unroll 4
  for (uint32_t i = first; i < last; ++i) {
    const float *src = piece(tp.c0 + i);
#pragma unroll
    for (int j = 0; j < COLS; ++j) sum[j] += __ldcg(src + j * 128);
  }
  if constexpr (GROUPS > 1) {
    __shared__ float part[GROUPS - 1][COLS][256];
    if (group > 0) {
#pragma unroll
      for (int j = 0; j < COLS; ++j) part[group - 1][j][r] = sum[j];
    }
    __syncthreads();
    if (group > 0) return;
#pragma unroll
    for (int g = 0; g < GROUPS - 1; ++g)
#pragma unroll
      for (int j = 0; j < COLS; ++j) sum[j] += part[g][j][r];
  }
  const float unscale = (p.dyn != nullptr) ? p.dyn->unscale_c : 1.f;
  const float ar = p.alpha_r * unscale, ai = p.alpha_i * unscale;
  const float sgn = (r & 1u) ? 1.f : -1.f; // odd rows hold imaginary parts
#pragma unroll
  for (uint32_t j = 0; j < COLS; ++j) {
    float out = ar * sum[j];
    if (p.is_complex) out += sgn * ai * __shfl_xor_sync(0xffffffffu, sum[j], 1);
    if (read_c) {
      out = fmaf(p.beta_r, old[j], out);
      if (p.is_complex) out += sgn * p.beta_i * __shfl_xor_sync(0xffffffffu, old[j], 1);
    }
    if (row_ok && col0 + j < p.n) cp[j * p.ldc] = out;
  }
}

template <int COLS, int GROUPS>
cudaError_t launch(const FixupParams &p, uint32_t tiles, cudaStream_t stream) {
  return launch_chained(piece_fixup_kernel<COLS, GROUPS>, tiles * (p.tile_n / COLS), 256 * GROUPS, 0,
                        stream, p);
}

} // namespace

cudaError_t launch_piece_fixup(const PieceFixupArgs &a, const WorkPlan &w, cudaStream_t stream) {
  if (w.piece_clusters == 0 || a.partial == nullptr) return cudaErrorInvalidValue;
  FixupParams p;
  p.partial = a.partial;
  p.c = a.c;
  p.c_array = a.c_array;
  p.dyn = a.dyn;
  p.ldc = a.ldc;
  p.stride_c = a.stride_c;
  p.m = a.m;
  p.n = a.n;
  p.tiles_m = a.tiles_m;
  p.tiles_n = a.tiles_n;
  p.tile_n = a.tile_n;
  p.alpha_r = a.alpha_r;
  p.alpha_i = a.alpha_i;
  p.beta_r = a.beta_r;
  p.beta_i = a.beta_i;
  p.is_complex = a.is_complex ? 1u : 0u;
  p.w = w;
  const uint32_t tiles = w.total_tiles - w.whole_tiles;
  // One wave of blocks that fills the GPU (two of 1024 threads or eight of 256 per SM): narrow
  // blocks for few tiles, and thread groups that share the pieces when there are many per tile.
  // Measured, FP16TCEC, us per call with <COLS, GROUPS> = <1,4> <2,4> <4,4> <4,1> <8,1> <16,1>:
  //    1 tile  in 74 pieces (256 x 256 x 16384)           31  29  30  44  48  61
  //    1 tile, 128 columns  (256 x 128 x 16384)           18  19  20  31  34  44
  //    2 tiles in 74        (256 x 512 x 16384)           42  32  30  36  38  44
  //    6 tiles in 72        (512 x 768 x 8192)            58  46  38  32  32  34
  //    8 tiles in 72        (512 x 1024 x 8192)           63  49  46  37  37  38
  //   16 tiles in 64        (1024 x 1024 x 4096)          89  63  54  39  38  37
  //   16 of 90 tiles        (256 x 256 x 1536, batch 90)  128 101  94  79  79  80
  //   32 of 106 tiles       (the same, batch 106)         235 157 139  99  91  93
  // So one group is right from about six tiles on (768 x 768 x 3072, nine tiles in 72: 36 us with
  // four groups).
  if (tiles < 6u && w.piece_clusters >= 8u * tiles) {
    if (tiles == 1) return launch<1, 4>(p, tiles, stream);
    if (tiles == 2) return launch<2, 4>(p, tiles, stream);
    return launch<4, 4>(p, tiles, stream);
  }
  if (tiles <= 16) return launch<4, 1>(p, tiles, stream);
  if (tiles <= 32) return launch<8, 1>(p, tiles, stream);
  return launch<16, 1>(p, tiles, stream);
}

} // namespace cumpsgemm_b200
