// Host dispatch of the TCEC GEMM and the C ABI around it.
//
// Reference counterparts: cumpsgemm::gemm<T> (src/cumpsgemm.cu:228-419),
// cumpsgemm::gemm_stridedBatch<T> (:421-547), the extern "C" wrappers
// (:549-605) and the AUTO / FP16TCEC_SCALING orchestration of the
// interception layer (src/cumpsgemm_cublas.cu:445-577, :829-961).
//
// A call takes one of these routes, all on the handle's stream: split pass -> tcgen05 GEMM on the
// panels, on single CTAs (tcec_gemm.cu) or pairs (tcec_gemm_pair.cu); one kernel on CTA pairs or single
// CTAs that splits its operands behind TMA (tcec_gemm_stream.cu); for small products one that loads
// and splits them itself (tcec_gemm_small.cu).  Tiles cut along K are added by one more launch.  (A fifth
// kernel, tcec_gemm_fused.cu, runs only where a switch asks for it.)  The reference's module
// table (364 instantiations per arch, src/instance_sm80.cu) collapses to a few tile widths because
// op N/T/C, leading dimensions and edges are absorbed where the operands are split.
#include "gemm_common.cuh"
#include "work_list.cuh"

#include <cumpsgemm/cumpsgemm_ext.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace cumpsgemm_b200 {
namespace {

constexpr std::size_t kDefaultWorkspaceLimit = 8ull << 30;

inline std::uint64_t round_up(std::uint64_t x, std::uint64_t a) { return (x + a - 1) / a * a; }

// Whether memory may be allocated and freed now: not while the stream is being captured into a
// graph, where either would end the capture.
bool may_allocate(const cuMpSGEMM_handle *h) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(h->cuda_stream, &cap) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return cap == cudaStreamCaptureStatusNone;
}

// Makes the workspace hold `bytes`.  Returns false, with the old workspace untouched, while the
// stream is being captured, and false without a workspace if there is no memory.
bool ensure_workspace(cuMpSGEMM_handle *h, std::size_t bytes) {
  if (h->workspace_bytes >= bytes) return true;
  if (!may_allocate(h)) return false;
  if (h->workspace != nullptr) {
    if (h->workspace_in_graph) h->graph_workspaces.push_back(h->workspace);
    else cudaFree(h->workspace); // waits for work that may still read the old buffer
  }
  h->workspace_in_graph = false;
  h->workspace = nullptr;
  h->workspace_bytes = 0;
  if (cudaMalloc(&h->workspace, bytes) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  h->workspace_bytes = bytes;
  return true;
}

__global__ void dyn_params_from_flag_kernel(DynParams *out, const int *flag) {
  CUMPSGEMM_CHAINED_KERNEL_ENTRY();
  out->scale_a = 1.f;
  out->scale_b = 1.f;
  out->unscale_c = 1.f;
  const int mode = flag_gemm_mode(*flag);
  out->gemm_mode = (mode == CUMPSGEMM_TF32TCEC) ? CUMPSGEMM_TF32TCEC : CUMPSGEMM_FP16TCEC;
}

template <class T> struct Scalar;
template <> struct Scalar<float> {
  static float re(const float *p) { return *p; }
  static float im(const float *) { return 0.f; }
};
template <> struct Scalar<cuComplex> {
  static float re(const cuComplex *p) { return p->x; }
  static float im(const cuComplex *p) { return p->y; }
};

// ---------------------------------------------------------------- which kernel
//
// Estimated time of a call on the pre-split and the streaming paths, in microseconds.  A call is
// one or more waves of tiles, each as long as its K loop; what the paths trade is idle SMs against
// operand traffic, the split pass against converting every operand element once per tile that
// uses it, and cutting tiles along K against adding the pieces.
//
// Two steps.  single(), pair() and split_k() choose the tile of the pre-split path; they are fits to 104
// problems of 1-80 pair tiles and k = 128-8192 (B200, mean error 5-9 %), and leave out what all tiles
// have in common.  presplit_call() adds that, and the call goes where it is estimated to end first.
// What it adds, and the estimates of streaming, are fits to 580 random problems in each of FP16TCEC and TF32TCEC
// with every path forced in turn: single products of 1-111 pair tiles (m, n 32-4096, k 128-131072)
// and batches of 8-2048 (m, n 16-1024, k 32-2048), real and complex, every op, beta = 0 and 0.5,
// operands on 16 bytes; the GPU's time in runs of twelve calls.  Mean error on as many others: 10 % pre-split, 5-7 %
// streaming.  On 1150 calls drawn once more, choosing by these estimates was 0.5 % slower than the best
// path of each (largest 1.38); the constants before, fitted to fewer sizes and to no batches, lost 1 to 10 %
// by kind of problem there (10 % in batches of 8-48 matrices of at most 128 rows, largest 1.9).
// A unit of 64 k values is one stage in FP16TCEC and two in TF32TCEC, for all paths alike.
struct PathModel {
  double units, stages, sms, pairs;
  double split; // megabytes the split pass reads and writes, without padding
  double c_passes; // over C: 2 if it is read too
  std::uint64_t m, n, k, batch;

  static double waves(std::uint64_t tiles, double slots) { return std::ceil(tiles / slots); }
  PathModel(unsigned num_sms, std::uint64_t m_, std::uint64_t n_, std::uint64_t k_,
            std::uint64_t batch_, bool tf32, bool reads_c = false)
      : units(static_cast<double>((k_ + 63) / 64)), stages(tf32 ? 2 * units : units), sms(num_sms),
        pairs(num_sms / 2), c_passes(reads_c ? 2.0 : 1.0), m(m_), n(n_), k(k_), batch(batch_) {
    split = 1e-6 * static_cast<double>(m + n) * k * batch * (tf32 ? 12 : 8);
  }
  std::uint64_t tiles(std::uint64_t bm, std::uint64_t bn) const {
    return ((m + bm - 1) / bm) * ((n + bn - 1) / bn) * batch;
  }
  // One CTA per 128 x bn tile.  A stage takes longer the more SMs compete for L2 (and power).
  double single(int bn) const {
    const std::uint64_t t = tiles(128, bn);
    const double busy = std::min(1.0, t / sms);
    const double w = waves(t, sms) * stages;
    if (bn == 64) return 5.7 + 0.073 * split + w * (0.45 + 0.11 * busy);
    if (bn == 128) return 6.1 + 0.100 * split + w * (0.53 + 0.15 * busy);
    return 6.8 + 0.108 * split + w * (0.97 + 0.26 * busy);
  }
  double pair(const WorkPlan &w) const { // 256 x 256 tiles, left-over ones perhaps in K pieces
    double length = waves(w.whole_tiles, pairs) * units, t = 8.8 + 0.169 * split;
    if (w.piece_clusters > 0) {
      const double left = w.total_tiles - w.whole_tiles;
      length += w.slice_units != 0 ? w.slice_units : std::ceil(left * units / w.piece_clusters);
      t += 4.0 + 0.06 * left;
    }
    return t + length * stages / units * (0.86 + 0.29 * std::min(1.0, w.total_tiles / pairs));
  }
  double split_k(std::uint32_t slices) const { // K slices of the widest tiles, then a reduction
    return 2.0 + 0.15 * split + 1.32 * std::ceil(stages / slices) +
           0.69e-6 * 4 * static_cast<double>(m) * n * batch * slices;
  }
  // The whole call, `t` being the estimate its tile (tile_m x tile_n) was chosen by.  Beyond that: the rows and k
  // values that pad the panels, the stores of every wave, and where pieces of pair tiles are laid end to end, two
  // to park for every pair instead of one.
  double presplit_call(double t, int tile_m, int tile_n, double waves_of_tiles, double parked) const {
    const auto up = [](std::uint64_t v, std::uint64_t q) { return static_cast<double>((v + q - 1) / q * q); };
    const double lo_hi = stages > units ? 8e-6 : 4e-6;
    const double padding = lo_hi * batch * ((up(m, tile_m) + up(n, tile_n)) * up(k, 64) -
                                            static_cast<double>(m + n) * static_cast<double>(k));
    return t + 0.2 * padding + 0.8 * c_passes * waves_of_tiles * (tile_n / 128.0) + 0.3 * parked;
  }
  // tcec_gemm_stream.cu on single CTAs, 128 x 128 tiles
  double stream_solo(const StreamPlan &pl) const {
    const double busy = std::min(1.0, pl.total_tiles / sms), a = stages > units ? 1.62 : 0.83;
    return 4.0 + waves(pl.total_tiles, sms) * (units * (a + 0.24 * busy) + 1.7 * c_passes);
  }
  // tcec_gemm_stream.cu on pairs
  double stream(const StreamPlan &pl) const {
    const bool tf32 = stages > units, wide = pl.tile_n == 256;
    const double busy =
        std::min(1.0, std::max<double>(pl.whole_tiles, pl.piece_clusters) / pairs);
    const double unit = wide ? (tf32 ? 1.90 + 0.63 * busy : 0.96 + 0.52 * busy)
                             : (tf32 ? 1.39 + 0.39 * busy : 0.62 + 0.30 * busy);
    const double w = waves(pl.whole_tiles, pairs);
    double t = (wide ? 6.5 : 6.0) + w * (units * unit + (wide ? 2.2 : 1.55) * c_passes);
    if (pl.piece_clusters > 0) {
      const double left = pl.total_tiles - pl.whole_tiles;
      t += std::ceil(left * units / pl.piece_clusters) * unit + (wide ? 7.1 + 0.1 * left : 5.5 + 0.03 * left);
    }
    return t;
  }
};

// Tile of the pre-split path: width 256 / 128 / 64 of the single-CTA kernel (128 rows), or the
// CTA-pair kernel's 256 x 256 tile (error-corrected modes only).  CUMPSGEMM_TILE_N forces the
// width, CUMPSGEMM_PAIR=0/1 the kernel.
} // namespace

TileChoice pick_tile(const Tuning &tuning, unsigned num_sms, std::uint64_t m_exp, std::uint64_t n,
                     std::uint64_t k_exp, std::uint64_t batch, bool ec, bool tf32, bool can_cut) {
  const bool pair_off = tuning.pair == 0;
  if (tuning.tile_n == 256) return {256, ec && !pair_off, 0.0};
  if (tuning.tile_n == 128 || tuning.tile_n == 64) return {tuning.tile_n, false, 0.0};
  const PathModel model(num_sms, m_exp, n, k_exp, batch, tf32);
  if (!ec) { // a third of the products: the widest tile that gives two thirds of the SMs one
    const std::uint64_t sms = num_sms;
    if (3 * model.tiles(128, 256) >= 2 * sms) return {256, false, 0.0};
    return {3 * model.tiles(128, 128) >= 2 * sms ? 128 : 64, false, 0.0};
  }
  TileChoice best = {64, false, model.single(64)};
  for (int bn : {128, 256})
    if (const double t = model.single(bn); t < best.us) best = {bn, false, t};
  const std::uint64_t pair_tiles = model.tiles(256, 256);
  if (!pair_off && num_sms >= 2 && pair_tiles <= 0x7fffffffull) {
    // (more than one wave of pair tiles: always pairs, 4096^3 277 us against 338 for 128 x 256
    // tiles, GEMM kernel; the model is fitted to less)
    const WorkPlan w = plan_pair(tuning, tf32, can_cut, static_cast<std::uint32_t>(pair_tiles),
                                 static_cast<std::uint32_t>(model.units), num_sms / 2);
    const double t = model.pair(w);
    if (tuning.pair == 1 || pair_tiles > num_sms / 2 || t < best.us) best = {256, true, t};
  }
  return best;
}

namespace {

// The kernel that splits operands on the fly (tcec_gemm_fused.cu), for FP16TCEC (with or without fused
// scaling) on 16-byte aligned strided operands in the layouts its converters know.  Streaming is faster on
// all that was measured of what it can take (us, this kernel / streaming: 256 x 256 x 8192 23.4 / 16.8, 384 x
// 384 x 32768 73 / 48, 9 x 300 x 300 x 900 44 / 20, 2048 x 128^3 76.5 / 66.8), so it runs only where
// CUMPSGEMM_FUSED=1 asks for it or, by the rule below, where a switch keeps streaming off.
// Returns false when the call has to take another path.
template <class T>
bool fused_args(const cuMpSGEMM_handle *h, cublasOperation_t op_A, cublasOperation_t op_B,
                std::uint64_t m, std::uint64_t n, std::uint64_t k, const T *a, std::uint64_t lda,
                std::uint64_t stridea, const T *b, std::uint64_t ldb, std::uint64_t strideb,
                std::uint64_t batch, FusedGemmArgs *out) {
  constexpr bool is_complex = std::is_same<T, cuComplex>::value;
  constexpr std::uint64_t fpe = is_complex ? 2 : 1;
  if (h->tuning.fused == 0 || (h->tuning.fused != 1 && !h->tuning.streaming_off())) return false;
  if (batch > 0x7fffffffull) return false;
  if (is_complex && (op_A != CUBLAS_OP_N || op_B != CUBLAS_OP_N)) return false;
  const std::uint64_t lda_f = lda * fpe, ldb_f = ldb * fpe;
  const std::uint64_t sa_f = (batch > 1 ? stridea : 0) * fpe, sb_f = (batch > 1 ? strideb : 0) * fpe;
  const bool aligned = (reinterpret_cast<std::uintptr_t>(a) % 16 == 0) &&
                       (reinterpret_cast<std::uintptr_t>(b) % 16 == 0) && lda_f % 4 == 0 &&
                       ldb_f % 4 == 0 && sa_f % 4 == 0 && sb_f % 4 == 0;
  if (!aligned) return false;
  const std::uint64_t m_exp = m * fpe, k_exp = k * fpe;
  if (h->tuning.fused != 1) {
    // Measured crossover without streaming (B200, FP16TCEC, one call, ms; pre-split path / this kernel):
    //   512 x complex 256^3      0.51 / 0.43      2048 x real 128^3        0.38 / 0.09
    //   512 x real 256^3         0.20 / 0.15      64 x real 1024^3         0.53 / 0.87
    //   real 4096 x 4096 x 512   0.086 / 0.113    real 8192 x 8192 x 256   0.17 / 0.24
    //   real 1024^3              0.025 / 0.036    real 4096^3              0.37 / 0.81
    // The on-the-fly split wins for strided batches of small matrices, where the split pass,
    // its workspace traffic and a second launch weigh as much as the products; a single
    // matrix, large tiles counts or a long K loop are better off pre-split (every operand
    // element is converted once per tile that uses it).
    // A handful of tiles and a very long K loop: this kernel with its K loop cut over the SMs
    // (split-K below) against the pre-split split-K path, ms per call, NN:
    //   256 x 256 x 65536   0.068 / 0.085     128 x 128 x 131072   0.054 / 0.080
    //   384 x 384 x 32768   0.070 / 0.079     256 x 256 x 8192     0.021 / 0.025
    //   512 x 512 x 16384   0.064 / 0.056 (sixteen tiles: the pre-split path wins again)
    // There the split pass alone moves twice the operand bytes the products need.
    const std::uint64_t tiles = ((m_exp + 127) / 128) * ((n + 127) / 128) * batch;
    const bool few_long = h->tuning.split_k != 0 && h->tuning.pair != 1 &&
                          h->tuning.tile_n != 256 && tiles <= 9 && k_exp >= 8192;
    if (!few_long && (batch < 8 || m_exp > 512 || n > 512 || k_exp > 1024)) return false;
  }
  out->a = reinterpret_cast<const float *>(a);
  out->b = reinterpret_cast<const float *>(b);
  out->lda = lda_f;
  out->ldb = ldb_f;
  out->stride_a = sa_f;
  out->stride_b = sb_f;
  if (is_complex) {
    out->layout_a = 2;
    out->layout_b = 0;
  } else {
    out->layout_a = (op_A == CUBLAS_OP_N) ? 1 : 0;
    out->layout_b = (op_B == CUBLAS_OP_N) ? 0 : 1;
  }
  out->m = static_cast<std::uint32_t>(m_exp);
  out->n = static_cast<std::uint32_t>(n);
  out->k = static_cast<std::uint32_t>(k_exp);
  out->batch = static_cast<std::uint32_t>(batch);
  out->is_complex = is_complex;
  out->tile_n = (h->tuning.tile_n == 64 || n <= 64) ? 64 : 128;
  out->tuning = h->tuning;
  // split-K when the tiles leave at least half of the SMs idle and K is long: as many slices
  // as fill the GPU, each at least four stages (256 k values) long
  out->k_slices = 1;
  out->partial = nullptr;
  {
    const std::uint64_t tiles =
        ((m_exp + 127) / 128) * ((n + out->tile_n - 1) / out->tile_n) * batch;
    const std::uint64_t stages = (k_exp + 63) / 64;
    if (h->tuning.split_k != 0 && 2 * tiles <= h->num_sms && stages >= 8) {
      std::uint64_t want = h->num_sms / tiles;
      if (h->tuning.split_k > 1) want = static_cast<std::uint64_t>(h->tuning.split_k);
      want = std::min<std::uint64_t>(want, stages / 4);
      if (want > 1) {
        const std::uint64_t per = (stages + want - 1) / want;
        out->k_slices = static_cast<std::uint32_t>((stages + per - 1) / per);
      }
    }
  }
  return true;
}

// Operands of a call for the streaming pair kernel (tcec_gemm_stream.cu).  TMA reads them in
// place, so bases, leading dimensions and batch strides have to be multiples of 16 bytes; every
// op and both kinds are handled.  Returns false when the call has to take another path.
template <class T>
bool stream_args(const cuMpSGEMM_handle *h, cublasOperation_t op_A, cublasOperation_t op_B,
                 std::uint64_t m, std::uint64_t n, std::uint64_t k, const T *a, std::uint64_t lda,
                 std::uint64_t stridea, const T *b, std::uint64_t ldb, std::uint64_t strideb,
                 std::uint64_t batch, bool reads_c, StreamKind kind, double presplit_us,
                 StreamGemmArgs *out) {
  constexpr bool is_complex = std::is_same<T, cuComplex>::value;
  constexpr std::uint64_t fpe = is_complex ? 2 : 1;
  const Tuning &t = h->tuning;
  if (t.streaming_off()) return false;
  const std::uint64_t sa = batch > 1 ? stridea * fpe : 0, sb = batch > 1 ? strideb * fpe : 0;
  const bool aligned = (reinterpret_cast<std::uintptr_t>(a) % 16 == 0) &&
                       (reinterpret_cast<std::uintptr_t>(b) % 16 == 0) && (lda * fpe) % 4 == 0 &&
                       (ldb * fpe) % 4 == 0 && sa % 4 == 0 && sb % 4 == 0;
  constexpr std::uint64_t kMaxStride = (1ull << 38) - 1; // floats: TMA strides are below 2^40 bytes
  if (!aligned || lda * fpe > kMaxStride || ldb * fpe > kMaxStride || sa > kMaxStride ||
      sb > kMaxStride)
    return false;
  const std::uint64_t m_exp = m * fpe, k_exp = k * fpe;
  if (batch > 0x3fffffffull || n > 0x3fffffffull) return false; // (TMA coordinates are 32-bit)
  const auto estimate = [&](const StreamPlan &pl) {
    // (the kind of an AUTO call is not known here: the mean of both)
    double us = 0.0;
    for (const bool tf32 : {false, true}) {
      if (kind == (tf32 ? StreamKind::fp16 : StreamKind::tf32)) continue;
      const PathModel model(h->num_sms, m_exp, n, k_exp, batch, tf32, reads_c);
      us += pl.tile_m == 128 ? model.stream_solo(pl) : model.stream(pl);
    }
    return kind == StreamKind::device ? 0.5 * us : us;
  };
  // The kernel and its width: forced, or the one estimated to be fastest, if that is 3 % faster than the
  // pre-split path (within that neither is faster as a rule, and that path gives the bits of the
  // allocation-free entry point; on the problems behind PathModel a margin of 3 % loses 0.7 % against the best
  // path of each, none 0.8, 5 % 0.8).
  StreamPlan plan = {};
  double best = t.stream == -1 ? 0.97 * presplit_us : 1e30;
  const auto consider = [&](const StreamPlan &pl) {
    const double us = estimate(pl);
    if (us < best) {
      best = us;
      plan = pl;
    }
  };
  // Batches of matrices with at most 128 rows would leave one CTA of every pair idle, so single CTAs stand
  // beside pairs there; pairs can cut a few tiles with a long K loop.  us, pre-split / pairs / single CTAs:
  // FP16TCEC 1327 x 64 x 64 x 96 150 / 66 / 38, 1051 x 108 x 476 x 132 453 / 301 / 215, 9 x 32 x 32 x
  // 1940 19.4 / 15.1 / 33, 18 x complex 28 x 192 x 512 18.8 / 20.0 / 21.3.
  const bool few_rows = t.stream <= 1 && batch >= 8 && m_exp <= 128 && n <= 1024;
  if (few_rows) {
    const StreamPlan pl = plan_stream_solo(m_exp, n, k_exp, batch);
    if (pl.total_tiles != 0) consider(pl);
  }
  for (const int tile_n : {256, 128}) {
    if ((t.stream == 128 || t.stream == 256) ? tile_n != t.stream : (n <= 128 && tile_n == 256)) continue;
    int clusters = 0;
    if (stream_max_clusters(kind, tile_n, &clusters) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    const StreamPlan pl = plan_stream(t, tile_n, m_exp, n, k_exp, batch,
                                      static_cast<std::uint32_t>(clusters));
    if (pl.total_tiles == 0) continue;
    if (t.stream != -1 && !few_rows) {
      plan = pl;
      break;
    }
    // beyond one and a half waves of wide tiles the operands of large matrices are reused by too many tiles
    // to convert them again for each (4096 x 4096 x 1024: 102 us against 91), and the model is fitted to batches
    // of small ones only
    const bool small_matrices = batch >= 8 && m_exp <= 1024 && n <= 1024;
    if (!small_matrices &&
        2ull * pl.total_tiles > 3ull * (256 / tile_n) * static_cast<std::uint64_t>(clusters))
      continue;
    consider(pl);
  }
  if (plan.total_tiles == 0) return false;
  *out = StreamGemmArgs{};
  out->kind = kind;
  out->a = StreamOperand{reinterpret_cast<const float *>(a), lda * fpe, sa};
  out->b = StreamOperand{reinterpret_cast<const float *>(b), ldb * fpe, sb};
  if (is_complex) {
    out->layout_a = (op_A == CUBLAS_OP_N) ? 2 : 3;
    out->layout_b = (op_B == CUBLAS_OP_N) ? 0 : 4;
    out->conj_a = (op_A == CUBLAS_OP_C);
    out->conj_b = (op_B == CUBLAS_OP_C);
  } else {
    out->layout_a = (op_A == CUBLAS_OP_N) ? 1 : 0;
    out->layout_b = (op_B == CUBLAS_OP_N) ? 0 : 1;
  }
  out->is_complex = is_complex;
  out->m = static_cast<std::uint32_t>(m_exp);
  out->n = static_cast<std::uint32_t>(n);
  out->k = static_cast<std::uint32_t>(k_exp);
  out->batch = static_cast<std::uint32_t>(batch);
  out->plan = plan;
  return true;
}

// Tile or K slices of the pre-split path.
struct PresplitChoice {
  TileChoice tile;
  std::uint32_t k_slices; // > 1: K slices of single-CTA tiles, added by a second kernel
  double us;
};
PresplitChoice choose_presplit(const cuMpSGEMM_handle *h, std::uint64_t m_exp, std::uint64_t n,
                               std::uint64_t k_exp, std::uint64_t batch, bool ec, bool tf32,
                               bool can_slice, bool reads_c) {
  const Tuning &t = h->tuning;
  const PathModel model(h->num_sms, m_exp, n, k_exp, batch, tf32, reads_c);
  PresplitChoice c;
  c.tile = pick_tile(t, h->num_sms, m_exp, n, k_exp, batch, ec, tf32, true);
  c.k_slices = 1;
  c.us = c.tile.us;
  // Few tiles and a long K loop (the shapes the reference hands to its atomic split-K kernel,
  // src/cumpsgemm.cu:272-304): cut K into slices, one CTA each, so that the tiles fill the
  // GPU; the slices' partial sums are added in a fixed order by a second kernel.  The widest
  // tile the problem fills is taken (fewest operand bytes per product), and each slice keeps
  // at least 256 k values.
  const std::uint32_t k_pad64 = static_cast<std::uint32_t>(round_up(k_exp, 64));
  const int wide = t.tile_n != 0 ? t.tile_n : (n > 128) ? 256 : (n > 64 ? 128 : 64);
  const std::uint64_t tiles = ((m_exp + 127) / 128) * ((n + wide - 1) / wide) * batch;
  const bool forced = t.split_k > 1;
  if (can_slice && t.split_k != 0 && t.pair != 1 &&
      (forced || (k_pad64 >= 2048 && 2 * tiles <= h->num_sms))) {
    std::uint32_t wanted = static_cast<std::uint32_t>(h->num_sms / tiles);
    wanted = std::min<std::uint32_t>(wanted, k_pad64 / 256);
    if (forced) wanted = static_cast<std::uint32_t>(t.split_k);
    const std::uint32_t slices = split_k_slices(k_pad64, wanted);
    const double us = slices > 1 ? model.split_k(slices) : 0.0;
    if (slices > 1 && (forced || !ec || t.tile_n != 0 || us < c.us)) {
      c.k_slices = slices;
      c.tile = TileChoice{wide, false, us};
      // (6 us: a third launch, which the choice between slices and tiles has not been given)
      c.us = model.presplit_call(us + 6.0, 128, wide, 0.0, 0.0);
      return c;
    }
  }
  if (!ec) return c; // nothing to compare with
  if (c.tile.pair) {
    const std::uint64_t pair_tiles = model.tiles(256, 256);
    const WorkPlan w = plan_pair(t, tf32, true, static_cast<std::uint32_t>(pair_tiles),
                                 static_cast<std::uint32_t>(model.units), h->num_sms / 2);
    const double parked =
        w.piece_clusters > 0 && w.slice_units == 0 ? w.total_tiles - w.whole_tiles : 0.0;
    c.us = model.presplit_call(c.us, 256, 256, PathModel::waves(w.whole_tiles, model.pairs), parked);
  } else {
    c.us = model.presplit_call(c.us, 128, c.tile.tile_n,
                               PathModel::waves(model.tiles(128, c.tile.tile_n), model.sms), 0.0);
  }
  return c;
}

// Whether a launch of the pair kernel on `batch` products cuts any tile along K, given memory.
bool pair_cuts(const Tuning &t, bool tf32, std::uint64_t m_exp, std::uint64_t n, std::uint32_t k_pad,
               std::uint64_t batch, int clusters) {
  const std::uint64_t tiles = ((m_exp + 255) / 256) * ((n + 255) / 256) * batch;
  return tiles <= 0x7fffffffull &&
         plan_pair(t, tf32, true, static_cast<std::uint32_t>(tiles), k_pad / 64,
                   static_cast<std::uint32_t>(clusters))
                 .piece_clusters > 0;
}

// The reference's module ids name tile classes.
inline unsigned tile_class(int tile_n) { return (tile_n == 256) ? 0u : (tile_n == 128) ? 1u : 2u; }

} // namespace

template <class T>
cublasStatus_t gemm_dispatch(cuMpSGEMM_handle *h, cublasOperation_t op_A, cublasOperation_t op_B,
                             std::uint64_t m, std::uint64_t n, std::uint64_t k, const T *alpha,
                             const T *a, std::uint64_t lda, std::uint64_t stridea, const T *b,
                             std::uint64_t ldb, std::uint64_t strideb, const T *beta, T *c,
                             std::uint64_t ldc, std::uint64_t stridec, std::uint64_t batch,
                             cuMpSGEMM_compute_mode_t mode, const DynParams *dyn,
                             unsigned *used_kernel_module_id, const T *const *a_array,
                             const T *const *b_array, T *const *c_array) {
  constexpr bool is_complex = std::is_same<T, cuComplex>::value;
  if (h == nullptr) return CUBLAS_STATUS_NOT_INITIALIZED;
  if (mode == CUMPSGEMM_DRY_RUN) return CUBLAS_STATUS_SUCCESS;
  h->last_route = CUMPSGEMM_ROUTE_NONE;
  h->last_cut_along_k = false;
  const bool ptr_arrays = (a_array != nullptr) || (b_array != nullptr) || (c_array != nullptr);
  if (ptr_arrays && (a_array == nullptr || b_array == nullptr || c_array == nullptr))
    return CUBLAS_STATUS_INVALID_VALUE;
  if (m == 0 || n == 0 || k == 0 || batch == 0 || alpha == nullptr || beta == nullptr ||
      (!ptr_arrays && (a == nullptr || b == nullptr || c == nullptr)))
    return CUBLAS_STATUS_INVALID_VALUE;
  const bool a_n = (op_A == CUBLAS_OP_N), b_n = (op_B == CUBLAS_OP_N);
  if (lda < (a_n ? m : k) || ldb < (b_n ? k : n) || ldc < m) return CUBLAS_STATUS_INVALID_VALUE;
  if (m > 0x3fffffffull || n > 0x7fffffffull || k > 0x3fffffffull || batch > 0x3fffffffull)
    return CUBLAS_STATUS_INVALID_VALUE;

  bool want_fp16 = false, want_tf32 = false, ec = true;
  switch (mode) {
  case CUMPSGEMM_FP16TCEC:
    want_fp16 = true;
    break;
  case CUMPSGEMM_TF32TCEC:
    want_tf32 = true;
    break;
  case CUMPSGEMM_FP16TC:
    want_fp16 = true;
    ec = false;
    break;
  case CUMPSGEMM_TF32TC:
    want_tf32 = true;
    ec = false;
    break;
  case CUMPSGEMM_AUTO:
    want_fp16 = want_tf32 = true; // both launched, gated on the device-side decision
    break;
  default:
    log_error(std::string("compute mode ") + cuMpSGEMM_get_compute_mode_string(mode) +
              " is not computed by cuMpSGEMM kernels");
    return CUBLAS_STATUS_NOT_SUPPORTED;
  }

  DeviceGuard guard(h->device);
  if (mode == CUMPSGEMM_AUTO && dyn == nullptr) {
    // Direct API use: the caller enabled a flag slot (or none: slot 0 = TF32TCEC).
    DynParams *slot = h->dev_dyn_params + h->dyn_params_next;
    h->dyn_params_next = (h->dyn_params_next + 1) % h->dyn_params_length;
    const unsigned id = h->dyn_launch.enabled ? h->dyn_launch.enabled_id : 0u;
    launch_chained(dyn_params_from_flag_kernel, 1, 1, 0, h->cuda_stream, slot,
                   static_cast<const int *>(h->dyn_launch.flag_buffer + id));
    dyn = slot;
  }

  const std::uint64_t fpe = is_complex ? 2 : 1;
  const std::uint64_t m_exp = m * fpe; // rows of the expanded real problem
  const std::uint64_t k_exp = k * fpe;

  // A single wave of 128 x 64 tiles and at most 12 units of K: that tile has the smallest constant and
  // the smallest slope of all estimates then, so a small call, whose time is mostly the host's,
  // does not work the others out.  (Measured on 183 such problems with k > 128, each kind: never slower
  // than a wider tile; faster than streaming in all FP16TCEC and all but a few TF32TCEC ones, by a quarter on
  // average; 256 x 320 x 720 TF32TCEC, the largest loss, is 6 % slower.)
  const bool small = ec && batch < 8 && k_exp <= 768 && m_exp + n <= 4096 &&
                     h->tuning.untouched() &&
                     ((m_exp + 127) / 128) * ((n + 63) / 64) * batch <= h->num_sms;

  // ---- one launch for what is mostly fixed costs.  A chunk of K (64 values in FP16TCEC, 32 in TF32TCEC)
  // takes this kernel 0.9 to 1.2 us and the pre-split GEMM 0.5, whose second launch costs 2.4 us of
  // host time.  Measured in loops, pre-split / one launch, us: 64^3 8.9 / 6.2, 128^3 8.8 / 6.5, 512 x 512 x
  // 128 8.8 / 6.0 (TF32TCEC, four chunks: 8.5 / 6.6), complex 128^3 (four) 9.3 / 6.7, 256^3 (four) 8.9 /
  // 7.8, 251 x 864 x 300 (five) 8.8 / 10; 1024 x 1024 x 128, 256 tiles, 8.7 / 9.2.  With statistics in
  // front the GPU's time counts and not the host's: 251 x 864 x 300 FP16TCEC_SCALING 14.8 / 16.4.
  const std::uint64_t small_chunks = (k_exp + (want_tf32 ? 31 : 63)) / (want_tf32 ? 32 : 64);
  const std::uint64_t small_tiles = ((m_exp + 127) / 128) * ((n + 31) / 32) * batch;
  if (small && small_tiles <= h->num_sms && small_chunks <= (dyn == nullptr ? 4u : 2u) &&
      lda * fpe <= 0xffffffffull && ldb * fpe <= 0xffffffffull && ldc * fpe <= 0xffffffffull) {
    SmallGemmArgs sa;
    sa.kind = (want_fp16 && want_tf32) ? StreamKind::device
              : want_fp16              ? StreamKind::fp16
                                       : StreamKind::tf32;
    sa.pointers = ptr_arrays;
    sa.a = ptr_arrays ? static_cast<const void *>(a_array) : a;
    sa.b = ptr_arrays ? static_cast<const void *>(b_array) : b;
    sa.c = ptr_arrays ? const_cast<void *>(static_cast<const void *>(c_array)) : c;
    sa.lda = static_cast<std::uint32_t>(lda * fpe);
    sa.ldb = static_cast<std::uint32_t>(ldb * fpe);
    sa.ldc = static_cast<std::uint32_t>(ldc * fpe);
    sa.stride_a = stridea * fpe;
    sa.stride_b = strideb * fpe;
    sa.stride_c = stridec * fpe;
    sa.m = static_cast<std::uint32_t>(m_exp);
    sa.n = static_cast<std::uint32_t>(n);
    sa.k = static_cast<std::uint32_t>(k_exp);
    sa.batch = static_cast<std::uint32_t>(batch);
    sa.a_k_contig = !a_n;
    sa.b_k_contig = b_n;
    sa.is_complex = is_complex;
    sa.conj_a = is_complex && op_A == CUBLAS_OP_C;
    sa.conj_b = is_complex && op_B == CUBLAS_OP_C;
    sa.alpha_r = Scalar<T>::re(alpha);
    sa.alpha_i = Scalar<T>::im(alpha);
    sa.beta_r = Scalar<T>::re(beta);
    sa.beta_i = Scalar<T>::im(beta);
    sa.dyn = dyn;
    sa.dev_status = h->dev_status;
    if (used_kernel_module_id != nullptr) *used_kernel_module_id = tile_class(64);
    const bool prof = h->exp_stats.profiling_enabled;
    if (prof) h->exp_stats.profiler.start("gemm_kernel", h->cuda_stream);
    cuMpSGEMM_handle::TimingTriple tt{};
    if (h->kernel_timing) {
      for (auto &e : tt.e) cudaEventCreate(&e);
      cudaEventRecord(tt.e[0], h->cuda_stream);
      cudaEventRecord(tt.e[1], h->cuda_stream);
    }
    const cudaError_t serr = launch_tcec_gemm_small(sa, h->cuda_stream);
    if (h->kernel_timing) {
      cudaEventRecord(tt.e[2], h->cuda_stream);
      h->timing_events.push_back(tt);
    }
    if (prof) h->exp_stats.profiler.stop("gemm_kernel", h->cuda_stream);
    mark_stream_work(h);
    if (serr != cudaSuccess) {
      log_error(std::string("kernel launch failed: ") + cudaGetErrorString(serr));
      return CUBLAS_STATUS_EXECUTION_FAILED;
    }
    h->last_route = CUMPSGEMM_ROUTE_ON_THE_FLY;
    h->last_tile_rows = 128;
    h->last_tile_cols = 32;
    return CUBLAS_STATUS_SUCCESS;
  }

  // ---- the pre-split path's tile or K slices, and what it would take
  const bool auto_kind = want_fp16 && want_tf32;
  const StreamKind stream_kind = auto_kind ? StreamKind::device
                                 : want_fp16 ? StreamKind::fp16 : StreamKind::tf32;
  PresplitChoice pre = {{64, false, 0.0}, 1, 0.0};
  const bool reads_c = Scalar<T>::re(beta) != 0.f || Scalar<T>::im(beta) != 0.f;
  if (!small) pre = choose_presplit(h, m_exp, n, k_exp, batch, ec, want_tf32, !ptr_arrays, reads_c);
  if (auto_kind && !small)
    pre.us = 0.5 * (pre.us +
                    choose_presplit(h, m_exp, n, k_exp, batch, ec, false, !ptr_arrays, reads_c).us);

  // ---- one launch, operands split between TMA and the tensor core.  Returns whether the call was taken, that is
  // whether the kernel can take it and is estimated to end before `bound_us`.
  cublasStatus_t stream_status = CUBLAS_STATUS_SUCCESS;
  const auto stream_call = [&](double bound_us) {
    StreamGemmArgs ga;
    if (!ec || ptr_arrays ||
        !stream_args<T>(h, op_A, op_B, m, n, k, a, lda, stridea, b, ldb, strideb, batch, reads_c,
                        stream_kind, bound_us, &ga))
      return false;
    if (ga.plan.piece_clusters > 0) {
      const std::size_t bytes = stream_scratch_bytes(ga.plan);
      const std::size_t limit =
          h->workspace_limit_bytes ? h->workspace_limit_bytes : kDefaultWorkspaceLimit;
      if (bytes > limit || !ensure_workspace(h, bytes)) {
        // no room for the pieces' sums: whole tiles only, which need no memory
        ga.plan.whole_tiles = ga.plan.total_tiles;
        ga.plan.piece_clusters = 0;
        ga.plan.slices = 0;
      }
    }
    ga.c = reinterpret_cast<float *>(c);
    ga.ldc = ldc * fpe;
    ga.stride_c = stridec * fpe;
    ga.alpha_r = Scalar<T>::re(alpha);
    ga.alpha_i = Scalar<T>::im(alpha);
    ga.beta_r = Scalar<T>::re(beta);
    ga.beta_i = Scalar<T>::im(beta);
    ga.dyn = dyn;
    ga.dev_status = h->dev_status;
    ga.debug = h->debug_buffer;
    ga.partial = reinterpret_cast<float *>(h->workspace);
    if (used_kernel_module_id != nullptr) {
      *used_kernel_module_id = (ga.plan.slices > 1) ? 100u : tile_class(pre.tile.tile_n);
    }
    const bool prof = h->exp_stats.profiling_enabled;
    if (prof) h->exp_stats.profiler.start("gemm_kernel", h->cuda_stream);
    cuMpSGEMM_handle::TimingTriple tt{};
    if (h->kernel_timing) {
      for (auto &e : tt.e) cudaEventCreate(&e);
      cudaEventRecord(tt.e[0], h->cuda_stream);
      cudaEventRecord(tt.e[1], h->cuda_stream);
    }
    cudaError_t gerr = launch_tcec_gemm_stream(ga, h->cuda_stream);
    const bool addressable = gerr != cudaErrorNotSupported;
    if (h->kernel_timing && addressable) {
      cudaEventRecord(tt.e[2], h->cuda_stream);
      h->timing_events.push_back(tt);
    } else if (h->kernel_timing) {
      for (auto &e : tt.e) cudaEventDestroy(e);
    }
    if (prof) h->exp_stats.profiler.stop("gemm_kernel", h->cuda_stream);
    if (!addressable) return false;
    mark_stream_work(h);
    if (gerr != cudaSuccess) {
      log_error(std::string("kernel launch failed: ") + cudaGetErrorString(gerr));
      stream_status = CUBLAS_STATUS_EXECUTION_FAILED;
      return true;
    }
    h->last_route = CUMPSGEMM_ROUTE_STREAMING;
    h->last_cut_along_k = ga.plan.piece_clusters > 0;
    h->last_tile_rows = ga.plan.tile_m;
    h->last_tile_cols = ga.plan.tile_n;
    return true;
  };
  // (Without statistics in front the host's time counts too: 8.8 us for the two launches of the pre-split path
  // in a loop, 6.6 for one.)
  constexpr double kTwoLaunchesUs = 8.8;
  if (!small && stream_call(dyn == nullptr ? std::max(pre.us, kTwoLaunchesUs) : pre.us)) return stream_status;

  // ---- one launch, no workspace: operands split inside the GEMM kernel (switches only)
  FusedGemmArgs fa;
  if (!small && mode == CUMPSGEMM_FP16TCEC && !ptr_arrays &&
      fused_args<T>(h, op_A, op_B, m, n, k, a, lda, stridea, b, ldb, strideb, batch, &fa)) {
    fa.c = reinterpret_cast<float *>(c);
    fa.ldc = ldc * fpe;
    fa.stride_c = stridec * fpe;
    fa.alpha_r = Scalar<T>::re(alpha);
    fa.alpha_i = Scalar<T>::im(alpha);
    fa.beta_r = Scalar<T>::re(beta);
    fa.beta_i = Scalar<T>::im(beta);
    fa.dyn = dyn;
    fa.dev_status = h->dev_status;
    if (fa.k_slices > 1) {
      const std::size_t bytes = static_cast<std::size_t>(fa.k_slices) * fa.m * fa.n * fa.batch *
                                sizeof(float);
      const std::size_t limit =
          h->workspace_limit_bytes ? h->workspace_limit_bytes : kDefaultWorkspaceLimit;
      if (bytes > limit || !ensure_workspace(h, bytes)) fa.k_slices = 1; // no room: no split
      else fa.partial = reinterpret_cast<float *>(h->workspace);
    }
    if (used_kernel_module_id != nullptr)
      *used_kernel_module_id = (fa.k_slices > 1) ? 100u : (fa.tile_n == 128) ? 1u : 2u;
    const bool prof = h->exp_stats.profiling_enabled;
    if (prof) h->exp_stats.profiler.start("gemm_kernel", h->cuda_stream);
    cuMpSGEMM_handle::TimingTriple tt{};
    if (h->kernel_timing) {
      for (auto &e : tt.e) cudaEventCreate(&e);
      cudaEventRecord(tt.e[0], h->cuda_stream);
      cudaEventRecord(tt.e[1], h->cuda_stream);
    }
    cudaError_t ferr = launch_tcec_gemm_fused(fa, h->cuda_stream);
    if (ferr == cudaSuccess && fa.k_slices > 1) {
      TcecGemmArgs r = {};
      r.m = fa.m;
      r.n = fa.n;
      r.batch = fa.batch;
      r.c = fa.c;
      r.ldc = fa.ldc;
      r.stride_c = fa.stride_c;
      r.alpha_r = fa.alpha_r;
      r.alpha_i = fa.alpha_i;
      r.beta_r = fa.beta_r;
      r.beta_i = fa.beta_i;
      r.is_complex = fa.is_complex;
      r.dyn = fa.dyn;
      r.k_slices = fa.k_slices;
      r.partial = fa.partial;
      ferr = launch_splitk_reduce(r, h->cuda_stream);
    }
    if (h->kernel_timing) {
      cudaEventRecord(tt.e[2], h->cuda_stream);
      h->timing_events.push_back(tt);
    }
    if (prof) h->exp_stats.profiler.stop("gemm_kernel", h->cuda_stream);
    mark_stream_work(h);
    if (ferr != cudaSuccess) {
      log_error(std::string("kernel launch failed: ") + cudaGetErrorString(ferr));
      return CUBLAS_STATUS_EXECUTION_FAILED;
    }
    h->last_route = CUMPSGEMM_ROUTE_ON_THE_FLY;
    h->last_cut_along_k = fa.k_slices > 1;
    h->last_tile_rows = 128;
    h->last_tile_cols = fa.tile_n;
    return CUBLAS_STATUS_SUCCESS;
  }

  const std::uint32_t k_slices = pre.k_slices;
  const int tile_n = pre.tile.tile_n;
  const bool use_pair = pre.tile.pair;
  // tile class, or 100 for the split-K path as in the reference (src/cumpsgemm.cu:283-285)
  if (used_kernel_module_id != nullptr)
    *used_kernel_module_id = (k_slices > 1) ? 100u : tile_class(tile_n);

  const std::uint32_t rows_pad_a =
      static_cast<std::uint32_t>(round_up(m_exp, use_pair ? 256 : 128));
  const std::uint32_t rows_pad_b = static_cast<std::uint32_t>(round_up(n, tile_n));
  const std::uint32_t k_pad = static_cast<std::uint32_t>(round_up(k_exp, 64));
  const std::size_t es_max = want_tf32 ? 4 : 2;
  const std::size_t planes = ec ? 2 : 1;
  const std::size_t bytes_a_1 = planes * rows_pad_a * static_cast<std::size_t>(k_pad) * es_max;
  const std::size_t bytes_b_1 = planes * rows_pad_b * static_cast<std::size_t>(k_pad) * es_max;
  const std::size_t limit =
      h->workspace_limit_bytes ? h->workspace_limit_bytes : kDefaultWorkspaceLimit;
  // split-K partial sums: k_slices blocks of m x n floats per batch entry, behind the panels
  const std::size_t bytes_p_1 =
      (k_slices > 1) ? static_cast<std::size_t>(k_slices) * m_exp * n * sizeof(float) : 0;
  std::uint64_t chunk = std::max<std::uint64_t>(1, limit / (bytes_a_1 + bytes_b_1 + bytes_p_1));
  chunk = std::min<std::uint64_t>(chunk, batch);
  chunk = std::min<std::uint64_t>(chunk, 32768); // planes of a tensor map, tiles of a launch
  const std::size_t bytes_panels = chunk * (bytes_a_1 + bytes_b_1 + bytes_p_1);
  // Scratch for the K pieces of pair tiles (once per call, behind everything else), if any launch
  // of the call cuts one.  It never takes a call over a limit that the panels keep; and where it
  // cannot be had (the workspace of a captured call only holds the panels, no memory) the tiles
  // stay whole.
  std::size_t bytes_tail = 0;
  if (use_pair) {
    int clusters = 1;
    const bool cuts =
        pair_max_clusters(stream_kind, &clusters) == cudaSuccess &&
        (pair_cuts(h->tuning, !want_fp16, m_exp, n, k_pad, chunk, clusters) ||
         (batch % chunk != 0 &&
          pair_cuts(h->tuning, !want_fp16, m_exp, n, k_pad, batch % chunk, clusters)));
    const std::size_t bytes = cuts ? pair_tail_scratch_bytes(h->num_sms) : 0;
    if ((bytes_panels + bytes <= limit || bytes_panels > limit) &&
        ensure_workspace(h, bytes_panels + bytes))
      bytes_tail = bytes;
  }
  if (!ensure_workspace(h, bytes_panels)) {
    // no memory for the panels (a captured call on a handle that has made none of its size before):
    // streaming needs none
    if (stream_call(1e30)) return stream_status;
    log_error(may_allocate(h) ? "failed to allocate the operand workspace"
                              : "the operand workspace cannot grow while the stream is captured; "
                                "make one call of this size before the capture");
    return CUBLAS_STATUS_ALLOC_FAILED;
  }
  char *ws_a = reinterpret_cast<char *>(h->workspace);
  char *ws_b = ws_a + chunk * bytes_a_1;
  float *ws_p = reinterpret_cast<float *>(ws_b + chunk * bytes_b_1);
  float *ws_t = reinterpret_cast<float *>(reinterpret_cast<char *>(ws_p) + chunk * bytes_p_1);

  const bool prof = h->exp_stats.profiling_enabled;
  if (prof) h->exp_stats.profiler.start("gemm_kernel", h->cuda_stream);
  cudaError_t err = cudaSuccess;
  for (std::uint64_t b0 = 0; b0 < batch && err == cudaSuccess; b0 += chunk) {
    const std::uint32_t nb = static_cast<std::uint32_t>(std::min<std::uint64_t>(chunk, batch - b0));
    // AUTO: one split launch and one GEMM launch whose kernels read the device-side decision
    // and run the FP16 or the TF32 pipeline; every other mode: the one kind it names.
    const SplitKind kind = want_fp16 ? SplitKind::fp16 : SplitKind::tf32;
    SplitArgs sa;
    sa.kind = kind;
    sa.operand = Operand::A;
    sa.is_complex = is_complex;
    sa.conjugate = is_complex && op_A == CUBLAS_OP_C;
    sa.src_k_contig = !a_n;
    sa.rows = m;
    sa.k = k;
    sa.src = ptr_arrays ? nullptr : a + b0 * stridea;
    sa.src_array = ptr_arrays ? reinterpret_cast<const void *const *>(a_array + b0) : nullptr;
    sa.ld = lda;
    sa.stride = stridea;
    sa.batch = nb;
    sa.panel = ws_a;
    sa.rows_pad = rows_pad_a;
    sa.k_pad = k_pad;
    sa.with_lo = ec;
    sa.dyn = dyn;
    if (use_pair) sa.zero_word = reinterpret_cast<unsigned int *>(h->dev_status + 1);
    cuMpSGEMM_handle::TimingTriple tt{};
    if (h->kernel_timing) {
      for (auto &e : tt.e) cudaEventCreate(&e);
      cudaEventRecord(tt.e[0], h->cuda_stream);
    }
    SplitArgs sb = sa;
    sb.operand = Operand::B;
    sb.conjugate = is_complex && op_B == CUBLAS_OP_C;
    sb.src_k_contig = b_n;
    sb.rows = n;
    sb.src = ptr_arrays ? nullptr : b + b0 * strideb;
    sb.src_array = ptr_arrays ? reinterpret_cast<const void *const *>(b_array + b0) : nullptr;
    sb.ld = ldb;
    sb.stride = strideb;
    sb.panel = ws_b;
    sb.rows_pad = rows_pad_b;
    err = auto_kind ? launch_split_pair_auto(sa, sb, h->cuda_stream)
                    : launch_split_pair(sa, sb, h->cuda_stream);
    if (err != cudaSuccess) break;
    if (h->kernel_timing) cudaEventRecord(tt.e[1], h->cuda_stream);

    TcecGemmArgs g;
    g.kind = kind;
    g.error_correction = ec;
    g.m = static_cast<std::uint32_t>(m_exp);
    g.n = static_cast<std::uint32_t>(n);
    g.k_pad = k_pad;
    g.rows_pad_a = rows_pad_a;
    g.rows_pad_b = rows_pad_b;
    g.batch = nb;
    g.panel_a = ws_a;
    g.panel_b = ws_b;
    g.c = ptr_arrays ? nullptr : reinterpret_cast<float *>(c + b0 * stridec);
    g.c_array = ptr_arrays ? reinterpret_cast<float *const *>(c_array + b0) : nullptr;
    g.ldc = ldc * fpe;
    g.stride_c = stridec * fpe;
    g.alpha_r = Scalar<T>::re(alpha);
    g.alpha_i = Scalar<T>::im(alpha);
    g.beta_r = Scalar<T>::re(beta);
    g.beta_i = Scalar<T>::im(beta);
    g.is_complex = is_complex;
    g.dyn = dyn;
    g.tile_n = tile_n;
    g.dev_status = h->dev_status;
    g.wave_counter = reinterpret_cast<unsigned int *>(h->dev_status + 1);
    g.debug = h->debug_buffer;
    g.tuning = h->tuning;
    g.k_slices = k_slices;
    g.partial = (k_slices > 1) ? ws_p : nullptr;
    g.tail_partial = bytes_tail > 0 ? ws_t : nullptr;
    if (auto_kind)
      err = use_pair ? launch_tcec_gemm_pair_auto(g, h->cuda_stream)
                     : launch_tcec_gemm_auto(g, h->cuda_stream);
    else
      err = use_pair ? launch_tcec_gemm_pair(g, h->cuda_stream)
                     : launch_tcec_gemm(g, h->cuda_stream);
    if (err == cudaSuccess && k_slices > 1) err = launch_splitk_reduce(g, h->cuda_stream);
    if (h->kernel_timing) {
      cudaEventRecord(tt.e[2], h->cuda_stream);
      h->timing_events.push_back(tt);
    }
  }
  if (prof) h->exp_stats.profiler.stop("gemm_kernel", h->cuda_stream);
  mark_stream_work(h);
  if (err != cudaSuccess) {
    log_error(std::string("kernel launch failed: ") + cudaGetErrorString(err));
    return CUBLAS_STATUS_EXECUTION_FAILED;
  }
  h->last_route = use_pair ? CUMPSGEMM_ROUTE_PRESPLIT_PAIR : CUMPSGEMM_ROUTE_PRESPLIT_SINGLE;
  h->last_cut_along_k = k_slices > 1 || bytes_tail > 0; // (the scratch is only there to be used)
  h->last_tile_rows = use_pair ? 256 : 128;
  h->last_tile_cols = tile_n;
  return CUBLAS_STATUS_SUCCESS;
}

template <class T>
cublasStatus_t gemm_with_statistics(cuMpSGEMM_handle *h, cublasOperation_t op_A,
                                    cublasOperation_t op_B, std::uint64_t m, std::uint64_t n,
                                    std::uint64_t k, const T *alpha, const T *a, std::uint64_t lda,
                                    std::uint64_t stridea, const T *b, std::uint64_t ldb,
                                    std::uint64_t strideb, const T *beta, T *c, std::uint64_t ldc,
                                    std::uint64_t stridec, std::uint64_t batch,
                                    cuMpSGEMM_compute_mode_t mode, unsigned *stats_id_a_out,
                                    unsigned *stats_id_b_out, unsigned *flag_id_out) {
  if (h == nullptr) return CUBLAS_STATUS_NOT_INITIALIZED;
  h->last_route = CUMPSGEMM_ROUTE_NONE;
  if (mode != CUMPSGEMM_AUTO && mode != CUMPSGEMM_FP16TCEC_SCALING)
    return CUBLAS_STATUS_INVALID_VALUE;
  if (m == 0 || n == 0 || k == 0 || batch == 0 || a == nullptr || b == nullptr)
    return CUBLAS_STATUS_INVALID_VALUE;
  if (m > 0xffffffffull || n > 0xffffffffull || k > 0xffffffffull || lda > 0xffffffffull ||
      ldb > 0xffffffffull || stridea > 0xffffffffull || strideb > 0xffffffffull ||
      batch > 0xffffffffull)
    return CUBLAS_STATUS_INVALID_VALUE;
  DeviceGuard guard(h->device);
  // stored extents of A and B (before op)
  const unsigned am = static_cast<unsigned>(op_A == CUBLAS_OP_N ? m : k);
  const unsigned an = static_cast<unsigned>(op_A == CUBLAS_OP_N ? k : m);
  const unsigned bm = static_cast<unsigned>(op_B == CUBLAS_OP_N ? k : n);
  const unsigned bn = static_cast<unsigned>(op_B == CUBLAS_OP_N ? n : k);
  // A batch of one is a single matrix whatever the stride says.
  const unsigned sa = batch > 1 ? static_cast<unsigned>(stridea) : 0u;
  const unsigned sb = batch > 1 ? static_cast<unsigned>(strideb) : 0u;
  unsigned id_a, id_b, flag_id;
  cuMpSGEMM_compute_mode_t gemm_mode;
  const DynParams *dyn;
  const bool fused_scans = !h->exp_stats.profiling_enabled;
  if (fused_scans) {
    // both operands share the scan launches; the slot ids are taken in the usual order
    id_a = next_exp_stats_id(h);
    id_b = next_exp_stats_id(h);
    exp_stats_pair<T>(h, mode == CUMPSGEMM_AUTO, id_a, am, an, a, static_cast<unsigned>(lda), sa,
                      id_b, bm, bn, b, static_cast<unsigned>(ldb), sb,
                      static_cast<unsigned>(batch));
  }
  if (mode == CUMPSGEMM_AUTO) {
    if (!fused_scans) {
      id_a = cumpsgemm::exp_stats_ext<T>(h, am, an, a, static_cast<unsigned>(lda),
                                         static_cast<unsigned>(batch), sa);
      id_b = cumpsgemm::exp_stats_ext<T>(h, bm, bn, b, static_cast<unsigned>(ldb),
                                         static_cast<unsigned>(batch), sb);
    }
    flag_id = next_dyn_launch_id(h);
    dyn = prepare_dyn_params_from_stats(h, flag_id, id_a, id_b);
    gemm_mode = CUMPSGEMM_AUTO;
  } else {
    if (!fused_scans) {
      id_a = cumpsgemm::exp_max_ext<T>(h, am, an, a, static_cast<unsigned>(lda),
                                       static_cast<unsigned>(batch), sa);
      id_b = cumpsgemm::exp_max_ext<T>(h, bm, bn, b, static_cast<unsigned>(ldb),
                                       static_cast<unsigned>(batch), sb);
    }
    flag_id = 1; // reserved slot: FP16TCEC with both scale bits
    dyn = prepare_dyn_params(h, flag_id, id_a, id_b);
    gemm_mode = CUMPSGEMM_FP16TCEC;
  }
  if (stats_id_a_out) *stats_id_a_out = id_a;
  if (stats_id_b_out) *stats_id_b_out = id_b;
  if (flag_id_out) *flag_id_out = flag_id;
  return gemm_dispatch<T>(h, op_A, op_B, m, n, k, alpha, a, lda, stridea, b, ldb, strideb, beta, c,
                          ldc, stridec, batch, gemm_mode, dyn, nullptr);
}

#define INSTANTIATE(T)                                                                            \
  template cublasStatus_t gemm_dispatch<T>(                                                       \
      cuMpSGEMM_handle *, cublasOperation_t, cublasOperation_t, std::uint64_t, std::uint64_t,     \
      std::uint64_t, const T *, const T *, std::uint64_t, std::uint64_t, const T *, std::uint64_t, \
      std::uint64_t, const T *, T *, std::uint64_t, std::uint64_t, std::uint64_t,                 \
      cuMpSGEMM_compute_mode_t, const DynParams *, unsigned *, const T *const *,                  \
      const T *const *, T *const *);                                                              \
  template cublasStatus_t gemm_with_statistics<T>(                                                \
      cuMpSGEMM_handle *, cublasOperation_t, cublasOperation_t, std::uint64_t, std::uint64_t,     \
      std::uint64_t, const T *, const T *, std::uint64_t, std::uint64_t, const T *, std::uint64_t, \
      std::uint64_t, const T *, T *, std::uint64_t, std::uint64_t, std::uint64_t,                 \
      cuMpSGEMM_compute_mode_t, unsigned *, unsigned *, unsigned *);
INSTANTIATE(float)
INSTANTIATE(cuComplex)
#undef INSTANTIATE

} // namespace cumpsgemm_b200

// ---------------------------------------------------------------- public C++ API
namespace cumpsgemm {
using namespace cumpsgemm_b200;

template <class T>
cublasStatus_t gemm(cuMpSGEMM_handle_t handle, const cublasOperation_t op_A,
                    const cublasOperation_t op_B, const uint64_t m, const uint64_t n,
                    const uint64_t k, const T *alpha, const T *const a_dmem_ptr,
                    const uint64_t lda, const T *const b_dmem_ptr, const uint64_t ldb,
                    const T *beta, T *const c_dmem_ptr, const uint64_t ldc,
                    const cuMpSGEMM_compute_mode_t compute_mode,
                    unsigned *const used_kernel_module_id) {
  if (compute_mode == CUMPSGEMM_FP16TCEC_SCALING) {
    return gemm_with_statistics<T>(handle, op_A, op_B, m, n, k, alpha, a_dmem_ptr, lda, 0,
                                   b_dmem_ptr, ldb, 0, beta, c_dmem_ptr, ldc, 0, 1, compute_mode,
                                   nullptr, nullptr, nullptr);
  }
  return gemm_dispatch<T>(handle, op_A, op_B, m, n, k, alpha, a_dmem_ptr, lda, 0, b_dmem_ptr, ldb,
                          0, beta, c_dmem_ptr, ldc, 0, 1, compute_mode, nullptr,
                          used_kernel_module_id);
}

template <class T>
cublasStatus_t gemm_stridedBatch(cuMpSGEMM_handle_t handle, const cublasOperation_t op_A,
                                 const cublasOperation_t op_B, const uint64_t m, const uint64_t n,
                                 const uint64_t k, const T *alpha, const T *const a_dmem_ptr,
                                 const uint64_t lda, const uint64_t stridea,
                                 const T *const b_dmem_ptr, const uint64_t ldb,
                                 const uint64_t strideb, const T *beta, T *const c_dmem_ptr,
                                 const uint64_t ldc, const uint64_t stridec,
                                 const uint64_t batch_count,
                                 const cuMpSGEMM_compute_mode_t compute_mode,
                                 unsigned *const used_kernel_module_id) {
  if (compute_mode == CUMPSGEMM_FP16TCEC_SCALING) {
    return gemm_with_statistics<T>(handle, op_A, op_B, m, n, k, alpha, a_dmem_ptr, lda, stridea,
                                   b_dmem_ptr, ldb, strideb, beta, c_dmem_ptr, ldc, stridec,
                                   batch_count, compute_mode, nullptr, nullptr, nullptr);
  }
  return gemm_dispatch<T>(handle, op_A, op_B, m, n, k, alpha, a_dmem_ptr, lda, stridea,
                          b_dmem_ptr, ldb, strideb, beta, c_dmem_ptr, ldc, stridec, batch_count,
                          compute_mode, nullptr, used_kernel_module_id);
}

#define INSTANTIATE(T)                                                                           \
  template cublasStatus_t gemm<T>(cuMpSGEMM_handle_t, const cublasOperation_t,                   \
                                  const cublasOperation_t, const uint64_t, const uint64_t,       \
                                  const uint64_t, const T *, const T *const, const uint64_t,     \
                                  const T *const, const uint64_t, const T *, T *const,           \
                                  const uint64_t, const cuMpSGEMM_compute_mode_t,                \
                                  unsigned *const);                                              \
  template cublasStatus_t gemm_stridedBatch<T>(                                                  \
      cuMpSGEMM_handle_t, const cublasOperation_t, const cublasOperation_t, const uint64_t,      \
      const uint64_t, const uint64_t, const T *, const T *const, const uint64_t, const uint64_t, \
      const T *const, const uint64_t, const uint64_t, const T *, T *const, const uint64_t,       \
      const uint64_t, const uint64_t, const cuMpSGEMM_compute_mode_t, unsigned *const);
INSTANTIATE(float)
INSTANTIATE(cuComplex)
#undef INSTANTIATE
} // namespace cumpsgemm

// ---------------------------------------------------------------- C ABI
extern "C" {

cublasStatus_t cuMpSGEMM_sgemm(cuMpSGEMM_handle_t handle, const cublasOperation_t op_A,
                               const cublasOperation_t op_B, const uint64_t m, const uint64_t n,
                               const uint64_t k, const float *alpha, const float *const a_dmem_ptr,
                               const uint64_t lda, const float *const b_dmem_ptr,
                               const uint64_t ldb, const float *beta, float *const c_dmem_ptr,
                               const uint64_t ldc, const cuMpSGEMM_compute_mode_t compute_mode) {
  if (op_A == CUBLAS_OP_C || op_B == CUBLAS_OP_C) return CUBLAS_STATUS_INVALID_VALUE;
  return cumpsgemm::gemm<float>(handle, op_A, op_B, m, n, k, alpha, a_dmem_ptr, lda, b_dmem_ptr,
                                ldb, beta, c_dmem_ptr, ldc, compute_mode);
}

cublasStatus_t cuMpSGEMM_cgemm(cuMpSGEMM_handle_t handle, const cublasOperation_t op_A,
                               const cublasOperation_t op_B, const uint64_t m, const uint64_t n,
                               const uint64_t k, const cuComplex *alpha,
                               const cuComplex *const a_dmem_ptr, const uint64_t lda,
                               const cuComplex *const b_dmem_ptr, const uint64_t ldb,
                               const cuComplex *beta, cuComplex *const c_dmem_ptr,
                               const uint64_t ldc, const cuMpSGEMM_compute_mode_t compute_mode) {
  return cumpsgemm::gemm<cuComplex>(handle, op_A, op_B, m, n, k, alpha, a_dmem_ptr, lda,
                                    b_dmem_ptr, ldb, beta, c_dmem_ptr, ldc, compute_mode);
}

cublasStatus_t cuMpSGEMM_sgemm_strided_batch(
    cuMpSGEMM_handle_t handle, const cublasOperation_t op_A, const cublasOperation_t op_B,
    const uint64_t m, const uint64_t n, const uint64_t k, const float *alpha,
    const float *const a_dmem_ptr, const uint64_t lda, const uint64_t stridea,
    const float *const b_dmem_ptr, const uint64_t ldb, const uint64_t strideb, const float *beta,
    float *const c_dmem_ptr, const uint64_t ldc, const uint64_t stridec,
    const uint64_t batch_count, const cuMpSGEMM_compute_mode_t compute_mode) {
  if (op_A == CUBLAS_OP_C || op_B == CUBLAS_OP_C) return CUBLAS_STATUS_INVALID_VALUE;
  return cumpsgemm::gemm_stridedBatch<float>(handle, op_A, op_B, m, n, k, alpha, a_dmem_ptr, lda,
                                             stridea, b_dmem_ptr, ldb, strideb, beta, c_dmem_ptr,
                                             ldc, stridec, batch_count, compute_mode);
}

cublasStatus_t cuMpSGEMM_cgemm_strided_batch(
    cuMpSGEMM_handle_t handle, const cublasOperation_t op_A, const cublasOperation_t op_B,
    const uint64_t m, const uint64_t n, const uint64_t k, const cuComplex *alpha,
    const cuComplex *const a_dmem_ptr, const uint64_t lda, const uint64_t stridea,
    const cuComplex *const b_dmem_ptr, const uint64_t ldb, const uint64_t strideb,
    const cuComplex *beta, cuComplex *const c_dmem_ptr, const uint64_t ldc,
    const uint64_t stridec, const uint64_t batch_count,
    const cuMpSGEMM_compute_mode_t compute_mode) {
  return cumpsgemm::gemm_stridedBatch<cuComplex>(handle, op_A, op_B, m, n, k, alpha, a_dmem_ptr,
                                                 lda, stridea, b_dmem_ptr, ldb, strideb, beta,
                                                 c_dmem_ptr, ldc, stridec, batch_count,
                                                 compute_mode);
}

} // extern "C"
