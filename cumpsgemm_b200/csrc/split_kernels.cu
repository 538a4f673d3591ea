// Operand split pass: FP32 / complex64 column-major operand -> K-major hi/lo panels.
//
// Restates, as one HBM-bound pass per operand, the FP32 -> (hi, lo) split the
// reference performs inside its fragment loads for every warp and every k-step
// (src/device_tcec_wrapper.hpp:72-80 calling mtk::wmma::tcec::load_matrix_sync),
// together with the operand addressing of its global->shared loaders
// (src/dmem_accessor.hpp:8-170: op N/T/C, leading dimension, edge zero fill,
// conjugation).
//
//   FP16:  hi = RN_fp16(v),  lo = RN_fp16((v - float(hi)) * 2^11)
//   TF32:  hi = RNA_tf32(v), lo = RNA_tf32(v - hi)
// where v = x * scale (scale is an exact power of two, 1 when no scaling).
//
// Panel layout (element type half or float), blocked along K in units of 128 bytes
// (KBE = 64 half or 32 float elements), z = 0 (hi), 1 (lo):
//   panel[(((b * planes + z) * (k_pad / KBE) + kk / KBE) * rows_pad + r) * KBE + kk % KBE]
// so the 128-byte K slices of consecutive rows are contiguous: the box one TMA load of the
// GEMM kernel fetches (128 rows x 128 bytes) is one 16 KiB run of memory instead of 128 lines
// a whole panel row apart.  rows_pad / k_pad are multiples of 64 and every padding element is
// written as zero on every call, so the GEMM kernel needs no edge handling.
//
// Complex operands are expanded to real ones so that the GEMM kernel is a real
// GEMM producing interleaved (re, im) rows of C:
//   A' (2m x 2k): rows (2i, 2i+1), cols (2l, 2l+1) = [[re, -im], [im, re]] of a(i,l)
//   B' (n x 2k):  row j, cols (2l, 2l+1) = (re, im) of b(l,j)
// (a, b after op; op C conjugates).
#include "internal.hpp"

#include <cuda_fp16.h>

namespace cumpsgemm_b200 {
namespace {

constexpr int TILE = 64;       // expanded rows and expanded K per CTA
constexpr int THREADS = 256;

__device__ __forceinline__ float to_tf32(float v) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
  return __uint_as_float(r);
}

// Offset of element (r, kk) inside one plane of a panel (see the layout above).
template <int KIND>
__device__ __forceinline__ uint64_t panel_offset(uint64_t r, uint64_t kk, uint32_t rows_pad) {
  constexpr uint64_t KBE = (KIND == 0) ? 64 : 32;
  return ((kk / KBE) * rows_pad + r) * KBE + (kk % KBE);
}

// Eight lanes (g = 0..7) share the 64 k values of a row.  Which of them lane g converts is chosen so
// that every 16-byte store of the eight lanes together fills whole 128-byte lines of the panel: 8g
// ... 8g + 7 for FP16 (one store per plane), 4g ... 4g + 3 and 32 + 4g ... for TF32 (two).
template <int KIND> __device__ __forceinline__ int k_of(int g, int j) {
  if constexpr (KIND == 0) return 8 * g + j;
  return (j < 4) ? 4 * g + j : 32 + 4 * g + (j - 4);
}

// Splits lane g's eight values of row r, k values k0 + k_of(g, j), and stores them to the panel
// (`batch_off`: first element of this batch entry's hi plane).
template <int KIND>
__device__ __forceinline__ void convert_store8(const float (&v)[8], void *panel, uint64_t batch_off,
                                               uint64_t r, uint64_t k0, int g, uint32_t rows_pad,
                                               uint64_t plane_elems, uint32_t planes) {
  if constexpr (KIND == 0) {
    __align__(16) __half hi[8];
    __align__(16) __half lo[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      hi[j] = __float2half_rn(v[j]);
      lo[j] = __float2half_rn((v[j] - __half2float(hi[j])) * 2048.f);
    }
    __half *ph = reinterpret_cast<__half *>(panel) + batch_off +
                 panel_offset<KIND>(r, k0 + 8 * g, rows_pad);
    *reinterpret_cast<uint4 *>(ph) = *reinterpret_cast<const uint4 *>(hi);
    if (planes == 2)
      *reinterpret_cast<uint4 *>(ph + plane_elems) = *reinterpret_cast<const uint4 *>(lo);
  } else {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      __align__(16) float hi[4];
      __align__(16) float lo[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        hi[j] = to_tf32(v[4 * half + j]);
        lo[j] = to_tf32(v[4 * half + j] - hi[j]);
      }
      float *ph = reinterpret_cast<float *>(panel) + batch_off +
                  panel_offset<KIND>(r, k0 + 32 * half + 4 * g, rows_pad);
      *reinterpret_cast<uint4 *>(ph) = *reinterpret_cast<const uint4 *>(hi);
      if (planes == 2)
        *reinterpret_cast<uint4 *>(ph + plane_elems) = *reinterpret_cast<const uint4 *>(lo);
    }
  }
}

struct SplitParams {
  const float *src; // complex sources are addressed as pairs of floats
  const float *const *src_array; // pointer-array batches: matrix b starts at src_array[b]
  uint64_t ld, stride;
  uint64_t rows, k; // logical source extent (complex elements for complex input)
  void *panel;
  uint32_t rows_pad, k_pad;
  uint32_t planes; // 1 or 2
  const DynParams *dyn;
  int operand; // 0 = A, 1 = B
  int conj;
  int src_k_contig;
};

// MODE: 0 = real, 1 = complex A', 2 = complex B'
template <int KIND, int MODE>
__device__ __forceinline__ void split_generic_body(const SplitParams &p, const uint3 bid,
                                                   float (*tile)[TILE + 1]) {
  constexpr int MY_MODE = (KIND == 0) ? CUMPSGEMM_FP16TCEC : CUMPSGEMM_TF32TCEC;
  float scale = 1.f;
  if (p.dyn != nullptr) {
    if (p.dyn->gemm_mode != MY_MODE) return;
    scale = (p.operand == 0) ? p.dyn->scale_a : p.dyn->scale_b;
  }

  // Source tile in source coordinates; complex tiles store (re, im) in adjacent columns.
  constexpr int SR = (MODE == 1) ? TILE / 2 : TILE; // source rows per tile
  constexpr int SK = (MODE == 0) ? TILE : TILE / 2; // source k per tile
  constexpr int ES = (MODE == 0) ? 1 : 2;           // floats per source element

  const uint32_t b = bid.z;
  const uint64_t r0 = static_cast<uint64_t>(bid.y) * SR;
  const uint64_t k0 = static_cast<uint64_t>(bid.x) * SK;
  const float *src = (p.src_array != nullptr)
                         ? p.src_array[b]
                         : p.src + static_cast<uint64_t>(b) * p.stride * ES;

  // ---- phase 1: coalesced read along the source-contiguous dimension
  if constexpr (ES == 2) {
    // Complex: a thread's 4 (A') or 8 (B') loads are all issued before the first
    // shared-memory store; with one load per store the kernel spent over half of its warp
    // cycles waiting for the load just issued.
    constexpr int PER = SR * SK / THREADS;
    float2 v[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int idx = threadIdx.x + q * THREADS;
      const int r = p.src_k_contig ? idx / SK : idx % SR;
      const int kk = p.src_k_contig ? idx % SK : idx / SR;
      const uint64_t gr = r0 + r, gk = k0 + kk;
      v[q] = make_float2(0.f, 0.f);
      if (gr < p.rows && gk < p.k)
        v[q] = reinterpret_cast<const float2 *>(src)[p.src_k_contig ? (gk + gr * p.ld)
                                                                    : (gr + gk * p.ld)];
    }
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int idx = threadIdx.x + q * THREADS;
      const int r = p.src_k_contig ? idx / SK : idx % SR;
      const int kk = p.src_k_contig ? idx % SK : idx / SR;
      tile[r][2 * kk] = v[q].x * scale;
      tile[r][2 * kk + 1] = (p.conj ? -v[q].y : v[q].y) * scale;
    }
  } else {
    // Real: sources whose rows do not start on 16-byte boundaries, read 4 bytes per lane along the
    // contiguous dimension, all sixteen loads of a thread issued before the first store.  (One load
    // per store and a division per element, as first written: 47 us for the 56 MB of operands of
    // 1999 x 3001 x 2777, now 22; the panels are another 58 MB.)
    constexpr int PER = SR * SK / THREADS;
    const int fast = threadIdx.x % TILE, slow = threadIdx.x / TILE; // SR == SK == TILE
    constexpr int STEP = THREADS / TILE;
    float v[PER];
    const bool kc = p.src_k_contig != 0;
    const uint64_t f0 = (kc ? k0 : r0) + fast, s0 = (kc ? r0 : k0) + slow;
    const uint64_t f_end = kc ? p.k : p.rows, s_end = kc ? p.rows : p.k;
    const float *q = src + f0 + s0 * p.ld;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      v[i] = (f0 < f_end && s0 + i * STEP < s_end) ? *q : 0.f;
      q += STEP * p.ld;
    }
    // lanes run along k or along the rows; a row of the tile is 65 floats, so neither conflicts
    float *t = kc ? &tile[slow][fast] : &tile[fast][slow];
    const int step = kc ? STEP * (TILE + 1) : STEP;
#pragma unroll
    for (int i = 0; i < PER; ++i) t[i * step] = v[i] * scale;
  }
  __syncthreads();

  // ---- phase 2: each thread converts 8 expanded-K values of one expanded row
  const uint64_t er0 = static_cast<uint64_t>(bid.y) * TILE; // expanded row origin
  const uint64_t ek0 = static_cast<uint64_t>(bid.x) * TILE; // expanded K origin
  const uint64_t plane_elems = static_cast<uint64_t>(p.rows_pad) * p.k_pad;
#pragma unroll
  for (int it = 0; it < TILE * TILE / (THREADS * 8); ++it) {
    const int er = (threadIdx.x >> 3) + it * (THREADS >> 3);
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int c = k_of<KIND>(threadIdx.x & 7, j);
      if constexpr (MODE == 0 || MODE == 2) {
        v[j] = tile[er][c];
      } else {
        const int sr = er >> 1;
        const bool im_row = (er & 1) != 0;
        const bool odd = (c & 1) != 0;
        // [[re, -im], [im, re]]
        const float x = tile[sr][(c & ~1) + ((im_row != odd) ? 1 : 0)];
        v[j] = (!im_row && odd) ? -x : x;
      }
    }
    convert_store8<KIND>(v, p.panel, static_cast<uint64_t>(b) * p.planes * plane_elems, er0 + er, ek0,
                         threadIdx.x & 7, p.rows_pad, plane_elems, p.planes);
  }
}

// ---------------------------------------------------------------- vectorised real paths
// Used when the source base address, leading dimension and batch stride are multiples of
// 16 bytes; anything else (and every complex operand) takes split_kernel above.

// float4 at p if the whole vector is inside [.., limit), element-wise with zero fill otherwise
__device__ __forceinline__ float4 load4_guarded(const float *p, uint64_t first, uint64_t limit,
                                                bool row_ok) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (!row_ok) return v;
  if (first + 4 <= limit) return *reinterpret_cast<const float4 *>(p);
  if (first + 0 < limit) v.x = p[0];
  if (first + 1 < limit) v.y = p[1];
  if (first + 2 < limit) v.z = p[2];
  return v;
}

// Source is K-contiguous (element (r, kk) at [kk + r*ld]): no transpose, no shared memory.
// CTA = 128 rows x 64 k; thread = 4 rows x 8 consecutive k, all eight 16-byte loads first.
template <int KIND>
__device__ __forceinline__ void split_kcontig_body(const SplitParams &p, const uint3 bid) {
  constexpr int MY_MODE = (KIND == 0) ? CUMPSGEMM_FP16TCEC : CUMPSGEMM_TF32TCEC;
  float scale = 1.f;
  if (p.dyn != nullptr) {
    if (p.dyn->gemm_mode != MY_MODE) return;
    scale = (p.operand == 0) ? p.dyn->scale_a : p.dyn->scale_b;
  }
  const uint32_t b = bid.z;
  const float *src = p.src + static_cast<uint64_t>(b) * p.stride;
  const int g = threadIdx.x & 7;
  const uint64_t k0 = static_cast<uint64_t>(bid.x) * 64;
  const uint64_t ka = k0 + k_of<KIND>(g, 0), kb = k0 + k_of<KIND>(g, 4); // its two groups of four
  const uint64_t r_base = static_cast<uint64_t>(bid.y) * 128 + (threadIdx.x >> 3);
  const uint64_t plane_elems = static_cast<uint64_t>(p.rows_pad) * p.k_pad;
  float4 x[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint64_t r = r_base + i * 32;
    const bool row_ok = r < p.rows;
    const float *q = src + r * p.ld;
    x[i][0] = load4_guarded(q + ka, ka, p.k, row_ok);
    x[i][1] = load4_guarded(q + kb, kb, p.k, row_ok);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint64_t r = r_base + i * 32;
    if (r >= p.rows_pad) continue;
    const float v[8] = {x[i][0].x * scale, x[i][0].y * scale, x[i][0].z * scale, x[i][0].w * scale,
                        x[i][1].x * scale, x[i][1].y * scale, x[i][1].z * scale, x[i][1].w * scale};
    convert_store8<KIND>(v, p.panel, static_cast<uint64_t>(b) * p.planes * plane_elems, r, k0, g,
                         p.rows_pad, plane_elems, p.planes);
  }
}

// Source is row-contiguous (element (r, kk) at [r + kk*ld]): 64 x 64 transpose through
// shared memory with 16-byte loads along r.
template <int KIND>
__device__ __forceinline__ void split_rcontig_body(const SplitParams &p, const uint3 bid,
                                                   float (*tile)[TILE + 1]) {
  constexpr int MY_MODE = (KIND == 0) ? CUMPSGEMM_FP16TCEC : CUMPSGEMM_TF32TCEC;
  float scale = 1.f;
  if (p.dyn != nullptr) {
    if (p.dyn->gemm_mode != MY_MODE) return;
    scale = (p.operand == 0) ? p.dyn->scale_a : p.dyn->scale_b;
  }
  const uint32_t b = bid.z;
  const float *src = p.src + static_cast<uint64_t>(b) * p.stride;
  const uint64_t r0 = static_cast<uint64_t>(bid.y) * TILE;
  const uint64_t k0 = static_cast<uint64_t>(bid.x) * TILE;
  const int r4 = (threadIdx.x & 15) * 4;
  const int kq = threadIdx.x >> 4; // 0..15
  float4 x[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint64_t gk = k0 + kq + i * 16;
    x[i] = load4_guarded(src + gk * p.ld + r0 + r4, r0 + r4, p.rows, gk < p.k);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int kk = kq + i * 16;
    tile[r4 + 0][kk] = x[i].x * scale;
    tile[r4 + 1][kk] = x[i].y * scale;
    tile[r4 + 2][kk] = x[i].z * scale;
    tile[r4 + 3][kk] = x[i].w * scale;
  }
  __syncthreads();
  const uint64_t plane_elems = static_cast<uint64_t>(p.rows_pad) * p.k_pad;
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int er = (threadIdx.x >> 3) + it * 32;
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = tile[er][k_of<KIND>(threadIdx.x & 7, j)];
    convert_store8<KIND>(v, p.panel, static_cast<uint64_t>(b) * p.planes * plane_elems, r0 + er, k0,
                         threadIdx.x & 7, p.rows_pad, plane_elems, p.planes);
  }
}

// Which body handles an operand.
enum SplitPath : int { kPathReal = 0, kPathComplexA = 1, kPathComplexB = 2, kPathKContig = 3, kPathRContig = 4 };

// Which bodies a kernel contains.  Both operands of a call are real or both complex; keeping the
// sets apart keeps the register counts of the latency-bound generic bodies low, which is what
// decides how many of their blocks are resident.
enum SplitSet : int { kSetComplex = 0, kSetReal = 1, kSetRealVec = 2 };
template <int SET> constexpr int min_blocks() { return SET == kSetRealVec ? 5 : 6; }

template <int KIND, int SET>
__device__ __forceinline__ void split_dispatch(const SplitParams &p, int path, const uint3 bid,
                                               float (*tile)[TILE + 1]) {
  if constexpr (SET == kSetComplex) {
    if (path == kPathComplexA) split_generic_body<KIND, 1>(p, bid, tile);
    else split_generic_body<KIND, 2>(p, bid, tile);
  } else if constexpr (SET == kSetReal) {
    split_generic_body<KIND, 0>(p, bid, tile);
  } else {
    switch (path) {
    case kPathReal:
      split_generic_body<KIND, 0>(p, bid, tile);
      break;
    case kPathKContig:
      split_kcontig_body<KIND>(p, bid);
      break;
    default:
      split_rcontig_body<KIND>(p, bid, tile);
      break;
    }
  }
}

// One launch splits both operands of a GEMM: the first blocks_a blocks work on op(A), the
// rest on op(B).  Saves a launch (and its gap) per GEMM call, which matters for small problems.
struct SplitJob {
  SplitParams p;
  int path;
  uint32_t gx, gy, gz;
};

// The wave counter of the pair kernel behind the split pass starts from zero: written here it
// costs nothing, where a memset between the two kernels would cost a launch and keep them from
// being chained (4 us a call).
__device__ __forceinline__ void zero_word(unsigned int *z) {
  if (z != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *z = 0u;
}

template <int KIND, int SET>
__global__ void __launch_bounds__(THREADS, min_blocks<SET>())
    split_dual_kernel(const SplitJob a, const SplitJob b, unsigned int *z) {
  __shared__ float tile[TILE][TILE + 1]; // transposing staging tile shared by all paths
  // Chained behind the kernel that writes the scaling constants (AUTO / FP16TCEC_SCALING), and
  // the GEMM kernel that follows may be scheduled while this one drains: its prologue does not
  // depend on the panels, and its first panel load waits for this grid to complete.
  CUMPSGEMM_CHAINED_KERNEL_ENTRY();
  zero_word(z);
  const uint32_t blocks_a = a.gx * a.gy * a.gz;
  uint32_t id = blockIdx.x;
  const SplitJob &j = (id < blocks_a) ? a : b;
  if (id >= blocks_a) id -= blocks_a;
  const uint3 bid = make_uint3(id % j.gx, (id / j.gx) % j.gy, id / (j.gx * j.gy));
  split_dispatch<KIND, SET>(j.p, j.path, bid, tile);
}

// AUTO: the kind (FP16 or TF32 panels) is decided on the device.  Job geometry, source
// addressing and the workspace are the same for both kinds, so one launch reads the decision
// and runs the matching bodies (the reference launches the kernels of both kinds and lets the
// deselected one exit, src/cumpsgemm_kernel.cuh:478-489).
template <int SET>
__global__ void __launch_bounds__(THREADS, min_blocks<SET>())
    split_dual_auto_kernel(const SplitJob a, const SplitJob b, unsigned int *z) {
  __shared__ float tile[TILE][TILE + 1];
  CUMPSGEMM_CHAINED_KERNEL_ENTRY(); // see split_dual_kernel
  zero_word(z);
  const uint32_t blocks_a = a.gx * a.gy * a.gz;
  uint32_t id = blockIdx.x;
  const SplitJob &j = (id < blocks_a) ? a : b;
  if (id >= blocks_a) id -= blocks_a;
  const uint3 bid = make_uint3(id % j.gx, (id / j.gx) % j.gy, id / (j.gx * j.gy));
  if (j.p.dyn->gemm_mode == CUMPSGEMM_TF32TCEC)
    split_dispatch<1, SET>(j.p, j.path, bid, tile);
  else
    split_dispatch<0, SET>(j.p, j.path, bid, tile);
}

bool make_job(const SplitArgs &a, SplitJob *job) {
  if ((a.rows_pad % TILE) != 0 || (a.k_pad % TILE) != 0) return false;
  SplitParams &p = job->p;
  p.src = reinterpret_cast<const float *>(a.src);
  p.src_array = reinterpret_cast<const float *const *>(a.src_array);
  p.ld = a.ld;
  p.stride = a.stride;
  p.rows = a.rows;
  p.k = a.k;
  p.panel = a.panel;
  p.rows_pad = a.rows_pad;
  p.k_pad = a.k_pad;
  p.planes = a.with_lo ? 2u : 1u;
  p.dyn = a.dyn;
  p.operand = static_cast<int>(a.operand);
  p.conj = a.conjugate ? 1 : 0;
  p.src_k_contig = a.src_k_contig ? 1 : 0;
  job->gx = a.k_pad / TILE;
  job->gy = a.rows_pad / TILE;
  job->gz = a.batch;
  if (a.is_complex) {
    job->path = (a.operand == Operand::A) ? kPathComplexA : kPathComplexB;
  } else {
    const bool aligned = ((reinterpret_cast<uintptr_t>(a.src) & 15u) == 0) && (a.ld % 4 == 0) &&
                         (a.stride % 4 == 0);
    if (!aligned || a.src_array != nullptr) { // per-matrix alignment is unknown on the host
      job->path = kPathReal;
    } else if (a.src_k_contig) {
      job->path = kPathKContig;
      job->gy = (a.rows_pad + 127) / 128;
    } else {
      job->path = kPathRContig;
    }
  }
  return static_cast<uint64_t>(job->gx) * job->gy * job->gz <= 0x3fffffffull;
}

SplitSet split_set(const SplitArgs &a, const SplitJob &ja, const SplitJob &jb) {
  if (a.is_complex) return kSetComplex;
  return (ja.path >= kPathKContig || jb.path >= kPathKContig) ? kSetRealVec : kSetReal;
}

} // namespace

cudaError_t launch_split_pair_auto(const SplitArgs &a, const SplitArgs &b, cudaStream_t stream) {
  if (a.dyn == nullptr || b.dyn != a.dyn) return cudaErrorInvalidValue;
  SplitJob ja, jb;
  unsigned int *z = a.zero_word;
  if (!make_job(a, &ja) || !make_job(b, &jb)) return cudaErrorInvalidValue;
  const uint64_t blocks = static_cast<uint64_t>(ja.gx) * ja.gy * ja.gz +
                          static_cast<uint64_t>(jb.gx) * jb.gy * jb.gz;
  if (blocks == 0 || blocks > 0x7fffffffull) return cudaErrorInvalidValue;
  const unsigned grid = static_cast<unsigned>(blocks);
  switch (split_set(a, ja, jb)) {
  case kSetComplex:
    return launch_chained(split_dual_auto_kernel<kSetComplex>, grid, THREADS, 0, stream, ja, jb, z);
  case kSetReal:
    return launch_chained(split_dual_auto_kernel<kSetReal>, grid, THREADS, 0, stream, ja, jb, z);
  default:
    return launch_chained(split_dual_auto_kernel<kSetRealVec>, grid, THREADS, 0, stream, ja, jb, z);
  }
}

namespace {
template <int KIND>
cudaError_t launch_set(SplitSet set, unsigned grid, cudaStream_t stream, const SplitJob &ja,
                       const SplitJob &jb, unsigned int *z) {
  switch (set) {
  case kSetComplex:
    return launch_chained(split_dual_kernel<KIND, kSetComplex>, grid, THREADS, 0, stream, ja, jb, z);
  case kSetReal:
    return launch_chained(split_dual_kernel<KIND, kSetReal>, grid, THREADS, 0, stream, ja, jb, z);
  default:
    return launch_chained(split_dual_kernel<KIND, kSetRealVec>, grid, THREADS, 0, stream, ja, jb, z);
  }
}
} // namespace

cudaError_t launch_split_pair(const SplitArgs &a, const SplitArgs &b, cudaStream_t stream) {
  if (a.kind != b.kind) return cudaErrorInvalidValue;
  SplitJob ja, jb;
  unsigned int *z = a.zero_word;
  if (!make_job(a, &ja) || !make_job(b, &jb)) return cudaErrorInvalidValue;
  const uint64_t blocks = static_cast<uint64_t>(ja.gx) * ja.gy * ja.gz +
                          static_cast<uint64_t>(jb.gx) * jb.gy * jb.gz;
  if (blocks == 0 || blocks > 0x7fffffffull) return cudaErrorInvalidValue;
  const unsigned grid = static_cast<unsigned>(blocks);
  const SplitSet set = split_set(a, ja, jb);
  return a.kind == SplitKind::fp16 ? launch_set<0>(set, grid, stream, ja, jb, z)
                                   : launch_set<1>(set, grid, stream, ja, jb, z);
}

} // namespace cumpsgemm_b200
