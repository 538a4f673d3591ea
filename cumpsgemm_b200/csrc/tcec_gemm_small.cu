// Error-corrected tensor-core GEMM for small products: one launch, no workspace, any operand.
//
// A small call is fixed costs: with a split pass in front it is two launches, each about 2.4 us of
// host time, and the panels cross L2 twice.  Here every CTA owns a 128 x 32 tile of C, loads its rows of
// op(A) and op(B) straight into registers (any alignment, op, real or complex, strided or by pointer
// array), splits them (same bits as split_kernels.cu) into 128-byte-swizzled K-major tiles in shared
// memory and multiplies those.  Every element of A is converted n / 32 times, which is what limits the
// kernel to products whose tiles all run at once (see the rule in gemm_api.cu).
//
// One chunk is 128 bytes of K (64 FP16, 32 TF32 values), as a stage is in tcec_gemm.cu, and the sums are
// formed in the same order as there in narrow tiles: hi*hi and the corrections of a chunk, each added to
// an FP32 register sum of its own outside the tensor core.  All warps do everything: while the loads of
// chunk c + 1 are on their way they convert chunk c, one thread issues its products, and then they
// drain chunk c - 1.  Two stages and two accumulators are enough for that: a stage is overwritten two
// chunks later, after its products have been drained.  (At 64 registers a thread two CTAs would fit on
// an SM; what that spills costs more: complex 128^3 7.3 us against 6.7.)
//
// What bounds it: host time (one launch and its arguments, about 6 us a call in a loop), and on the GPU the
// chain of a chunk: loads from L2, conversion, barrier, products, drain.  Measured beside its rule.
//
// Every wait is bounded; a wait that gives up is seen by all threads at the next barrier.
#include "gemm_common.cuh"
#include "ptx.cuh"
#include "split_math.cuh"

#include <mutex>

namespace cumpsgemm_b200 {
namespace {

constexpr int BM = 128, BN = 32;
constexpr int NUM_THREADS = 512, NUM_WARPS = NUM_THREADS / 32;
constexpr int COLS = BN / (NUM_WARPS / 4); // columns of C per thread
constexpr uint32_t A_TILE = BM * kGemmRowBytes, B_TILE = BN * kGemmRowBytes;
constexpr uint32_t STAGE_BYTES = 2 * (A_TILE + B_TILE);
constexpr int SMEM_BYTES = 2 * STAGE_BYTES + 1024;
constexpr uint32_t TMEM_COLS = 128; // two accumulators of hi*hi | hi*lo + lo*hi
constexpr uint32_t D_COLS = 2 * BN;

// How an operand lies in memory (r: row of op(A) or column of op(B), after the complex expansion).
enum Layout : int {
  kK = 0,  // K contiguous: real operands, complex B with op N (interleaved re, im)
  kR = 1,  // rows contiguous, real
  kCR = 2, // rows contiguous, complex: A with op N, B with op T / C
  kCK = 3  // K contiguous, complex A with op T / C
};

struct SmallParams {
  const void *a, *b; // or arrays of pointers, see flags
  void *c;
  const DynParams *dyn;
  int *status;
  uint64_t stride_a, stride_b, stride_c; // in floats
  uint32_t lda, ldb, ldc;                // in floats
  uint32_t m, n, k;                      // extents of the expanded real product
  uint32_t tiles_m, tiles_n;
  float alpha_r, alpha_i, beta_r, beta_i;
  uint32_t flags;
};
static_assert(sizeof(SmallParams) <= 128, "kernel parameter structs stay within 128 bytes");
constexpr uint32_t kConjA = 1, kConjB = 2, kPairsA = 4, kPairsB = 8, kPointers = 16, kComplex = 32;

// What one thread holds of a chunk: ROWS x KC values of the operand over all threads.
//   kR, kCR   row t mod ROWS, a run of V consecutive k values
//   kK, kCK   a lane's pair of k values in V / 2 (kCK: V / 4) rows
// Rows beyond the operand repeat its last one: what they give is not stored.  (Loads without
// predicates: with a test per load the K loop took three times as long.)
template <int KIND, int ROWS, int LAYOUT, bool IS_A> struct Operand {
  static constexpr int KC = (KIND == 0) ? 64 : 32;
  static constexpr int V = ROWS * KC / NUM_THREADS;
  static constexpr int LANES = KC / 2;          // lanes that share a row (kK, kCK)
  static constexpr int RPS = 32 / LANES;        // rows of a warp's access
  static constexpr int HELD = (LAYOUT == kCK) ? V / 2 : V;
  float v[HELD];

  // first of this thread's k values in a chunk
  __device__ __forceinline__ static uint32_t my_k() {
    if constexpr (LAYOUT == kR || LAYOUT == kCR) return (threadIdx.x / ROWS) * V;
    else return 2u * ((threadIdx.x & 31u) % LANES);
  }
  // this thread's first row in the tile (kCK: of complex elements), and how far apart its rows are
  __device__ __forceinline__ static uint32_t my_row() {
    if constexpr (LAYOUT == kR || LAYOUT == kCR) return threadIdx.x % ROWS;
    else return RPS * (threadIdx.x >> 5) + (threadIdx.x & 31u) / LANES;
  }
  static constexpr uint32_t ROW_STEP = RPS * NUM_WARPS;

  // Loads chunk values [k0, k0 + KC); what lies outside the K range is zero.
  __device__ __forceinline__ void load(const float *src, uint32_t ld, uint32_t row0, uint32_t rows,
                                       uint32_t k0, uint32_t k, bool pairs) {
    if (k0 + KC <= k) load_part<false>(src, ld, row0, rows, k0, k, pairs);
    else load_part<true>(src, ld, row0, rows, k0, k, pairs);
  }
  template <bool TAIL>
  __device__ __forceinline__ void load_part(const float *src, uint32_t ld, uint32_t row0,
                                            uint32_t rows, uint32_t k0, uint32_t k, bool pairs) {
    const uint32_t kk = k0 + my_k();
    if constexpr (LAYOUT == kR) {
      const float *s = src + static_cast<uint64_t>(kk) * ld + min(row0 + my_row(), rows - 1);
#pragma unroll
      for (int i = 0; i < V; ++i, s += ld) v[i] = (!TAIL || kk + i < k) ? __ldcg(s) : 0.f;
    } else if constexpr (LAYOUT == kCR) {
      // two floats per complex element; A: both expanded rows of an element read it
      const uint32_t r = min(row0 + my_row(), rows - 1);
      const float *s = src + static_cast<uint64_t>(kk >> 1) * ld + (IS_A ? (r & ~1u) : 2u * r);
#pragma unroll
      for (int i = 0; i < V; i += 2, s += ld) {
        float2 x = make_float2(0.f, 0.f);
        if (!TAIL || kk + i < k) x = __ldcg(reinterpret_cast<const float2 *>(s));
        v[i] = x.x;
        v[i + 1] = x.y;
      }
    } else {
      const uint32_t first = (LAYOUT == kCK ? row0 >> 1 : row0) + my_row();
      const uint32_t last = (LAYOUT == kCK ? rows >> 1 : rows) - 1;
      if (LAYOUT == kCK || pairs) {
#pragma unroll
        for (int i = 0; i < HELD / 2; ++i) {
          const float *s = src + static_cast<uint64_t>(min(first + ROW_STEP * i, last)) * ld + kk;
          float2 x = make_float2(0.f, 0.f);
          if (!TAIL || kk < k) x = __ldcg(reinterpret_cast<const float2 *>(s));
          v[2 * i] = x.x;
          v[2 * i + 1] = x.y;
        }
      } else {
#pragma unroll
        for (int i = 0; i < HELD / 2; ++i) {
          const float *s = src + static_cast<uint64_t>(min(first + ROW_STEP * i, last)) * ld + kk;
          v[2 * i] = (!TAIL || kk < k) ? __ldcg(s) : 0.f;
          v[2 * i + 1] = (!TAIL || kk + 1 < k) ? __ldcg(s + 1) : 0.f;
        }
      }
    }
  }

  __device__ __forceinline__ static void split_pair(float x, float y, uint32_t at, uint32_t lo) {
    if constexpr (KIND == 0) {
      uint32_t h, l;
      split2_mixed(x, y, h, l);
      st_shared_u32(at, h);
      st_shared_u32(at + lo, l);
    } else {
      uint32_t h[2], l[2];
      split_tf32(x, h[0], l[0]);
      split_tf32(y, h[1], l[1]);
      st_shared_v2(at, h[0], h[1]);
      st_shared_v2(at + lo, l[0], l[1]);
    }
  }

  // Splits the values and stores them to the swizzled tile at `tile` (hi) and `tile + lo` (lo).
  __device__ __forceinline__ void store(uint32_t tile, uint32_t lo, float scale, uint32_t conj_mask) {
    if constexpr (LAYOUT == kR || LAYOUT == kCR) {
      const uint32_t r = my_row();
      if constexpr (LAYOUT == kCR) {
        const bool im_row = IS_A && (r & 1u) != 0;
#pragma unroll
        for (int i = 0; i < V; i += 2) {
          const float re = v[i], im = __uint_as_float(__float_as_uint(v[i + 1]) ^ conj_mask);
          v[i] = im_row ? im : re;
          v[i + 1] = IS_A ? (im_row ? re : -im) : im;
        }
      }
      constexpr int BYTES = (KIND == 0) ? 2 : 4;            // of a value
      constexpr int WORDS = (V * BYTES >= 16) ? 4 : V * BYTES / 4; // 32-bit words of a store
      constexpr int PER = 4 * WORDS / BYTES;                // values of a store
      static_assert(WORDS == 4 || WORDS == 2, "stores of 16 or 8 bytes");
#pragma unroll
      for (int g = 0; g < V / PER; ++g) {
        uint32_t h[WORDS], l[WORDS];
#pragma unroll
        for (int q = 0; q < WORDS; ++q) {
          if constexpr (KIND == 0)
            split2_mixed(v[PER * g + 2 * q] * scale, v[PER * g + 2 * q + 1] * scale, h[q], l[q]);
          else
            split_tf32(v[PER * g + q] * scale, h[q], l[q]);
        }
        const uint32_t byte = (my_k() + PER * g) * BYTES;
        const uint32_t at = tile + swz(r, byte >> 4) + (byte & 15u);
        if constexpr (WORDS == 4) {
          st_shared_v4(at, h[0], h[1], h[2], h[3]);
          st_shared_v4(at + lo, l[0], l[1], l[2], l[3]);
        } else {
          st_shared_v2(at, h[0], h[1]);
          st_shared_v2(at + lo, l[0], l[1]);
        }
      }
    } else {
      constexpr uint32_t PAIR_BYTES = (KIND == 0) ? 4 : 8;
      const uint32_t byte = (my_k() / 2u) * PAIR_BYTES;
#pragma unroll
      for (int i = 0; i < HELD / 2; ++i) {
        const uint32_t r = my_row() + ROW_STEP * i;
        const float x = v[2 * i] * scale, y = v[2 * i + 1] * scale;
        if constexpr (LAYOUT == kK) {
          split_pair(x, y, tile + swz(r, byte >> 4) + (byte & 15u), lo);
        } else {
          const float im = __uint_as_float(__float_as_uint(y) ^ conj_mask);
          split_pair(x, -im, tile + swz(2 * r, byte >> 4) + (byte & 15u), lo);
          split_pair(im, x, tile + swz(2 * r + 1, byte >> 4) + (byte & 15u), lo);
        }
      }
    }
  }
};

template <int KIND>
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  if constexpr (KIND == 0) ptx::mma_f16_ss(d, a, b, idesc, acc);
  else ptx::mma_tf32_ss(d, a, b, idesc, acc);
}

template <int KIND, int LA, int LB>
__device__ __forceinline__ void small_body(const SmallParams &p, uint32_t tiles, uint32_t done,
                                           volatile int *abort_flag, uint32_t tmem) {
  constexpr uint32_t KC = (KIND == 0) ? 64 : 32;
  constexpr uint32_t IDESC = ptx::make_idesc(KIND == 0 ? 0 : 2, BM, BN),
                     IDESC2 = ptx::make_idesc(KIND == 0 ? 0 : 2, BM, 2 * BN);
  constexpr float LO_SCALE_INV = (KIND == 0) ? (1.f / 2048.f) : 1.f;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;

  const uint32_t per_batch = p.tiles_m * p.tiles_n;
  const uint32_t batch = blockIdx.x / per_batch;
  const uint32_t in_batch = blockIdx.x - batch * per_batch;
  const uint32_t m0 = (in_batch % p.tiles_m) * BM, n0 = (in_batch / p.tiles_m) * BN;
  const float *a, *b;
  float *c;
  if (p.flags & kPointers) {
    a = static_cast<const float *const *>(p.a)[batch];
    b = static_cast<const float *const *>(p.b)[batch];
    c = static_cast<float *const *>(p.c)[batch];
  } else {
    a = static_cast<const float *>(p.a) + batch * p.stride_a;
    b = static_cast<const float *>(p.b) + batch * p.stride_b;
    c = static_cast<float *>(p.c) + batch * p.stride_c;
  }
  float scale_a = 1.f, scale_b = 1.f, unscale = 1.f;
  if (p.dyn != nullptr) {
    scale_a = p.dyn->scale_a;
    scale_b = p.dyn->scale_b;
    unscale = p.dyn->unscale_c;
  }
  const uint32_t conj_a = (p.flags & kConjA) ? 0x80000000u : 0u;
  const uint32_t conj_b = (p.flags & kConjB) ? 0x80000000u : 0u;
  const bool pairs_a = (p.flags & kPairsA) != 0, pairs_b = (p.flags & kPairsB) != 0;
  const uint32_t chunks = (p.k + KC - 1) / KC;

  float acc[COLS], cor[COLS];
#pragma unroll
  for (int i = 0; i < COLS; ++i) acc[i] = cor[i] = 0.f;
  const uint32_t quarter = warp & 3u, col0 = (warp >> 2) * COLS;
  const uint32_t t_mine = tmem + ((quarter * 32u) << 16) + col0;
  bool ok = true;
  // adds chunk c's products, which were committed on done[c & 1]
  auto drain = [&](uint32_t c2) {
    ok = ptx::warp_agrees(ok && ptx::mbar_wait(done + 8u * (c2 & 1u), (c2 >> 1) & 1u, abort_flag,
                                               p.status, ptx::kErrWaitD0Full));
    if (!ok) return;
    ptx::tc_fence_after();
    uint32_t v[COLS], w[COLS];
    ptx::tmem_ld_32x32b_x8(t_mine + (c2 & 1u) * D_COLS, v);
    ptx::tmem_ld_32x32b_x8(t_mine + (c2 & 1u) * D_COLS + BN, w);
    ptx::tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < COLS; ++i) {
      acc[i] += __uint_as_float(v[i]);
      cor[i] += __uint_as_float(w[i]);
    }
    ptx::tc_fence_before();
  };

  Operand<KIND, BM, LA, true> xa;
  Operand<KIND, BN, LB, false> xb;
  xa.load(a, p.lda, m0, p.m, 0, p.k, pairs_a);
  xb.load(b, p.ldb, n0, p.n, 0, p.k, pairs_b);
  uint32_t ch = 0;
  for (; ch < chunks; ++ch) {
    Operand<KIND, BM, LA, true> ya = xa;
    Operand<KIND, BN, LB, false> yb = xb;
    if (ch + 1 < chunks) {
      xa.load(a, p.lda, m0, p.m, (ch + 1) * KC, p.k, pairs_a);
      xb.load(b, p.ldb, n0, p.n, (ch + 1) * KC, p.k, pairs_b);
    }
    const uint32_t stage = tiles + (ch & 1u) * STAGE_BYTES;
    ya.store(stage, A_TILE, scale_a, conj_a);
    yb.store(stage + 2 * A_TILE, B_TILE, scale_b, conj_b);
    fence_proxy_async_shared();
    if (__syncthreads_or(!ok)) break;
    if (warp == 0 && ptx::elect_one()) {
      ptx::tc_fence_after();
      const uint64_t a_hi = ptx::make_kmajor_desc<kGemmRowBytes>(stage);
      // (B_hi and B_lo lie next to each other: one product of twice the width)
      const uint64_t a_lo = a_hi + (A_TILE >> 4), b_hi = a_hi + ((2 * A_TILE) >> 4);
      const uint32_t d = tmem + (ch & 1u) * D_COLS;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) mma<KIND>(d, a_hi + 2 * ks, b_hi + 2 * ks, IDESC2, ks > 0);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) mma<KIND>(d + BN, a_lo + 2 * ks, b_hi + 2 * ks, IDESC, 1u);
      ptx::tc_commit(done + 8u * (ch & 1u));
    }
    __syncwarp();
    if (ch > 0) drain(ch - 1);
  }

  const uint32_t row = m0 + quarter * 32u + lane;
  const bool row_ok = row < p.m;
  float *cp = c + static_cast<uint64_t>(n0 + col0) * p.ldc + row;
  const bool read_c = p.beta_r != 0.f || p.beta_i != 0.f;
  float old[COLS];
  if (read_c) { // on their way while the last products finish
#pragma unroll
    for (uint32_t i = 0; i < COLS; ++i)
      old[i] = (row_ok && n0 + col0 + i < p.n) ? __ldcg(cp + static_cast<uint64_t>(i) * p.ldc) : 0.f;
  }
  if (ch != chunks) return; // a wait gave up
  drain(chunks - 1);
  if (!ok) return;
#pragma unroll
  for (int i = 0; i < COLS; ++i) acc[i] = fmaf(cor[i], LO_SCALE_INV, acc[i]);
  const float ar = p.alpha_r * unscale, ai = p.alpha_i * unscale;
  const float sgn = (lane & 1u) ? 1.f : -1.f; // odd rows hold imaginary parts
  const bool cplx = (p.flags & kComplex) != 0;
#pragma unroll
  for (uint32_t i = 0; i < COLS; ++i) {
    // (written out: which product is fused is the same as in epilogue.cuh)
    float out = __fmul_rn(ar, acc[i]);
    if (cplx)
      out = fmaf(ar, acc[i], __fmul_rn(sgn * ai, __shfl_xor_sync(0xffffffffu, acc[i], 1)));
    if (read_c) {
      out = fmaf(p.beta_r, old[i], out);
      if (cplx) out = fmaf(sgn * p.beta_i, __shfl_xor_sync(0xffffffffu, old[i], 1), out);
    }
    if (row_ok && n0 + col0 + i < p.n) *cp = out;
    cp += p.ldc;
  }
}

// KIND: 0 = FP16, 1 = TF32, 2 = decided on the device (AUTO)
template <int KIND, int LA, int LB>
__global__ void __launch_bounds__(NUM_THREADS, 1) tcec_gemm_small_kernel(const SmallParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t done[2];
  __shared__ uint32_t tmem_ptr;
  __shared__ volatile int abort_flag;
  const uint32_t tiles = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  if (threadIdx.x == 0) {
    ptx::mbar_init(ptx::smem_u32(&done[0]), 1);
    ptx::mbar_init(ptx::smem_u32(&done[1]), 1);
    abort_flag = 0;
    ptx::mbar_init_fence();
  }
  if (threadIdx.x < 32) {
    ptx::tmem_alloc(ptx::smem_u32(&tmem_ptr), TMEM_COLS);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = tmem_ptr;
  // chained behind the kernel before it: from here on global memory is read and written
  CUMPSGEMM_CHAINED_KERNEL_ENTRY();
  const uint32_t bars = ptx::smem_u32(&done[0]);
  if (KIND == 1 || (KIND == 2 && p.dyn->gemm_mode == CUMPSGEMM_TF32TCEC))
    small_body<(KIND == 2 ? 1 : KIND), LA, LB>(p, tiles, bars, &abort_flag, tmem);
  if (KIND == 0 || (KIND == 2 && p.dyn->gemm_mode != CUMPSGEMM_TF32TCEC))
    small_body<0, LA, LB>(p, tiles, bars, &abort_flag, tmem);
  ptx::tc_fence_before();
  __syncthreads();
  if (abort_flag) { // a wait gave up: let products still in flight land
    const uint64_t t0 = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (threadIdx.x < 32) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, TMEM_COLS);
  }
}

template <int KIND, int LA, int LB>
cudaError_t launch_kernel(const SmallParams &p, unsigned grid, cudaStream_t stream) {
  static std::once_flag once[64];
  static cudaError_t setup[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::call_once(once[dev], [&]() {
    setup[dev] = cudaFuncSetAttribute(tcec_gemm_small_kernel<KIND, LA, LB>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  });
  if (setup[dev] != cudaSuccess) return setup[dev];
  return launch_chained(tcec_gemm_small_kernel<KIND, LA, LB>, grid, NUM_THREADS, SMEM_BYTES, stream, p);
}

template <int LA, int LB>
cudaError_t launch_by_kind(StreamKind kind, const SmallParams &p, unsigned grid, cudaStream_t stream) {
  switch (kind) {
  case StreamKind::fp16:
    return launch_kernel<0, LA, LB>(p, grid, stream);
  case StreamKind::tf32:
    return launch_kernel<1, LA, LB>(p, grid, stream);
  default:
    return p.dyn != nullptr ? launch_kernel<2, LA, LB>(p, grid, stream) : cudaErrorInvalidValue;
  }
}

} // namespace

cudaError_t launch_tcec_gemm_small(const SmallGemmArgs &a, cudaStream_t stream) {
  SmallParams p;
  p.a = a.a;
  p.b = a.b;
  p.c = a.c;
  p.dyn = a.dyn;
  p.status = a.dev_status;
  p.stride_a = a.stride_a;
  p.stride_b = a.stride_b;
  p.stride_c = a.stride_c;
  p.lda = a.lda;
  p.ldb = a.ldb;
  p.ldc = a.ldc;
  p.m = a.m;
  p.n = a.n;
  p.k = a.k;
  p.tiles_m = (a.m + BM - 1) / BM;
  p.tiles_n = (a.n + BN - 1) / BN;
  p.alpha_r = a.alpha_r;
  p.alpha_i = a.alpha_i;
  p.beta_r = a.beta_r;
  p.beta_i = a.beta_i;
  // two values at a time where every row begins on eight bytes and K is even (a pair of a real operand
  // is then never half outside)
  const auto pairs = [&](const void *base, uint32_t ld, uint64_t stride) {
    return !a.pointers && reinterpret_cast<std::uintptr_t>(base) % 8 == 0 && ld % 2 == 0 &&
           stride % 2 == 0 && a.k % 2 == 0;
  };
  p.flags = (a.conj_a ? kConjA : 0u) | (a.conj_b ? kConjB : 0u) |
            (pairs(a.a, a.lda, a.stride_a) ? kPairsA : 0u) |
            (pairs(a.b, a.ldb, a.stride_b) ? kPairsB : 0u) | (a.pointers ? kPointers : 0u) |
            (a.is_complex ? kComplex : 0u);
  const unsigned grid = p.tiles_m * p.tiles_n * a.batch;
  if (a.is_complex) {
    if (a.a_k_contig)
      return a.b_k_contig ? launch_by_kind<kCK, kK>(a.kind, p, grid, stream)
                          : launch_by_kind<kCK, kCR>(a.kind, p, grid, stream);
    return a.b_k_contig ? launch_by_kind<kCR, kK>(a.kind, p, grid, stream)
                        : launch_by_kind<kCR, kCR>(a.kind, p, grid, stream);
  }
  if (a.a_k_contig)
    return a.b_k_contig ? launch_by_kind<kK, kK>(a.kind, p, grid, stream)
                        : launch_by_kind<kK, kR>(a.kind, p, grid, stream);
  return a.b_k_contig ? launch_by_kind<kR, kK>(a.kind, p, grid, stream)
                      : launch_by_kind<kR, kR>(a.kind, p, grid, stream);
}

} // namespace cumpsgemm_b200
