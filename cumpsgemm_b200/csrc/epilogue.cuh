// The alpha / beta epilogue shared by the TCEC GEMM kernels.
//
// A drain warp ends a tile with CPT running sums per thread in registers (thread = row of C,
// register = column).  Registers cannot be indexed by a loop variable, so an epilogue that works
// on them directly is CPT copies of the column code: tens of kilobytes of instructions that
// are executed once per tile and come from L2 each time.  Measured that way (128 columns, B200):
// 42,000 cycles per tile with beta != 0, 10,000 with beta = 0, i.e. 20 and 5 us at the end of every
// launch, against 30 us for all of the products of m = n = k = 2048.  So the sums go back to
// TMEM, into accumulator columns the warp has just drained (eight instructions), and a rolled loop
// fetches them 16 columns at a time.  With beta != 0 the loop loads the next group's C values
// before it stores the current one.  GEMM kernels before / after, us: 2048^3 beta = 0.5 (128 x 256
// tiles) 53.3 / 45.6; 1999 x 3001 x 2777 beta = 0.5 (pairs) 118 / 94; complex 1280 x 960 x 1500
// 71.7 / 64.9; TF32TCEC 4096 x 1024 x 2048 beta = 0 89.7 / 76.5.  (Where many short tiles per launch keep
// the unrolled stores in the instruction cache, they stay: see the direct stores of tcec_gemm_stream.cu;
// and the on-the-fly kernel, tcec_gemm_fused.cu, which the round trip through TMEM cost 82 -> 93 us on
// 2048 products of 128^3.)
#pragma once
#include "ptx.cuh"

namespace cumpsgemm_b200 {

constexpr int kEpiGroup = 16; // columns per iteration of the epilogue loops

// A copy of x the compiler cannot trace back.  The loop that drains the main accumulator holds CPT
// running sums; whatever the epilogue derives from the tile index (row pointers, bounds) is
// recomputed from such a copy behind the loop, or it would be computed in front of it and push
// sums out to local memory (4096^3 TF32TCEC took 705 instead of 585 us that way).
__device__ __forceinline__ uint32_t opaque(uint32_t x) {
  uint32_t y;
  asm volatile("mov.u32 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}

// acc += TMEM columns [taddr, taddr + CPT) of this warp's lanes
template <int CPT> __device__ __forceinline__ void drain_sums(uint32_t taddr, float (&acc)[CPT]) {
#pragma unroll
  for (int c = 0; c < CPT; c += 16) {
    uint32_t v[16];
    ptx::tmem_ld_32x32b_x16(taddr + c, v);
    ptx::tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      acc[c + i] += __uint_as_float(v[i]);
      asm volatile("" : "+f"(acc[c + i])); // added here and now, not where the sum is next used
    }
  }
}

// The same on pairs of sums, one packed instruction per two columns.
__device__ __forceinline__ void add_pair(unsigned long long &acc, uint32_t x, uint32_t y) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(x), "r"(y));
  asm volatile("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(v));
}
template <int CPT>
__device__ __forceinline__ void drain_pairs(uint32_t taddr, unsigned long long (&acc)[CPT / 2]) {
#pragma unroll
  for (int c = 0; c < CPT; c += 16) {
    uint32_t v[16];
    ptx::tmem_ld_32x32b_x16(taddr + c, v);
    ptx::tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 8; ++i) add_pair(acc[c / 2 + i], v[2 * i], v[2 * i + 1]);
  }
}
// acc += s * TMEM columns, which lie in runs of RUN, a run every STEP columns
template <int CPT, int RUN, int STEP>
__device__ __forceinline__ void add_corrections_to_pairs(uint32_t taddr,
                                                         unsigned long long (&acc)[CPT / 2], float s) {
  unsigned long long s2;
  asm("mov.b64 %0, {%1, %1};" : "=l"(s2) : "f"(s));
#pragma unroll
  for (int c = 0; c < CPT; c += 16) {
    uint32_t v[16];
    ptx::tmem_ld_32x32b_x16(taddr + c / RUN * STEP + c % RUN, v);
    ptx::tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      unsigned long long x;
      asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "r"(v[2 * i]), "r"(v[2 * i + 1]));
      asm volatile("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[c / 2 + i]) : "l"(x), "l"(s2));
    }
  }
}
// acc + TMEM columns + s * corrections, left in the columns (the corrections as above)
template <int CPT, int RUN, int STEP>
__device__ __forceinline__ void finish_pairs_in_tmem(uint32_t taddr, uint32_t t_cor,
                                                     unsigned long long (&acc)[CPT / 2], float s) {
  unsigned long long s2;
  asm("mov.b64 %0, {%1, %1};" : "=l"(s2) : "f"(s));
#pragma unroll
  for (int c = 0; c < CPT; c += 16) {
    uint32_t v[16];
    ptx::tmem_ld_32x32b_x16(taddr + c, v);
    ptx::tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 8; ++i) add_pair(acc[c / 2 + i], v[2 * i], v[2 * i + 1]);
    ptx::tmem_ld_32x32b_x16(t_cor + c / RUN * STEP + c % RUN, v);
    ptx::tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      unsigned long long x;
      asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "r"(v[2 * i]), "r"(v[2 * i + 1]));
      asm volatile("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[c / 2 + i]) : "l"(x), "l"(s2));
      asm("mov.b64 {%0, %1}, %2;" : "=r"(v[2 * i]), "=r"(v[2 * i + 1]) : "l"(acc[c / 2 + i]));
    }
    ptx::tmem_st_32x32b_x16(taddr + c, v);
  }
  ptx::tmem_st_wait();
}

// acc -> TMEM columns [taddr, taddr + CPT) of this warp's lanes
template <int CPT> __device__ __forceinline__ void sums_to_tmem(uint32_t taddr, const float (&acc)[CPT]) {
#pragma unroll
  for (int c = 0; c < CPT; c += 16) {
    uint32_t v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(acc[c + i]);
    ptx::tmem_st_32x32b_x16(taddr + c, v);
  }
  ptx::tmem_st_wait();
}

// acc + corrections * scale, the corrections taken from TMEM columns [taddr, taddr + CPT) and the
// sums left in their place (in the registers the corrections came in: no copies, no spills)
template <int CPT>
__device__ __forceinline__ void add_corrections_in_tmem(uint32_t taddr, const float (&acc)[CPT],
                                                        float scale) {
#pragma unroll
  for (int c = 0; c < CPT; c += 16) {
    uint32_t v[16];
    ptx::tmem_ld_32x32b_x16(taddr + c, v);
    ptx::tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 16; ++i)
      v[i] = __float_as_uint(fmaf(__uint_as_float(v[i]), scale, acc[c + i]));
    ptx::tmem_st_32x32b_x16(taddr + c, v);
  }
  ptx::tmem_st_wait();
}

// C(row, col) = alpha * acc for columns [col0, col0 + CPT), straight from the registers.  A complex
// alpha is multiplied out whatever its imaginary part, as in store_loop: an infinite sum gives the
// same NaN in the other component on every path.
template <int CPT>
__device__ __forceinline__ void store_registers(const float (&acc)[CPT], float *cbase, uint64_t ldc,
                                                uint32_t col0, uint32_t n, bool row_ok, float ar,
                                                float ai, bool is_complex) {
  if (col0 >= n) return; // uniform over the warp
  const uint32_t cols = n - col0;
  float *cp = cbase + static_cast<uint64_t>(col0) * ldc;
  if (!is_complex) {
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
      if (row_ok && static_cast<uint32_t>(i) < cols) __stcs(cp, ar * acc[i]);
      cp += ldc;
    }
  } else {
    const float sai = (threadIdx.x & 1) ? ai : -ai; // odd rows hold imaginary parts
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
      const float out = ar * acc[i] + sai * __shfl_xor_sync(0xffffffffu, acc[i], 1);
      if (row_ok && static_cast<uint32_t>(i) < cols) __stcs(cp, out);
      cp += ldc;
    }
  }
}

template <int CPT, bool READ_C, bool COMPLEX>
__device__ __forceinline__ void store_loop(uint32_t taddr, float *cp, uint64_t ldc, uint32_t cols,
                                           bool row_ok, float ar, float ai, float br, float bi) {
  constexpr uint32_t G = kEpiGroup;
  const float sgn = (threadIdx.x & 1) ? 1.f : -1.f; // odd rows hold imaginary parts
  const float sai = sgn * ai, sbi = sgn * bi;
  float old[G];
  if constexpr (READ_C) {
    const float *lp = cp;
#pragma unroll
    for (uint32_t j = 0; j < G; ++j, lp += ldc) old[j] = (row_ok && j < cols) ? __ldcs(lp) : 0.f;
  }
  uint32_t v[G];
  ptx::tmem_ld_32x32b_x16(taddr, v);
  ptx::tmem_ld_wait();
#pragma unroll 1
  for (uint32_t c = 0; c < cols; c += G) {
    // the next group (the last iteration fetches its own again) is on its way during the stores
    uint32_t nv[G];
    ptx::tmem_ld_32x32b_x16(taddr + min(c + G, static_cast<uint32_t>(CPT) - G), nv);
    float next[G];
    if constexpr (READ_C) {
      const float *lp = cp + static_cast<uint64_t>(G) * ldc;
#pragma unroll
      for (uint32_t j = 0; j < G; ++j, lp += ldc)
        next[j] = (row_ok && c + G + j < cols) ? __ldcs(lp) : 0.f;
    }
#pragma unroll
    for (uint32_t j = 0; j < G; ++j) {
      const float x = __uint_as_float(v[j]);
      float out = ar * x;
      if constexpr (COMPLEX) out += sai * __shfl_xor_sync(0xffffffffu, x, 1);
      if constexpr (READ_C) {
        out = fmaf(br, old[j], out);
        if constexpr (COMPLEX) out += sbi * __shfl_xor_sync(0xffffffffu, old[j], 1);
        old[j] = next[j];
      }
      if (row_ok && c + j < cols) *cp = out;
      cp += ldc;
    }
    ptx::tmem_ld_wait();
#pragma unroll
    for (uint32_t j = 0; j < G; ++j) v[j] = nv[j];
  }
}

// C(row, col) = alpha * sum + beta * C(row, col) for columns [col0, col0 + CPT) of one row per lane.
// cbase points at column 0 of the row; lanes hold consecutive rows of the column-major C, so
// each warp access covers 128 contiguous bytes.  beta == 0 never reads C.
template <int CPT>
__device__ __forceinline__ void store_tile(uint32_t taddr, float *cbase, uint64_t ldc, uint32_t col0,
                                           uint32_t n, bool row_ok, float ar, float ai, float br,
                                           float bi, bool is_complex) {
  static_assert(CPT % kEpiGroup == 0, "whole groups");
  if (col0 >= n) return; // uniform over the warp
  const uint32_t cols = min(n - col0, static_cast<uint32_t>(CPT));
  float *cp = cbase + static_cast<uint64_t>(col0) * ldc;
  if (br != 0.f || bi != 0.f) {
    if (is_complex) store_loop<CPT, true, true>(taddr, cp, ldc, cols, row_ok, ar, ai, br, bi);
    else store_loop<CPT, true, false>(taddr, cp, ldc, cols, row_ok, ar, ai, br, bi);
  } else {
    if (is_complex) store_loop<CPT, false, true>(taddr, cp, ldc, cols, row_ok, ar, ai, br, bi);
    else store_loop<CPT, false, false>(taddr, cp, ldc, cols, row_ok, ar, ai, br, bi);
  }
}

} // namespace cumpsgemm_b200
