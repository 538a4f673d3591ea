// Pieces shared by the kernels that split FP32 operands inside the GEMM kernel
// (tcec_gemm_fused.cu, tcec_gemm_stream.cu): the hi / lo arithmetic (bit for bit the one of
// split_kernels.cu) and the shared-memory side of it.
#pragma once
#include <cstdint>
#include <cuda_fp16.h>

namespace cumpsgemm_b200 {

// Byte offset of (row r, 16-byte chunk c) inside a K-major tile with 128-byte rows and the
// 128-byte swizzle: 8-row groups of 1 KiB, chunk index XORed with the row index modulo 8.
__device__ __forceinline__ uint32_t swz(uint32_t r, uint32_t c) {
  return (r >> 3) * 1024u + (r & 7u) * 128u + ((c ^ (r & 7u)) << 4);
}

// hi = RN_fp16(v), lo = RN_fp16((v - hi) * 2^11) for two values, packed (v0 in the low half).
// (Packed FP32x2 arithmetic for the difference saves two instructions per pair on paper; the
// register pairs it needs cost more: 2048 products of 128^3 82 -> 103 us.)
__device__ __forceinline__ void split2(float v0, float v1, uint32_t &hi, uint32_t &lo) {
  const __half2 h = __floats2half2_rn(v0, v1);
  const float2 hf = __half22float2(h);
  const __half2 l = __floats2half2_rn((v0 - hf.x) * 2048.f, (v1 - hf.y) * 2048.f);
  hi = *reinterpret_cast<const uint32_t *>(&h);
  lo = *reinterpret_cast<const uint32_t *>(&l);
}

// The same values with v - hi already scaled: fma(hi, -2^11, v * 2^11) is exact, and taking hi as FP16
// saves the conversion back.
__device__ __forceinline__ void split2_mixed(float v0, float v1, uint32_t &hi, uint32_t &lo) {
  unsigned long long v, w;
  float w0, w1, d0, d1;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(v0), "f"(v1));
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(w) : "l"(v), "l"(0x4500000045000000ull)); // 2^11, twice
  asm("mov.b64 {%0, %1}, %2;" : "=f"(w0), "=f"(w1) : "l"(w));
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(v1), "f"(v0));
  asm("{\n\t"
      ".reg .b16 h0, h1, c;\n\t"
      "mov.b32 {h0, h1}, %2;\n\t"
      "mov.b16 c, 0xE800;\n\t" // -2^11
      "fma.rn.f32.f16 %0, h0, c, %3;\n\t"
      "fma.rn.f32.f16 %1, h1, c, %4;\n\t"
      "}"
      : "=f"(d0), "=f"(d1)
      : "r"(hi), "f"(w0), "f"(w1));
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(d1), "f"(d0));
}

// hi = RNA_tf32(v), lo = RNA_tf32(v - hi)
__device__ __forceinline__ void split_tf32(float v, uint32_t &hi, uint32_t &lo) {
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(v));
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(v - __uint_as_float(hi)));
}

__device__ __forceinline__ void st_shared_u32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_shared_v2(uint32_t addr, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t x, uint32_t y, uint32_t z,
                                             uint32_t w) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x), "r"(y), "r"(z),
               "r"(w)
               : "memory");
}
// volatile: stays behind the barrier wait in front of it (waits and arrivals are volatile too)
__device__ __forceinline__ float ld_shared_f1(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ float2 ld_shared_f2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ float4 ld_shared_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr));
  return v;
}
// generic-proxy writes to shared memory become visible to the async proxy (the tensor core)
__device__ __forceinline__ void fence_proxy_async_shared() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

} // namespace cumpsgemm_b200
