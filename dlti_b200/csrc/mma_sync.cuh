// Warp-level bf16 fragments (ldmatrix, mma.m16n8k16 with fp32 accumulators) and 16-byte cp.async, for the kernels whose
// operands do not come in tcgen05-sized tiles: paged attention over arbitrary head sizes and the chunked recurrences.
#pragma once
#include "common.cuh"

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// log2(e) cap tanh(s scale / cap) as cap (1 - 2 / (1 + e^(2 x))): absolute error about 3e-7 cap
__device__ __forceinline__ float capped_log2(float s, float scale, float cap) {
  const float c = cap * 1.4426950408889634f;
  return c - 2.f * c * __fdividef(1.f, 1.f + ex2(s * (2.f * 1.4426950408889634f * scale / cap)));
}
// two fp32 values as a bf16 pair and the bf16 pair of what the rounding left
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  const float2 f = __bfloat1622float2(h);
  const __nv_bfloat162 l = __floats2bfloat162_rn(a - f.x, b - f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
// the same for both 16-bit types
template <typename T>
__device__ __forceinline__ void mma_16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) { mma_bf16(c, a, b0, b1); }
template <>
__device__ __forceinline__ void mma_16<__half>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// two fp32 values as three 16-bit pairs: 24 bits and more, so nothing is left
template <typename T>
__device__ __forceinline__ void split3_pair_16(float a, float b, uint32_t (&t)[3]);
template <>
__device__ __forceinline__ void split3_pair_16<__nv_bfloat16>(float a, float b, uint32_t (&t)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    const float2 f = __bfloat1622float2(h);
    a -= f.x;
    b -= f.y;
    t[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
}
template <>
__device__ __forceinline__ void split3_pair_16<__half>(float a, float b, uint32_t (&t)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    a -= f.x;
    b -= f.y;
    t[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
}
// infinities as the largest finite values: the lower terms of a split are zero or of either sign
template <typename T>
__device__ __forceinline__ uint32_t finite_pair_16(uint32_t v);
template <>
__device__ __forceinline__ uint32_t finite_pair_16<__nv_bfloat16>(uint32_t v) {
  const uint32_t top = 0x7f7f7f7fu, low = 0xff7fff7fu;
  const __nv_bfloat162 x = __hmax2(__hmin2(*reinterpret_cast<const __nv_bfloat162*>(&v), *reinterpret_cast<const __nv_bfloat162*>(&top)),
                                   *reinterpret_cast<const __nv_bfloat162*>(&low));
  return *reinterpret_cast<const uint32_t*>(&x);
}
template <>
__device__ __forceinline__ uint32_t finite_pair_16<__half>(uint32_t v) {
  const uint32_t top = 0x7bff7bffu, low = 0xfbfffbffu;
  const __half2 x = __hmax2(__hmin2(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&top)),
                            *reinterpret_cast<const __half2*>(&low));
  return *reinterpret_cast<const uint32_t*>(&x);
}
