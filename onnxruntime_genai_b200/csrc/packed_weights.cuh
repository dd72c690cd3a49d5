// Records of packed 4-bit weights and their expansion to 16-bit operands: int4 block-32 (described in gemm_w4.cu) and MXFP4 block-32
// (described in gemm_fp4.cu).  One record holds 128 weight rows x 64 k values.
#pragma once
#include <cuda_fp16.h>

#include "gemm_common.cuh"

namespace ogb {

constexpr int W4_RECORD_BYTES = GEMM_BLOCK_N * 32 + GEMM_BLOCK_N * 8;    // 5120
constexpr int FP4_RECORD_BYTES = GEMM_BLOCK_N * 32 + GEMM_BLOCK_N * 2;   // 4352

// untiled bulk copy global -> shared, completion on an mbarrier (transaction bytes)
__device__ __forceinline__ void bulk_copy_g2s(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ------------------------------------------------------------------------------- int4 block-32
__device__ __forceinline__ uint32_t deq_pair(uint32_t word, int shift, __nv_bfloat162 z2, __nv_bfloat162 hi2, __nv_bfloat162 lo2) {
  uint32_t t = ((word >> shift) & 0x000F000Fu) | 0x43004300u;  // two bf16 numbers 128 + q
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&t);
  v = __hsub2(v, z2);
  v = __hfma2(v, hi2, __hmul2(v, lo2));                          // round((q - zp) * (hi + lo)) in one rounding
  return *reinterpret_cast<uint32_t*>(&v);
}
// (scale, zero point) field of a block -> its zero point and the two parts of its scale, in both halves of a register
struct W4Scale { __nv_bfloat162 z2, hi2, lo2; };
__device__ __forceinline__ W4Scale w4_scale(uint32_t packed) {
  const __nv_bfloat16 hi = __ushort_as_bfloat16(uint16_t(packed & 0xFFFF)), lo = __ushort_as_bfloat16(uint16_t((packed >> 16) & 0xFFF0));
  const __nv_bfloat16 zp = __ushort_as_bfloat16(uint16_t(0x4300u | ((packed >> 16) & 0xF)));
  return {__halves2bfloat162(zp, zp), __halves2bfloat162(hi, hi), __halves2bfloat162(lo, lo)};
}
// eight codes of a record word -> four bf16x2 registers (consecutive k)
__device__ __forceinline__ uint4 deq_w4_word(uint32_t word, const W4Scale& s) {
  return make_uint4(deq_pair(word, 0, s.z2, s.hi2, s.lo2), deq_pair(word, 4, s.z2, s.hi2, s.lo2), deq_pair(word, 8, s.z2, s.hi2, s.lo2),
                    deq_pair(word, 12, s.z2, s.hi2, s.lo2));
}

// ------------------------------------------------------------------------------- MXFP4
// two e2m1 codes (low nibbles of the two halves of `u`) times the block's power-of-two multiplier
__device__ __forceinline__ uint32_t deq_fp4_pair(uint32_t u, __nv_bfloat162 s2) {
  uint32_t t = ((u & 0x00070007u) << 6) | ((u & 0x00080008u) << 12);
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&t);
  v = __hmul2(v, s2);
  return *reinterpret_cast<uint32_t*>(&v);
}
// eight codes of a record word -> four bf16x2 registers (consecutive k); m8: the block's multiplier byte (a bf16 exponent field)
__device__ __forceinline__ uint4 deq_fp4_word_bf16(uint32_t word, uint32_t m8) {
  const uint32_t sb = (m8 << 7) | (m8 << 23);
  const __nv_bfloat162 s2 = *reinterpret_cast<const __nv_bfloat162*>(&sb);
  return make_uint4(deq_fp4_pair(word, s2), deq_fp4_pair(word >> 4, s2), deq_fp4_pair(word >> 8, s2), deq_fp4_pair(word >> 12, s2));
}

// fp16 form.  A record word holds eight consecutive k values: byte i = (element i in the low nibble, element 4 + i in the
// high nibble).  `cvt.rn.f16x2.e2m1x2` turns a byte into the fp16 pair (element i, element 4 + i); two byte permutes put
// consecutive elements side by side for the K-major tile; one `mul.f16x2` applies the block's power of two.
// the four bytes of a record word -> four fp16x2 registers: byte i = (k value i, k value 4 + i)
__device__ __forceinline__ void cvt_e2m1x8_f16(uint32_t word, uint32_t (&h)[4]) {
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
      "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
      "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
      : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3]) : "r"(word));
}
__device__ __forceinline__ uint32_t hmul2_bits(uint32_t a, uint32_t b) {
  __half2 v = __hmul2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
  return *reinterpret_cast<uint32_t*>(&v);
}
// eight codes of a record word -> four fp16x2 registers (consecutive k) times the block's multiplier
__device__ __forceinline__ uint4 deq_fp4_word_f16(uint32_t word, uint32_t s) {
  uint32_t h[4];
  cvt_e2m1x8_f16(word, h);       // (k0 k4) (k1 k5) (k2 k6) (k3 k7)
  return make_uint4(hmul2_bits(__byte_perm(h[0], h[1], 0x5410), s), hmul2_bits(__byte_perm(h[2], h[3], 0x5410), s),
                    hmul2_bits(__byte_perm(h[0], h[1], 0x7632), s), hmul2_bits(__byte_perm(h[2], h[3], 0x7632), s));
}

}  // namespace ogb
