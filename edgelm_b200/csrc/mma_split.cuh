// Products of a float32 operand with a bfloat16 one on the tensor cores: the float32 operand goes as the sum of three bfloat16
// terms (8 + 8 + 8 of its 24 mantissa bits), each of which multiplies exactly, sums in float32.
#pragma once
#include "common.cuh"

namespace edgelm {

__device__ __forceinline__ uint32_t sp_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void sp_mma(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void sp_ldmatrix_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void sp_ldmatrix_x2(uint32_t addr, uint32_t& r0, uint32_t& r1) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr));
}
__device__ __forceinline__ void sp_ldmatrix_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void sp_cp16(uint32_t dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}

// Two float32 values as three packed pairs of bfloat16 terms: x = t1 + t2 + t3 up to float32 rounding (each term the
// rounding of what the terms before left over; the remainders are exact in float32).  Both values of a pair in one conversion and one
// packed multiply-add a term: 9 instructions a pair (17 with a conversion a value; the attention below was bound by these).
__device__ __forceinline__ uint32_t sp_next_term(unsigned long long& xy) {
  uint32_t t;
  asm("{\n\t.reg .b32 x, y, hx, hy;\n\t.reg .b64 h;\n\t"
      "mov.b64 {x, y}, %1;\n\t"
      "cvt.rn.bf16x2.f32 %0, y, x;\n\t"
      "shl.b32 hx, %0, 16;\n\t"
      "and.b32 hy, %0, 0xffff0000;\n\t"
      "mov.b64 h, {hx, hy};\n\t"
      "fma.rn.f32x2 %1, h, %2, %1;\n\t}"
      : "=&r"(t), "+l"(xy)
      : "l"(0xbf800000bf800000ull));
  return t;
}
__device__ __forceinline__ void sp_split(float x, float y, uint32_t& t1, uint32_t& t2, uint32_t& t3) {
  unsigned long long xy = (unsigned long long)__float_as_uint(y) << 32 | __float_as_uint(x);
  t1 = sp_next_term(xy);
  t2 = sp_next_term(xy);
  const __nv_bfloat162 last = __floats2bfloat162_rn(__uint_as_float((uint32_t)xy), __uint_as_float((uint32_t)(xy >> 32)));
  t3 = *reinterpret_cast<const uint32_t*>(&last);
}
// 2^x on the special-function unit (results under 2^-126 count as zero)
__device__ __forceinline__ float sp_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

}  // namespace edgelm
