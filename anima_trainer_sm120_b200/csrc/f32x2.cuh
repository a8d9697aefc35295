// Packed and mixed-precision fp32 arithmetic of sm_100: two fp32 lanes per instruction (add / mul / fma.f32x2), and
// bf16 operands taken without widening them first (add / sub / fma.f32.bf16). Every operation rounds once, exactly as
// its scalar fp32 counterpart on the widened values, so using them changes the instruction count and not a bit.
#pragma once

#include "common.cuh"

namespace anima {

using f2 = unsigned long long;   // {lo, hi} fp32

__device__ __forceinline__ f2 f2_make(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ f2 f2_dup(float v) { return f2_make(v, v); }
__device__ __forceinline__ float f2_lo(f2 a) {
  return __uint_as_float(static_cast<uint32_t>(a));
}
__device__ __forceinline__ float f2_hi(f2 a) {
  return __uint_as_float(static_cast<uint32_t>(a >> 32));
}
__device__ __forceinline__ float f2_sum(f2 a) { return f2_lo(a) + f2_hi(a); }
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// the two bf16 halves of a word, widened
__device__ __forceinline__ f2 f2_of_bf16(uint32_t w) {
  return f2_make(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
__device__ __forceinline__ uint32_t bf16_of_f2(f2 a) {   // round to nearest even, both halves
  const __nv_bfloat162 r = __floats2bfloat162_rn(f2_lo(a), f2_hi(a));
  return *reinterpret_cast<const uint32_t*>(&r);
}
// {w.lo - m, w.hi - m}
__device__ __forceinline__ f2 f2_bf16_minus(uint32_t w, float m) {
  float lo, hi;
  asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\t"
      "sub.f32.bf16 %0, l, %3;\n\tsub.f32.bf16 %1, h, %3;\n\t}"
      : "=f"(lo), "=f"(hi)
      : "r"(w), "f"(m));
  return f2_make(lo, hi);
}
// a += w.lo, b += w.hi
__device__ __forceinline__ void add_bf16(float& a, float& b, uint32_t w) {
  asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\t"
      "add.f32.bf16 %0, l, %0;\n\tadd.f32.bf16 %1, h, %1;\n\t}"
      : "+f"(a), "+f"(b)
      : "r"(w));
}
// {x.lo * y.lo + c.lo, x.hi * y.hi + c.hi} of bf16 pairs x, y and fp32 c
__device__ __forceinline__ f2 f2_fma_bf16(uint32_t x, uint32_t y, f2 c) {
  float lo = f2_lo(c), hi = f2_hi(c);
  asm("{\n\t.reg .b16 xl, xh, yl, yh;\n\tmov.b32 {xl, xh}, %2;\n\tmov.b32 {yl, yh}, %3;\n\t"
      "fma.rn.f32.bf16 %0, xl, yl, %0;\n\tfma.rn.f32.bf16 %1, xh, yh, %1;\n\t}"
      : "+f"(lo), "+f"(hi)
      : "r"(x), "r"(y));
  return f2_make(lo, hi);
}
__device__ __forceinline__ uint32_t bf16x2_add(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hadd2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}

}  // namespace anima
