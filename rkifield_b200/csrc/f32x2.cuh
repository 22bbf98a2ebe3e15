// f32x2.cuh — packed pairs of FP32 values for sm_100a's two-wide FP32
// instructions (PTX add/sub/mul/fma .rn.f32x2, PTX ISA 8.6).  Each lane of a
// pair is rounded exactly as the scalar instruction rounds it (IEEE
// round-to-nearest-even, no flush of subnormals), so a packed chain gives the
// same bits as the scalar chain it replaces, in half the instructions --
// except that the assembler may join f2_mul and an f2_add or f2_sub of its result into
// one fma (seen with CUDA 12.9, .rn notwithstanding): take such a product by scalars.
#pragma once

#include <cstdint>

namespace rkf {

using f2 = unsigned long long;  // (lo, hi) = (first, second) float

__device__ __forceinline__ f2 f2_pack(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(f2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
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

}  // namespace rkf
