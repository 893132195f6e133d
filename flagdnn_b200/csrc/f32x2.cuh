// Pairs of fp32 values in one 64-bit register (fma.rn.f32x2), shared by the depthwise kernels.
#pragma once
#include <stdint.h>

namespace fdnn {

// Two fp32 values (of neighbouring channels) in one 64-bit register, the operand form of fma.rn.f32x2 (two
// independent, correctly rounded fp32 FMAs per instruction).  They are kept as 64-bit integers so that the
// compiler carries each pair through branches and loops as one value instead of splitting and re-joining it.
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2_make(uint32_t lo_bits, uint32_t hi_bits) {
  F2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo_bits), "r"(hi_bits));
  return d;
}
__device__ __forceinline__ void f2_split(F2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
}  // namespace fdnn
