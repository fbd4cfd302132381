// Two FP32 fused multiply-adds in one instruction (fma.rn.f32x2): each half is the same correctly rounded FMA as fmaf, so a
// chain of them has the bits of the scalar chain, at half the issue slots.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ds41 {

using float2x = unsigned long long;  // (low, high) halves of a register pair

__device__ __forceinline__ float2x pack_f32x2(float lo, float hi) {
  float2x v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void unpack_f32x2(float2x v, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ float2x fma_f32x2(float2x a, float2x b, float2x c) {
  float2x d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// The two BF16 values of a 32-bit word, promoted to FP32.
__device__ __forceinline__ float2x promote_bf16x2(uint32_t w) {
  return pack_f32x2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

}  // namespace ds41
