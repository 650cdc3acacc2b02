// Packed FP32 arithmetic (sm_100a): add / mul / fma on two lanes at once.
//
// A packed instruction does two FP32 operations, each rounded as the scalar
// one, in one issue slot (the FP32 pipe takes two cycles for it: 125 lane
// operations a clock and SM measured, against 110 for scalar instructions).
// In scalar arithmetic the FFT kernels were bound by instruction issue (54-71%
// of cycles issued while the FP32 pipe was 30-37% busy), so halving the
// instructions of the same arithmetic is worth what fewer operations would be.
// Operands may name either half of a register pair for each lane, with a sign:
// broadcasting, swapping and negating the parts of a complex value cost no
// instruction.
#pragma once
#include <cuda_runtime.h>

namespace cuvhs {

struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ F2 f2(float2 a) { return f2(a.x, a.y); }
__device__ __forceinline__ float2 parts(F2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

}  // namespace cuvhs
