// Packed FP32 pairs (sm_100's f32x2 operations): two multiply-adds or additions per instruction, at the
// scalar operations' rate per element and half their issue slots.  Each half is rounded as the scalar operation.
#pragma once

#include <cuda_runtime.h>

namespace dcaacc {

using Pair = unsigned long long;  // two FP32, the first in the low half

__device__ inline Pair pairOf(float a, float b) {
  Pair p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(a), "f"(b));
  return p;
}
__device__ inline float2 floatsOf(Pair p) {
  float2 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ inline void fma2(Pair& c, Pair a, Pair b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ inline Pair add2(Pair a, Pair b) {
  Pair c;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(c) : "l"(a), "l"(b));
  return c;
}
__device__ inline Pair mul2(Pair a, Pair b) {
  Pair c;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(c) : "l"(a), "l"(b));
  return c;
}
__device__ inline Pair sub2(Pair a, Pair b) {  // exact: b times -1
  fma2(a, b, pairOf(-1.f, -1.f));
  return a;
}

}  // namespace dcaacc
