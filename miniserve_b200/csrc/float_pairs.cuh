// Two neighbouring floats in a register pair: each half rounds as the plain instruction does.
#pragma once

namespace ms {

using f2 = unsigned long long;
__device__ __forceinline__ void f2_fma(f2& d, f2 a, f2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_pair(float x, float y) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 f2_halves(f2 x) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
  return r;
}
__device__ __forceinline__ float f2_sum(f2 x) {
  const float2 h = f2_halves(x);
  return h.x + h.y;
}

}  // namespace ms
