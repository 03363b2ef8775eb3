// What the recurrences' kernels share of float32: pairs in a register pair, four elements in a load, softplus.
#pragma once
#include "common.cuh"

namespace ms {

// ---- two neighbouring floats in a register pair: each half rounds as the plain instruction does
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

// ---- four consecutive elements as they lie in memory (an address that is a multiple of their size), and as float32
template <typename T> struct Four { using raw = float4; };
template <> struct Four<__nv_bfloat16> { using raw = uint2; };
__device__ __forceinline__ float4 float4_of(const float4& r) { return r; }
__device__ __forceinline__ float4 float4_of(const uint2& r) {
  return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xffff0000u));
}
template <typename T>
__device__ __forceinline__ float4 load4(const T* p) { return float4_of(*reinterpret_cast<const typename Four<T>::raw*>(p)); }
// as they lie in memory, behind the wait on the kernels before (common.cuh)
__device__ __forceinline__ float4 behind_four(const float* p) { return behind_loadf4(p); }
__device__ __forceinline__ uint2 behind_four(const __nv_bfloat16* p) {
  uint2 v;
  asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
// whether rows `ld` apart of T in fours start where four are one load
template <typename T>
__device__ __forceinline__ bool in_fours(const T* p, int ld) {
  return (reinterpret_cast<uintptr_t>(p) % (4 * sizeof(T))) == 0 && ld % 4 == 0;
}

__device__ __forceinline__ float softplusf(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }

}  // namespace ms
