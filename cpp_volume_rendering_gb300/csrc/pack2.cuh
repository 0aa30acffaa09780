// pack2.cuh — pairs of FP32 values in one 64-bit register: sm_103a's packed
// add, subtract, multiply and fused multiply-add (f32x2) round each half as
// the scalar instruction does, for one issue slot instead of two.
#pragma once

#include <cuda_runtime.h>

namespace cvr {

struct f2 {
  unsigned long long v;
};
__device__ __forceinline__ f2 mk2(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f2 dup2(float a) { return mk2(a, a); }
__device__ __forceinline__ float2 un2(f2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ f2 add_rd2(f2 a, f2 b) {
  f2 r;
  asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
// lerp of both halves: fmaf(t, b - a, a).
__device__ __forceinline__ f2 lerp2(f2 t, f2 a, f2 b) { return fma2(t, sub2(b, a), a); }

// cell_of of both halves.
__device__ __forceinline__ int2 cell_of2(f2 u, f2& t) {
  const f2 magic = dup2(12582912.0f);
  const f2 r = add_rd2(u, magic);
  t = sub2(u, sub2(r, magic));
  const float2 b = un2(r);
  return make_int2(__float_as_int(b.x) - 0x4B400000, __float_as_int(b.y) - 0x4B400000);
}

// Two positions, component by component.
struct pos2 {
  f2 x, y, z;
};
// o + d * m for two distances m along one ray.
__device__ __forceinline__ pos2 along2(float3 o, float3 d, f2 m) {
  return pos2{fma2(dup2(d.x), m, dup2(o.x)), fma2(dup2(d.y), m, dup2(o.y)), fma2(dup2(d.z), m, dup2(o.z))};
}
__device__ __forceinline__ float3 pos_lo(const pos2& p) { return make_float3(un2(p.x).x, un2(p.y).x, un2(p.z).x); }
__device__ __forceinline__ float3 pos_hi(const pos2& p) { return make_float3(un2(p.x).y, un2(p.y).y, un2(p.z).y); }

}  // namespace cvr
