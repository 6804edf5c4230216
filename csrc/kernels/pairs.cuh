// Packed fp32 arithmetic: two neighbouring numbers per instruction (fma / mul / add .rn.f32x2, each half rounded like the scalar one).
#pragma once
#include "rb_common.cuh"

namespace rb {

struct Pair {
  unsigned long long v;
};
__device__ __forceinline__ Pair pair_of(float lo, float hi) {
  Pair p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p.v) : "f"(lo), "f"(hi));
  return p;
}
__device__ __forceinline__ float2 floats(Pair p) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(p.v));
  return f;
}
__device__ __forceinline__ Pair pair_of(uint32_t bf16x2) {
  const float2 f = unpack_bf16x2(bf16x2);
  return pair_of(f.x, f.y);
}
__device__ __forceinline__ uint32_t packed(Pair p) {
  const float2 f = floats(p);
  return pack_bf16x2(f.x, f.y);
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
  Pair d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return d;
}
__device__ __forceinline__ Pair mul2(Pair a, Pair b) {
  Pair d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ Pair add2(Pair a, Pair b) {
  Pair d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}

}  // namespace rb
