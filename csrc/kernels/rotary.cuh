// Rotation of 8 neighbouring pairs (i, i + half) of a head, for every kernel that rotates: written with explicit roundings, so that a token gets the
// same bits whichever kernel it passes through.
#pragma once
#include "rb_common.cuh"

namespace rb {

// cs(j): cosine and sine of pair j of the eight
template <class Turn>
__device__ __forceinline__ void rope_unit(uint4& lo, uint4& hi, Turn cs) {
  uint32_t* pl = reinterpret_cast<uint32_t*>(&lo);
  uint32_t* ph = reinterpret_cast<uint32_t*>(&hi);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 a = unpack_bf16x2(pl[j]), b = unpack_bf16x2(ph[j]), f = cs(2 * j), g = cs(2 * j + 1);
    pl[j] = pack_bf16x2(__fmaf_rn(a.x, f.x, -__fmul_rn(b.x, f.y)), __fmaf_rn(a.y, g.x, -__fmul_rn(b.y, g.y)));
    ph[j] = pack_bf16x2(__fmaf_rn(b.x, f.x, __fmul_rn(a.x, f.y)), __fmaf_rn(b.y, g.x, __fmul_rn(a.y, g.y)));
  }
}

}  // namespace rb
