// A row's norm, for every kernel that forms one: which lane holds which columns, and the arithmetic with explicit roundings, so that a row gets the
// same bits whichever kernel it passes through.  What is left to the order in the text: a lane adds up its columns from the first to the last, warp_sum
// adds up the lanes, and the sums of a row's warps are added in their order.
#pragma once
#include "rb_common.cuh"

namespace rb {

// First of the eight columns of piece c of a lane: a row belongs to WPR warps (`wr`: which of them), each lane holding CHUNKS pieces.
template <int CHUNKS, int WPR>
__device__ __forceinline__ int norm_col(int wr, int c, int lane) { return ((wr * CHUNKS + c) * 32 + lane) * 8; }

__device__ __forceinline__ float norm_mean(float sum, float inv_n) { return __fmul_rn(sum, inv_n); }
__device__ __forceinline__ float norm_square(float x, float mean, float sum) {
  const float d = __fsub_rn(x, mean);
  return __fmaf_rn(d, d, sum);
}
__device__ __forceinline__ float norm_rstd(float squares, float inv_n, float eps) { return rsqrtf(__fmaf_rn(squares, inv_n, eps)); }
__device__ __forceinline__ float norm_value(float x, float mean, float rstd, float gamma) {
  return __fmul_rn(__fmul_rn(__fsub_rn(x, mean), rstd), gamma);
}
__device__ __forceinline__ float norm_value(float x, float mean, float rstd, float gamma, float beta) {
  return __fmaf_rn(__fmul_rn(__fsub_rn(x, mean), rstd), gamma, beta);
}

}  // namespace rb
