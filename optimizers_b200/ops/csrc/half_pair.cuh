// Scaled fp16 pairs: the operand format of the grouped GEMM's kGemmHalfPair mode.
//
// A matrix x with |x| <= B is stored as s x = hi + lo with s the power of two that brings B into
// [2^14, 2^15), hi = fp16(s x), lo = fp16(s x - hi): 22 significant bits down to 2^-18 B and an absolute
// error of at most 2^-40 B below (the fp16 subnormal step is 2^-24).  A row is a sequence of 128-byte chunks, one for 32
// consecutive elements: 32 hi, then 32 lo, the last chunk padded with zeros.  An array of pairs thus has the
// size and pitch of an fp32 array of the same shape padded to 32 columns.
//
// PairMeta, two floats in device memory beside each array: [0] = B, [1] = an upper bound of the
// squared 2-norm of a row, or 0 where none is known.
#pragma once

#include <cstdint>
#include <cuda_fp16.h>

namespace ob200 {

constexpr int kPairChunk = 32;  // elements of one chunk

// Exponent field of the scale for bound B: 13 at the largest B (or an overflowed one), at most 2^110.
__device__ __forceinline__ int pair_scale_field(float bound) {
  const int e = static_cast<int>((__float_as_uint(bound) >> 23) & 255u);  // 255: B overflowed
  const int f = bound == 0.f ? 127 : 127 + 14 + 127 - e;
  return f > 237 ? 237 : f;
}

__device__ __forceinline__ float pair_scale(float bound) {
  return __uint_as_float(static_cast<uint32_t>(pair_scale_field(bound)) << 23);
}

__device__ __forceinline__ float pair_inverse_scale(float bound) {
  return __uint_as_float(static_cast<uint32_t>(254 - pair_scale_field(bound)) << 23);
}

// Upper bound of the 2-norm of a row of K elements.
__device__ __forceinline__ float pair_row_bound(const float* meta, int K) {
  const float by_max = meta[0] * sqrtf(static_cast<float>(K));
  const float sq = meta[1];
  return sq > 1e-30f ? fminf(by_max, 1.0001f * sqrtf(sq)) : by_max;  // (a tiny sum of squares may have underflowed)
}

// Largest magnitude, ignoring what is not finite (those entries make their rows NaN in any scale).
__device__ __forceinline__ float finite_abs(float x) {
  const float a = fabsf(x);
  return a <= 3.402823466e+38f ? a : 0.f;
}

__device__ __forceinline__ void split_pair(float x, float s, __half& hi, __half& lo) {
  const float v = x * s;
  hi = __float2half_rn(v);
  lo = __float2half_rn(v - __half2float(hi));
}

// Four consecutive elements, the first a multiple of 4 columns into the row that starts at `row`.
__device__ __forceinline__ void store_pair4(float* row, int col, const float (&v)[4], float s) {
  union { uint2 u; __half h[4]; } hi, lo;
#pragma unroll
  for (int k = 0; k < 4; ++k) split_pair(v[k], s, hi.h[k], lo.h[k]);
  char* chunk = reinterpret_cast<char*>(row + (col & ~(kPairChunk - 1))) + 2 * (col & (kPairChunk - 1));
  *reinterpret_cast<uint2*>(chunk) = hi.u;
  *reinterpret_cast<uint2*>(chunk + 64) = lo.u;
}

// A whole chunk by one thread (16-byte aligned).
__device__ __forceinline__ void store_pair_chunk(float* chunk, const float (&v)[32], float s) {
  uint4* dst = reinterpret_cast<uint4*>(chunk);
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    union { uint4 u; __half h[8]; } hi, lo;
#pragma unroll
    for (int k = 0; k < 8; ++k) split_pair(v[8 * g + k], s, hi.h[k], lo.h[k]);
    dst[g] = hi.u;
    dst[4 + g] = lo.u;
  }
}

}  // namespace ob200
