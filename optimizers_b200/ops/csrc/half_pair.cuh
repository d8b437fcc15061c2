// Scaled fp16 pairs: the operand format of the grouped GEMM's kGemmHalfPair modes.
//
// A row x with |x_k| <= B is stored as s x = hi + 2^-11 lo, with s the power of two that brings B into [2^14, 2^15),
// hi = fp16(s x) and lo = fp16(2^11 (s x - hi)).  The residual is at most half an ulp of hi, so lo is no larger than hi and
// has the same range: 22 significant bits down to 2^-28 B, and an absolute error of at most 2^-50 B below
// (hi then is a multiple of the fp16 subnormal step 2^-24, lo of 2^-35).  Every row has a scale of its own, so rows of any
// size keep their 22 bits; B may be a bound that no entry reaches, which costs as many bits of the 2^-28 as it is loose.
// Without the factor 2^11 the residual of an entry below 2^-17 B would be subnormal, and that of one below 2^-28 B zero.
//
// A row is a sequence of 128-byte chunks, one for 32 consecutive elements: 32 hi, then 32 lo, the last chunk padded with
// zeros.  An array of pairs thus has the size and pitch of an fp32 array of the same shape padded to 32 columns.  The bounds
// of the rows lie in an array of their own in device memory; rows may share one (GemmProblem::a_div).
#pragma once

#include <cstdint>
#include <cuda_fp16.h>

namespace ob200 {

constexpr int kPairChunk = 32;  // elements of one chunk
constexpr float kPairLo = 2048.f, kPairLoInv = 1.f / 2048.f;

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

// Largest magnitude, ignoring what is not finite (those entries make their rows NaN in any scale).
__device__ __forceinline__ float finite_abs(float x) {
  const float a = fabsf(x);
  return a <= 3.402823466e+38f ? a : 0.f;
}

// *dst = max(*dst, v) for non-negative floats, which order like their bits.  Most values do not exceed what is
// there already, and a plain load is cheaper than an atomic (a stale one only costs the atomic).
__device__ __forceinline__ void max_into(float* dst, float v) {
  if (v > __ldcg(dst)) atomicMax(reinterpret_cast<int*>(dst), __float_as_int(v));
}

__device__ __forceinline__ void split_pair(float x, float s, __half& hi, __half& lo) {
  const float v = x * s;
  hi = __float2half_rn(v);
  lo = __float2half_rn((v - __half2float(hi)) * kPairLo);
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

// A whole chunk of values times their scale by one thread (16-byte aligned).
__device__ __forceinline__ void store_pair_chunk(float* chunk, const float (&v)[32]) {
  uint4* dst = reinterpret_cast<uint4*>(chunk);
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    union { uint4 u; __half2 h[4]; } hi, lo;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float x = v[8 * g + 2 * k], y = v[8 * g + 2 * k + 1];
      hi.h[k] = __floats2half2_rn(x, y);
      const float2 f = __half22float2(hi.h[k]);
      lo.h[k] = __floats2half2_rn((x - f.x) * kPairLo, (y - f.y) * kPairLo);
    }
    dst[g] = hi.u;
    dst[4 + g] = lo.u;
  }
}

}  // namespace ob200
