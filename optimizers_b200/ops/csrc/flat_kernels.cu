// See flat_kernels.cuh.
#include "flat_kernels.cuh"
#include "ptx.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace ob200 {

namespace {

// torch.lerp semantics: the formula switches at weight 0.5 to stay monotone.
__device__ __forceinline__ float lerpf(float a, float b, float w) {
  const float d = b - a;
  return w < 0.5f ? a + w * d : b - d * (1.f - w);
}

template <typename T>
__device__ __forceinline__ float load_as_float(const void* base, long long i);
template <>
__device__ __forceinline__ float load_as_float<float>(const void* base, long long i) {
  return static_cast<const float*>(base)[i];
}
template <>
__device__ __forceinline__ float load_as_float<__nv_bfloat16>(const void* base, long long i) {
  return __bfloat162float(static_cast<const __nv_bfloat16*>(base)[i]);
}
template <>
__device__ __forceinline__ float load_as_float<__half>(const void* base, long long i) {
  return __half2float(static_cast<const __half*>(base)[i]);
}
template <typename T>
__device__ __forceinline__ void store_from_float(void* base, long long i, float x);
template <>
__device__ __forceinline__ void store_from_float<float>(void* base, long long i, float x) {
  static_cast<float*>(base)[i] = x;
}
template <>
__device__ __forceinline__ void store_from_float<__nv_bfloat16>(void* base, long long i, float x) {
  static_cast<__nv_bfloat16*>(base)[i] = __float2bfloat16_rn(x);
}
template <>
__device__ __forceinline__ void store_from_float<__half>(void* base, long long i, float x) {
  static_cast<__half*>(base)[i] = __float2half_rn(x);
}

__global__ void __launch_bounds__(256) tf32_split_kernel(const float* __restrict__ src, long long src_pitch,
                                                         float* __restrict__ hi, float* __restrict__ lo,
                                                         long long dst_pitch, int rows, int cols) {
  const long long total = static_cast<long long>(rows) * cols;
  for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(e / cols), j = static_cast<int>(e % cols);
    const float x = src[i * src_pitch + j];
    const float h = tf32_round(x);
    hi[i * dst_pitch + j] = h;
    lo[i * dst_pitch + j] = x - h;
  }
}

__global__ void __launch_bounds__(256) affine_identity_split_kernel(const MatOp* __restrict__ ops,
                                                                    const int2* __restrict__ chunks, int num_chunks,
                                                                    float a, float b) {
  for (int c = blockIdx.x; c < num_chunks; c += gridDim.x) {
    const int2 ref = chunks[c];
    const MatOp op = ops[ref.x];
    const int row0 = ref.y * kMatRowsPerChunk;
    const int rows = min(kMatRowsPerChunk, op.d - row0);
    const bool vec = ((op.d | op.ld_src | op.ld_dst) & 3) == 0 &&
                     ((reinterpret_cast<uintptr_t>(op.src) | reinterpret_cast<uintptr_t>(op.dst_hi) |
                       reinterpret_cast<uintptr_t>(op.dst_lo)) & 15) == 0;
    if (vec) {
      // 16-byte accesses: a thread owns four consecutive columns of a row.
      const int d4 = op.d >> 2;
      for (int e = threadIdx.x; e < rows * d4; e += blockDim.x) {
        const int i = row0 + e / d4, j = (e % d4) * 4;
        const float4 v = *reinterpret_cast<const float4*>(op.src + static_cast<long long>(i) * op.ld_src + j);
        float x[4] = {a * v.x, a * v.y, a * v.z, a * v.w};
        if (i >= j && i < j + 4) x[i - j] += b;
        const long long o = static_cast<long long>(i) * op.ld_dst + j;
        if (op.dst_lo != nullptr) {
          float h[4], l[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            h[k] = tf32_round(x[k]);
            l[k] = x[k] - h[k];
          }
          *reinterpret_cast<float4*>(op.dst_hi + o) = make_float4(h[0], h[1], h[2], h[3]);
          *reinterpret_cast<float4*>(op.dst_lo + o) = make_float4(l[0], l[1], l[2], l[3]);
        } else {
          *reinterpret_cast<float4*>(op.dst_hi + o) = make_float4(x[0], x[1], x[2], x[3]);
        }
      }
      continue;
    }
    for (int e = threadIdx.x; e < rows * op.d; e += blockDim.x) {
      const int i = row0 + e / op.d, j = e % op.d;
      float x = a * op.src[static_cast<long long>(i) * op.ld_src + j];
      if (i == j) x += b;
      const long long o = static_cast<long long>(i) * op.ld_dst + j;
      if (op.dst_lo != nullptr) {
        const float h = tf32_round(x);
        op.dst_hi[o] = h;
        op.dst_lo[o] = x - h;
      } else {
        op.dst_hi[o] = x;
      }
    }
  }
}

__global__ void __launch_bounds__(256) identity_error_kernel(const MatOp* __restrict__ ops,
                                                             const int2* __restrict__ chunks, int num_chunks) {
  __shared__ float red[8];
  for (int c = blockIdx.x; c < num_chunks; c += gridDim.x) {
    const int2 ref = chunks[c];
    const MatOp op = ops[ref.x];
    const int row0 = ref.y * kMatRowsPerChunk;
    const int rows = min(kMatRowsPerChunk, op.d - row0);
    float worst = 0.f;
    for (int e = threadIdx.x; e < rows * op.d; e += blockDim.x) {
      const int i = row0 + e / op.d, j = e % op.d;
      const float x = op.src[static_cast<long long>(i) * op.ld_src + j] - (i == j ? 1.f : 0.f);
      const float ax = fabsf(x);
      worst = (ax > worst || ax != ax) ? ax : worst;  // NaN propagates
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float other = __shfl_xor_sync(0xffffffffu, worst, o);
      worst = (other > worst || other != other) ? other : worst;
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = worst;
    __syncthreads();
    if (threadIdx.x == 0) {
      float w = 0.f;
      for (int k = 0; k < 8; ++k) w = (red[k] > w || red[k] != red[k]) ? red[k] : w;
      // Non-negative floats (and +NaN, which has the largest bit pattern) order like their bits.
      atomicMax(reinterpret_cast<int*>(op.err), __float_as_int(w));
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) peer_copy_kernel(const CopyDesc* __restrict__ table,
                                                        const int2* __restrict__ chunks, int num_chunks) {
  for (int c = blockIdx.x; c < num_chunks; c += gridDim.x) {
    const int2 ref = chunks[c];
    const CopyDesc d = table[ref.x];
    const long long begin = static_cast<long long>(ref.y) * kCopyChunkBytes;
    const long long left = d.bytes - begin;
    const int n = static_cast<int>(left < kCopyChunkBytes ? left : kCopyChunkBytes);
    const char* src = static_cast<const char*>(d.src) + begin;
    char* dst = static_cast<char*>(d.dst) + begin;
    if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0) {
      const int nv = n / 16;
      const uint4* s4 = reinterpret_cast<const uint4*>(src);
      uint4* d4 = reinterpret_cast<uint4*>(dst);
      // Four independent 16-byte loads per thread before the first store.
      int i = threadIdx.x;
      for (; i + 3 * 256 < nv; i += 4 * 256) {
        const uint4 a = s4[i], b = s4[i + 256], e = s4[i + 512], f = s4[i + 768];
        d4[i] = a; d4[i + 256] = b; d4[i + 512] = e; d4[i + 768] = f;
      }
      for (; i < nv; i += 256) d4[i] = s4[i];
      for (int k = nv * 16 / 4 + threadIdx.x; k < n / 4; k += 256)
        reinterpret_cast<uint32_t*>(dst)[k] = reinterpret_cast<const uint32_t*>(src)[k];
    } else {
      for (int k = threadIdx.x; k < n / 4; k += 256)
        reinterpret_cast<uint32_t*>(dst)[k] = reinterpret_cast<const uint32_t*>(src)[k];
    }
  }
}

constexpr int kJacobiThreads = 512;  // 16 warps, one pair of column blocks each at n = 128
constexpr int kJacobiPitch = kJacobiMaxN + 1;  // odd: column reads and row (transposed) reads are both conflict-free
constexpr int kJacobiCols = 4;                 // columns of a block
constexpr int kJacobiLen = kJacobiMaxN / 32;   // entries of a column held by one lane

// Two fp32 values in a register pair: one instruction multiplies (and adds) both.
using F2 = unsigned long long;
__device__ __forceinline__ F2 pack2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(F2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Two blocks of four columns of A V (x) and of V (y), and the squared norms of the former, in the registers of a warp.
struct JacobiPair {
  F2 x[2 * kJacobiCols][kJacobiLen / 2];
  F2 y[2 * kJacobiCols][kJacobiLen / 2];
  float norm[2 * kJacobiCols];
  bool rotated, significant;  // per lane: some rotation this lane worked out
};

__device__ __forceinline__ void jacobi_norms(JacobiPair& w) {
  const int lane = threadIdx.x & 31;
  float v[2 * kJacobiCols];
#pragma unroll
  for (int c = 0; c < 2 * kJacobiCols; ++c) {
    const float2 t = unpack2(fma2(w.x[c][0], w.x[c][0], mul2(w.x[c][1], w.x[c][1])));
    v[c] = t.x + t.y;
  }
  // 8 sums: three halving steps (lane l ends up with column l / 4), then the remaining two
#pragma unroll
  for (int h = 4; h >= 1; h >>= 1) {
    const bool upper = (lane & (4 * h)) != 0;
#pragma unroll
    for (int k = 0; k < h; ++k) {
      const float send = upper ? v[k] : v[k + h], keep = upper ? v[k + h] : v[k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * h);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
#pragma unroll
  for (int c = 0; c < 2 * kJacobiCols; ++c) w.norm[c] = __shfl_sync(0xffffffffu, v[0], 4 * c);
}

// Rotations of the four disjoint column pairs (P0, Q0) .. (P3, Q3) at once: their inner products share the
// shuffles, and lanes 8 k .. 8 k + 7 work out the angle of pair k.
template <int P0, int Q0, int P1, int Q1, int P2, int Q2, int P3, int Q3>
__device__ __forceinline__ void jacobi_rotate(JacobiPair& w, float tol) {
  constexpr int P[4] = {P0, P1, P2, P3}, Q[4] = {Q0, Q1, Q2, Q3};
  const int lane = threadIdx.x & 31;
  float g[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 t = unpack2(fma2(w.x[P[k]][0], w.x[Q[k]][0], mul2(w.x[P[k]][1], w.x[Q[k]][1])));
    g[k] = t.x + t.y;
  }
#pragma unroll
  for (int h = 2; h >= 1; h >>= 1) {
    const bool upper = (lane & (8 * h)) != 0;
#pragma unroll
    for (int k = 0; k < h; ++k) {
      const float send = upper ? g[k] : g[k + h], keep = upper ? g[k + h] : g[k];
      g[k] = keep + __shfl_xor_sync(0xffffffffu, send, 8 * h);
    }
  }
  float gamma = g[0];
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) gamma += __shfl_xor_sync(0xffffffffu, gamma, o);
  const int mine = lane >> 3;
  const float alpha = mine == 0 ? w.norm[P0] : mine == 1 ? w.norm[P1] : mine == 2 ? w.norm[P2] : w.norm[P3];
  const float beta = mine == 0 ? w.norm[Q0] : mine == 1 ? w.norm[Q1] : mine == 2 ? w.norm[Q2] : w.norm[Q3];
  // sqrt(alpha) * sqrt(beta), not sqrt(alpha * beta): for a leaf with entries of 1e-12 the
  // product of the squared norms underflows to zero and every pair would rotate for ever.
  const float scale = sqrt_approx(alpha) * sqrt_approx(beta);
  const bool turn = fabsf(gamma) > tol * scale && fabsf(gamma) > 1e-37f;
  if (!__any_sync(0xffffffffu, turn)) return;
  float c = 1.f, s = 0.f, shift = 0.f;
  if (turn) {
    // The angle only has to be close (what it leaves is rotated away later); c^2 + s^2 = 1 holds for any t.
    const float zeta = __fdividef(beta - alpha, 2.f * gamma);
    const float t = copysignf(__fdividef(1.f, fabsf(zeta) + sqrt_approx(fmaf(zeta, zeta, 1.f))), zeta);
    c = rsqrtf(1.f + t * t);
    s = c * t;
    shift = t * gamma;
    w.rotated = true;
    if (fabsf(gamma) > 8.f * tol * scale) w.significant = true;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float ck = __shfl_sync(0xffffffffu, c, 8 * k), sk = __shfl_sync(0xffffffffu, s, 8 * k);
    const float dk = __shfl_sync(0xffffffffu, shift, 8 * k);
    // A rotation moves t gamma from one squared norm to the other; rounding may leave a small one below zero.
    w.norm[P[k]] = fmaxf(w.norm[P[k]] - dk, 0.f);
    w.norm[Q[k]] = fmaxf(w.norm[Q[k]] + dk, 0.f);
    const F2 c2 = pack2(ck, ck), s2 = pack2(sk, sk), m2 = pack2(-sk, -sk);
#pragma unroll
    for (int u = 0; u < kJacobiLen / 2; ++u) {
      const F2 xp = w.x[P[k]][u], xq = w.x[Q[k]][u];
      w.x[P[k]][u] = fma2(m2, xq, mul2(c2, xp));
      w.x[Q[k]][u] = fma2(s2, xp, mul2(c2, xq));
      const F2 yp = w.y[P[k]][u], yq = w.y[Q[k]][u];
      w.y[P[k]][u] = fma2(m2, yq, mul2(c2, yp));
      w.y[Q[k]][u] = fma2(s2, yp, mul2(c2, yq));
    }
  }
}

// One-sided Jacobi in blocks of four columns.  A sweep of single column pairs read and wrote every column of A V and V
// once per rotation: 2560 cycles of shared memory per round of 64 rotations at n = 128, plus five times
// three shuffles each, which go through the same pipe.  Here a warp keeps two blocks in registers for the 16
// rotations between them (and, in the first round of a sweep, the 12 inside them), four at a time, with the
// squared norms updated instead of summed again until the next round.  What is left per round is the chain of
// latencies of the four rotation steps and 2048 cycles of shared memory.  100 matrices of 128 x 128 to
// convergence: 5.26 -> 1.87 ms (full rank), 5.85 -> 2.38 ms (rank 32 plus a ridge); 64 x 64: 1.11 -> 0.60 ms.
__global__ void __launch_bounds__(kJacobiThreads, 1) jacobi_eigh_kernel(const JacobiDesc* __restrict__ descs,
                                                                     int max_sweeps, float tol,
                                                                     int* __restrict__ sweeps_out) {
  extern __shared__ float jsm[];
  float* a = jsm;                                // column j of A V at a + j * pitch
  float* v = jsm + kJacobiMaxN * kJacobiPitch;   // column j of V
  __shared__ int rotated;
  __shared__ int significant;  // a rotation of the current sweep was well above the tolerance
  __shared__ float lam_s[kJacobiMaxN];
  const JacobiDesc d = descs[blockIdx.x];
  const int n = d.n;
  // Even number of blocks; columns from n on are zero and never rotate.
  const int blocks = max(2, ((n + kJacobiCols - 1) / kJacobiCols + 1) & ~1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kWarps = kJacobiThreads / 32;

  // A is symmetric: row j read contiguously is column j.
  for (int j = warp; j < blocks * kJacobiCols; j += kWarps) {
    for (int i = lane; i < kJacobiMaxN; i += 32) {
      a[j * kJacobiPitch + i] = (i < n && j < n) ? d.a[static_cast<long long>(j) * d.lda + i] : 0.f;
      v[j * kJacobiPitch + i] = (i == j) ? 1.f : 0.f;
    }
  }
  __syncthreads();
  float shift = 0.f;
  if (d.shift_scale > 0.f) {
    __shared__ float fro_parts[kWarps];
    __shared__ float shift_s;
    float ss = 0.f;
    for (int e = threadIdx.x; e < n * n; e += kJacobiThreads) {
      const float x = a[(e / n) * kJacobiPitch + (e % n)];
      ss = fmaf(x, x, ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) fro_parts[warp] = ss;
    __syncthreads();
    if (threadIdx.x == 0) {
      float total = 0.f;
      for (int w = 0; w < kWarps; ++w) total += fro_parts[w];
      shift_s = d.shift_scale * sqrtf(total);
    }
    __syncthreads();
    shift = shift_s;
    for (int j = threadIdx.x; j < n; j += kJacobiThreads) a[j * kJacobiPitch + j] += shift;
    __syncthreads();
  }

  int sweep = 0;
  bool converged = false, settled = false;
  for (; sweep < max_sweeps && !converged; ++sweep) {
    if (threadIdx.x == 0) rotated = significant = 0;
    __syncthreads();
    JacobiPair w;
    w.rotated = w.significant = false;
    for (int r = 0; r < blocks - 1; ++r) {
      // Round r of the round-robin tournament: block blocks-1 stays, the others rotate.
      if (warp < blocks / 2) {
        const int p = warp == 0 ? blocks - 1 : (r + warp) % (blocks - 1);
        const int q = warp == 0 ? r : (r - warp + (blocks - 1)) % (blocks - 1);
        const int off_p = p * kJacobiCols * kJacobiPitch + lane, off_q = q * kJacobiCols * kJacobiPitch + lane;
#pragma unroll
        for (int c = 0; c < kJacobiCols; ++c)
#pragma unroll
          for (int u = 0; u < kJacobiLen / 2; ++u) {
            const int o = c * kJacobiPitch + 64 * u;
            w.x[c][u] = pack2(a[off_p + o], a[off_p + o + 32]);
            w.x[kJacobiCols + c][u] = pack2(a[off_q + o], a[off_q + o + 32]);
            w.y[c][u] = pack2(v[off_p + o], v[off_p + o + 32]);
            w.y[kJacobiCols + c][u] = pack2(v[off_q + o], v[off_q + o + 32]);
          }
        jacobi_norms(w);
        if (r == 0) {  // the pairs inside the blocks, once per sweep
          jacobi_rotate<0, 1, 2, 3, 4, 5, 6, 7>(w, tol);
          jacobi_rotate<0, 2, 1, 3, 4, 6, 5, 7>(w, tol);
          jacobi_rotate<0, 3, 1, 2, 4, 7, 5, 6>(w, tol);
        }
        jacobi_rotate<0, 4, 1, 5, 2, 6, 3, 7>(w, tol);
        jacobi_rotate<0, 5, 1, 6, 2, 7, 3, 4>(w, tol);
        jacobi_rotate<0, 6, 1, 7, 2, 4, 3, 5>(w, tol);
        jacobi_rotate<0, 7, 1, 4, 2, 5, 3, 6>(w, tol);
#pragma unroll
        for (int c = 0; c < kJacobiCols; ++c)
#pragma unroll
          for (int u = 0; u < kJacobiLen / 2; ++u) {
            const int o = c * kJacobiPitch + 64 * u;
            const float2 xp = unpack2(w.x[c][u]), xq = unpack2(w.x[kJacobiCols + c][u]);
            const float2 yp = unpack2(w.y[c][u]), yq = unpack2(w.y[kJacobiCols + c][u]);
            a[off_p + o] = xp.x;
            a[off_p + o + 32] = xp.y;
            a[off_q + o] = xq.x;
            a[off_q + o + 32] = xq.y;
            v[off_p + o] = yp.x;
            v[off_p + o + 32] = yp.y;
            v[off_q + o] = yq.x;
            v[off_q + o + 32] = yq.y;
          }
      }
      __syncthreads();
    }
    if (w.rotated) rotated = 1;
    if (w.significant) significant = 1;
    __syncthreads();
    converged = rotated == 0;
    // Inner products of fp32 columns carry rounding noise of the order of the tolerance itself: a
    // pair can hover around it for ever.  A last sweep all of whose rotations were within 8 times
    // the tolerance has nothing left to remove.
    settled = converged || significant == 0;
    __syncthreads();
  }

  // lambda_j = v_j . (A v_j); ascending order by rank (ties broken by index).
  for (int j = warp; j < n; j += kWarps) {
    float dot = 0.f;
    for (int i = lane; i < n; i += 32) dot += v[j * kJacobiPitch + i] * a[j * kJacobiPitch + i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    if (lane == 0) lam_s[j] = dot;
  }
  __syncthreads();
  // Thousands of fp32 rotations leave V orthogonal only to ~3e-5; one Newton-Schulz step
  // V <- V (3 I - V^T V) / 2 squares that error.  M = 1.5 I - 0.5 V^T V goes where A V was.
  // A warp works out four rows at a time, a lane every 32nd column: eight shared-memory reads feed sixteen
  // multiply-adds.  Entry (j, k) and entry (k, j) are the same sum in the same order.
  for (int j0 = 4 * warp; j0 < n; j0 += 4 * kWarps) {
    float acc[4][kJacobiLen] = {};
    for (int i = 0; i < n; ++i) {
      float row[4], col[kJacobiLen];
#pragma unroll
      for (int q = 0; q < 4; ++q) row[q] = v[min(j0 + q, n - 1) * kJacobiPitch + i];
#pragma unroll
      for (int u = 0; u < kJacobiLen; ++u) col[u] = v[min(lane + 32 * u, n - 1) * kJacobiPitch + i];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int u = 0; u < kJacobiLen; ++u) acc[q][u] = fmaf(row[q], col[u], acc[q][u]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int u = 0; u < kJacobiLen; ++u) {
        const int j = j0 + q, k = lane + 32 * u;
        if (j < n && k < n) a[j * kJacobiPitch + k] = (j == k ? 1.5f : 0.f) - 0.5f * acc[q][u];
      }
  }
  __syncthreads();
  for (int i0 = 4 * warp; i0 < n; i0 += 4 * kWarps) {  // rows i0 .. i0 + 3 of V (components of every eigenvector) belong to one warp
    float acc[4][kJacobiLen] = {};
    for (int k = 0; k < n; ++k) {
      float row[4], col[kJacobiLen];
#pragma unroll
      for (int q = 0; q < 4; ++q) row[q] = v[k * kJacobiPitch + min(i0 + q, n - 1)];
#pragma unroll
      for (int u = 0; u < kJacobiLen; ++u) col[u] = a[k * kJacobiPitch + min(lane + 32 * u, n - 1)];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int u = 0; u < kJacobiLen; ++u) acc[q][u] = fmaf(row[q], col[u], acc[q][u]);
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int u = 0; u < kJacobiLen; ++u) {
        const int i = i0 + q, j = lane + 32 * u;
        if (i < n && j < n) v[j * kJacobiPitch + i] = acc[q][u];
      }
  }
  __syncthreads();
  int* rank_of = reinterpret_cast<int*>(a);  // M is no longer needed
  for (int j = threadIdx.x; j < n; j += kJacobiThreads) {
    const float x = lam_s[j];
    int rank = 0;
    for (int k = 0; k < n; ++k) rank += (lam_s[k] < x) || (lam_s[k] == x && k < j);
    rank_of[j] = rank;
    d.lam[rank] = x - shift;
  }
  __syncthreads();
  // Q[i][rank(j)] = v_j[i]; lanes run over j so that the scattered destination stays within a row.
  if (d.transposed) {
    // Row rank(j) of q is eigenvector j: lanes run over its components.
    for (int j = warp; j < n; j += kWarps)
      for (int i = lane; i < n; i += 32) d.q[static_cast<long long>(rank_of[j]) * d.ldq + i] = v[j * kJacobiPitch + i];
  } else {
    for (int i = warp; i < n; i += kWarps)
      for (int j = lane; j < n; j += 32) d.q[static_cast<long long>(i) * d.ldq + rank_of[j]] = v[j * kJacobiPitch + i];
  }
  if (threadIdx.x == 0) sweeps_out[blockIdx.x] = settled ? sweep : max_sweeps + 1;
}

struct GpaScalars {
  float lr, beta1, beta2, eps, bc1, bc2, wd, avg_coeff, mu_y;
  int wd_on_y;
};

template <typename T>
__device__ __forceinline__ void gpa_chunk(const GpaTensorDesc& d, long long begin, long long end, const GpaScalars& s) {
  const float y_step = s.lr * (s.mu_y * (1.f - s.avg_coeff) - 1.f);
  const float shrink = 1.f - s.lr * s.wd;
  for (long long i = begin + threadIdx.x; i < end; i += blockDim.x) {
    const float g = load_as_float<T>(d.grad, i);
    float y = load_as_float<T>(d.param, i);
    float z = d.z[i];
    const float m = lerpf(d.m[i], g, 1.f - s.beta1);
    const float v = s.beta2 * d.v[i] + (1.f - s.beta2) * g * g;
    d.m[i] = m;
    d.v[i] = v;
    const float gn = (m / s.bc1) / (sqrtf(v / s.bc2) + s.eps);
    if (s.wd != 0.f) {
      if (s.wd_on_y) {
        y *= shrink;
      } else {
        z *= shrink;
      }
    }
    y = lerpf(y, z, s.avg_coeff);
    y += y_step * gn;
    z -= s.lr * gn;
    store_from_float<T>(d.param, i, y);
    d.z[i] = z;
  }
}

__device__ __forceinline__ void gpa_element(float g, float& y, float& z, float& m, float& v, const GpaScalars& s,
                                            float y_step, float shrink) {
  m = lerpf(m, g, 1.f - s.beta1);
  v = s.beta2 * v + (1.f - s.beta2) * g * g;
  const float gn = (m / s.bc1) / (sqrtf(v / s.bc2) + s.eps);
  if (s.wd != 0.f) {
    if (s.wd_on_y) {
      y *= shrink;
    } else {
      z *= shrink;
    }
  }
  y = lerpf(y, z, s.avg_coeff);
  y += y_step * gn;
  z -= s.lr * gn;
}

// fp32 parameters with 16-byte aligned arrays: two 16-byte groups per thread and array are loaded
// before anything is stored, twice per 4096-element chunk.
__device__ __forceinline__ void gpa_chunk_vec4(const GpaTensorDesc& d, long long begin, long long end,
                                               const GpaScalars& s) {
  const float y_step = s.lr * (s.mu_y * (1.f - s.avg_coeff) - 1.f);
  const float shrink = 1.f - s.lr * s.wd;
  const float4* g4 = reinterpret_cast<const float4*>(static_cast<const float*>(d.grad) + begin);
  float4* y4 = reinterpret_cast<float4*>(static_cast<float*>(d.param) + begin);
  float4* z4 = reinterpret_cast<float4*>(d.z + begin);
  float4* m4 = reinterpret_cast<float4*>(d.m + begin);
  float4* v4 = reinterpret_cast<float4*>(d.v + begin);
  const int nvec = static_cast<int>((end - begin) / 4);
  for (int base = 0; base < nvec; base += 512) {
    float4 g[2], y[2], z[2], m[2], v[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = base + u * 256 + threadIdx.x;
      if (i < nvec) {
        g[u] = g4[i]; y[u] = y4[i]; z[u] = z4[i]; m[u] = m4[i]; v[u] = v4[i];
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = base + u * 256 + threadIdx.x;
      if (i < nvec) {
        gpa_element(g[u].x, y[u].x, z[u].x, m[u].x, v[u].x, s, y_step, shrink);
        gpa_element(g[u].y, y[u].y, z[u].y, m[u].y, v[u].y, s, y_step, shrink);
        gpa_element(g[u].z, y[u].z, z[u].z, m[u].z, v[u].z, s, y_step, shrink);
        gpa_element(g[u].w, y[u].w, z[u].w, m[u].w, v[u].w, s, y_step, shrink);
        y4[i] = y[u]; z4[i] = z[u]; m4[i] = m[u]; v4[i] = v[u];
      }
    }
  }
  // ragged tail of the last chunk
  for (long long i = begin + 4LL * nvec + threadIdx.x; i < end; i += blockDim.x) {
    float y = static_cast<float*>(d.param)[i], z = d.z[i], m = d.m[i], v = d.v[i];
    gpa_element(static_cast<const float*>(d.grad)[i], y, z, m, v, s, y_step, shrink);
    static_cast<float*>(d.param)[i] = y; d.z[i] = z; d.m[i] = m; d.v[i] = v;
  }
}

__device__ __forceinline__ bool gpa_aligned16(const GpaTensorDesc& d) {
  return ((reinterpret_cast<uintptr_t>(d.param) | reinterpret_cast<uintptr_t>(d.grad) | reinterpret_cast<uintptr_t>(d.z) |
           reinterpret_cast<uintptr_t>(d.m) | reinterpret_cast<uintptr_t>(d.v)) & 15) == 0;
}

__global__ void __launch_bounds__(256, 3) gpa_adamw_kernel(const GpaTensorDesc* __restrict__ table,
                                                        const int2* __restrict__ chunks, int num_chunks, GpaScalars s) {
  for (int c = blockIdx.x; c < num_chunks; c += gridDim.x) {
    const int2 ref = chunks[c];
    const GpaTensorDesc d = table[ref.x];
    if (d.grad == nullptr) continue;
    const long long begin = static_cast<long long>(ref.y) * kGpaChunk;
    const long long end = begin + kGpaChunk < d.numel ? begin + kGpaChunk : d.numel;
    if (d.dtype == 0) {
      if (gpa_aligned16(d)) {
        gpa_chunk_vec4(d, begin, end, s);
      } else {
        gpa_chunk<float>(d, begin, end, s);
      }
    } else if (d.dtype == 1) {
      gpa_chunk<__nv_bfloat16>(d, begin, end, s);
    } else {
      gpa_chunk<__half>(d, begin, end, s);
    }
  }
}

template <typename T>
__device__ __forceinline__ void lerp_chunk(const GpaTensorDesc& d, long long begin, long long end, float w) {
  for (long long i = begin + threadIdx.x; i < end; i += blockDim.x) {
    store_from_float<T>(d.param, i, lerpf(load_as_float<T>(d.param, i), d.z[i], w));
  }
}

__global__ void __launch_bounds__(256) gpa_lerp_kernel(const GpaTensorDesc* __restrict__ table,
                                                       const int2* __restrict__ chunks, int num_chunks, float w) {
  for (int c = blockIdx.x; c < num_chunks; c += gridDim.x) {
    const int2 ref = chunks[c];
    const GpaTensorDesc d = table[ref.x];
    const long long begin = static_cast<long long>(ref.y) * kGpaChunk;
    const long long end = begin + kGpaChunk < d.numel ? begin + kGpaChunk : d.numel;
    if (d.dtype == 0) {
      lerp_chunk<float>(d, begin, end, w);
    } else if (d.dtype == 1) {
      lerp_chunk<__nv_bfloat16>(d, begin, end, w);
    } else {
      lerp_chunk<__half>(d, begin, end, w);
    }
  }
}

int grid_for(long long work_items) {
  const long long cap = sm_count() * 8;
  return static_cast<int>(work_items < cap ? (work_items > 0 ? work_items : 1) : cap);
}

}  // namespace

void launch_affine_identity_split(const MatOp* ops, const int2* chunks, int num_chunks, float a, float b,
                                  cudaStream_t stream) {
  if (num_chunks <= 0) return;
  affine_identity_split_kernel<<<grid_for(num_chunks), 256, 0, stream>>>(ops, chunks, num_chunks, a, b);
}

void launch_identity_error(const MatOp* ops, const int2* chunks, int num_chunks, cudaStream_t stream) {
  if (num_chunks <= 0) return;
  identity_error_kernel<<<grid_for(num_chunks), 256, 0, stream>>>(ops, chunks, num_chunks);
}

void launch_jacobi_eigh(const JacobiDesc* descs, int count, int max_sweeps, float tol, int* sweeps,
                        cudaStream_t stream) {
  if (count <= 0) return;
  constexpr int smem = 2 * kJacobiMaxN * kJacobiPitch * static_cast<int>(sizeof(float));
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(jacobi_eigh_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    configured = true;
  }
  jacobi_eigh_kernel<<<count, kJacobiThreads, smem, stream>>>(descs, max_sweeps, tol, sweeps);
}

void launch_peer_copy(const CopyDesc* table, const int2* chunks, int num_chunks, cudaStream_t stream) {
  if (num_chunks <= 0) return;
  const int cap = sm_count() * 8;
  peer_copy_kernel<<<num_chunks < cap ? num_chunks : cap, 256, 0, stream>>>(table, chunks, num_chunks);
}

void launch_tf32_split(const float* src, long long src_pitch, float* hi, float* lo, long long dst_pitch, int rows,
                       int cols, cudaStream_t stream) {
  const long long total = static_cast<long long>(rows) * cols;
  if (total == 0) return;
  tf32_split_kernel<<<grid_for((total + 255) / 256), 256, 0, stream>>>(src, src_pitch, hi, lo, dst_pitch, rows, cols);
}

void launch_gpa_adamw(const GpaTensorDesc* table, const int2* chunks, int num_chunks, float lr, float beta1,
                      float beta2, float eps, float bias_correction1, float bias_correction2, float weight_decay,
                      bool wd_on_y, float avg_coeff, float train_interp_coeff, cudaStream_t stream) {
  if (num_chunks <= 0) return;
  GpaScalars s{lr, beta1, beta2, eps, bias_correction1, bias_correction2, weight_decay, avg_coeff, train_interp_coeff,
               wd_on_y ? 1 : 0};
  gpa_adamw_kernel<<<grid_for(num_chunks), 256, 0, stream>>>(table, chunks, num_chunks, s);
}

void launch_gpa_lerp(const GpaTensorDesc* table, const int2* chunks, int num_chunks, float weight,
                     cudaStream_t stream) {
  if (num_chunks <= 0) return;
  gpa_lerp_kernel<<<grid_for(num_chunks), 256, 0, stream>>>(table, chunks, num_chunks, weight);
}

}  // namespace ob200
