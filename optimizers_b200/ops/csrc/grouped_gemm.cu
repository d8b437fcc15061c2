// Grouped TN GEMM kernel for sm_100a (tcgen05 + TMEM + TMA).  See grouped_gemm.cuh for the
// contract.  Replaces, as one launch over a problem table, the per-block cuBLAS calls behind
// torch.tensordot in the reference (distributed_shampoo/preconditioner/
// shampoo_preconditioner_list.py:1499-1507 factor Gram matrices, :1563-1578 preconditioner
// application) together with the packing / EMA / norm kernels around them (:1525-1539).
#include "grouped_gemm.cuh"
#include "half_pair.cuh"
#include "ptx.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace ob200 {

namespace {

constexpr int kTileBytesA = kBM * kBK * 4;  // 16 KiB
constexpr int kTileBytesB = kBN * kBK * 4;  // 16 KiB
constexpr int kStagePitch = 33;             // floats per staged row: conflict-free transposition
constexpr uint32_t kIdesc = make_idesc(/*tf32*/ 2, kBM, kBN);
constexpr uint32_t kIdescHalf = make_idesc(/*f16*/ 0, kBM, 0);  // N is filled in per tile

template <int kMode>
struct Cfg {
  static constexpr bool kHalf = kMode == kGemmHalfPair || kMode == kGemmHalfPairSym;
  // Columns of one of two accumulator buffers (half pairs: main and cross sums of a tile of 128 columns).
  static constexpr int kAccCols = kHalf ? 2 * kBN : kBN;
  static constexpr int kTmemCols = 2 * kAccCols;
  // Half pairs: two warps per 32-row stripe, which take its 32-column chunks in turn.  With one accumulator buffer the
  // MMAs wait for the epilogue.
  static constexpr int kColumnGroups = kHalf ? 2 : 1;
  static constexpr int kEpilogueWarps = 4 * kColumnGroups;
  static constexpr int kThreads = 64 + 32 * kEpilogueWarps;
  // tf32x3: hi and lo of both operands; half pairs: one A tile and up to two B tiles (256 columns)
  static constexpr int kStageBytes =
      kMode == kGemmTf32x3 ? 2 * (kTileBytesA + kTileBytesB) : kTileBytesA + (kHalf ? 2 : 1) * kTileBytesB;
  static constexpr int kStages = kMode == kGemmTf32x3 ? 3 : kHalf ? 4 : 6;
  static constexpr int kStagingBytes = kEpilogueWarps * 32 * kStagePitch * 4;
  static constexpr int kBarrierBytes = 256;
  // 1024 B of slack so the stage buffers can be aligned for the 128-byte swizzle.
  static constexpr int kSmemBytes = 1024 + kStages * kStageBytes + kStagingBytes + kBarrierBytes;
};

// Partial sums of stripe q (32 rows) of one part: 32-column chunks, in each 8 groups of 4 columns by 32 rows.
__device__ __forceinline__ float4* stripe_of(const GemmTile& tile, int part, int q) {
  return reinterpret_cast<float4*>(tile.partial + static_cast<long long>(part) * kBM * tile.cols + q * 32 * tile.cols);
}

__device__ __forceinline__ void sum_parts(const GemmTile& tile, int q, int c, int lane, float (&v)[32]) {
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = 0.f;
#pragma unroll 1
  for (int part = 0; part < tile.parts; ++part) {
    const float4* src = stripe_of(tile, part, q) + c * 8 * 32 + lane;
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      const float4 x = __ldcg(src + g * 32);
      v[4 * g] += x.x;
      v[4 * g + 1] += x.y;
      v[4 * g + 2] += x.z;
      v[4 * g + 3] += x.w;
    }
  }
}

// Epilogue of one 32 x 32 chunk whose result is stored as half pairs: thread `lane` holds row row0 + lane and owns
// its 128-byte chunk (zero beyond N, which the next product reads as K padding).  The transposed copy of a symmetric
// result goes through the staging tile, after which a thread owns a row of the transpose.
__device__ __forceinline__ void half_pair_chunk(float (&v)[32], float* st, float* __restrict__ Cp, float* __restrict__ Dhi, int M,
                                                int N, int ldc, int ldd, int flags, int row0, int col0, int lane, float alpha,
                                                float beta, float gamma, float scale, bool mirror, bool diag_chunk, float& sq,
                                                float& tr) {
  const int row = row0 + lane;
  const bool live = row < M, write_c = !(flags & kFlagNoC);
  float* crow = write_c ? Cp + static_cast<long long>(row) * ldc + col0 : nullptr;
  const bool vec = write_c && col0 + 32 <= N && (ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(Cp) & 15) == 0;
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    float old[4] = {0.f, 0.f, 0.f, 0.f};
    if (write_c && beta != 0.f && live) {
      if (vec) {
        const float4 o = reinterpret_cast<const float4*>(crow)[g];
        old[0] = o.x; old[1] = o.y; old[2] = o.z; old[3] = o.w;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) old[k] = col0 + 4 * g + k < N ? crow[4 * g + k] : 0.f;
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int j = 4 * g + k;
      float x = alpha * v[j] + (write_c && beta != 0.f ? beta * old[k] : 0.f);
      if ((flags & kFlagAddDiag) && col0 + j == row) x += gamma;
      v[j] = live && col0 + j < N ? x : 0.f;
      if ((flags & kFlagTrace) && col0 + j == row) tr += v[j];
    }
  }
  if (mirror || diag_chunk) {
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 32; ++j) st[lane * kStagePitch + j] = v[j];
    __syncwarp();
  }
  if (diag_chunk) {  // symmetric bit for bit: entries below the diagonal are those above it
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = j >= lane ? v[j] : st[j * kStagePitch + lane];
  }
  if (flags & kFlagSumSq) {
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) s = fmaf(v[j], v[j], s);
    sq += mirror ? 2.f * s : s;
  }
  auto store_c = [&](float* dst, int count, bool v4) {
    if (v4) {
#pragma unroll
      for (int g = 0; g < 8; ++g) reinterpret_cast<float4*>(dst)[g] = make_float4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < count) dst[j] = v[j];
    }
  };
  auto store_d = [&](float* dst) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] *= scale;
    store_pair_chunk(dst, v);
  };
  if (live) {
    if (write_c) store_c(crow, N - col0, vec);
    store_d(Dhi + static_cast<long long>(row) * ldd + col0);
  }
  if (mirror) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = st[i * kStagePitch + lane];
    const int trow = col0 + lane;
    if (trow < N) {
      const bool tvec = row0 + 32 <= M && (ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(Cp) & 15) == 0;
      if (write_c) store_c(Cp + static_cast<long long>(trow) * ldc + row0, M - row0, tvec);
      store_d(Dhi + static_cast<long long>(trow) * ldd + row0);
    }
    __syncwarp();
  }
}

// kPush: instantiation whose epilogue also stores into the peers' gather buffers; kept apart so
// that the store loop of the common instantiation is not burdened with it.
template <int kMode, bool kPush>
__global__ void __launch_bounds__(Cfg<kMode>::kThreads, 1)
grouped_gemm_kernel(const GemmProblem* __restrict__ problems, const GemmTile* __restrict__ tiles, int num_tiles,
                    float alpha, float beta, float gamma, int* __restrict__ status, const PeerPush push) {
  using C = Cfg<kMode>;
  constexpr int kStages = C::kStages;
  constexpr bool kSplit = kMode == kGemmTf32x3, kHalf = C::kHalf, kSym = kMode == kGemmHalfPairSym;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stage_base = smem;
  float* staging = reinterpret_cast<float*>(smem + kStages * C::kStageBytes);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * C::kStageBytes + C::kStagingBytes);
  uint64_t* full_bar = bars;                 // [kStages]
  uint64_t* empty_bar = bars + kStages;      // [kStages]
  uint64_t* acc_full = bars + 2 * kStages;   // [2]
  uint64_t* acc_empty = acc_full + 2;        // [2]
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  float* norm_parts = reinterpret_cast<float*>(tmem_holder + 2);                 // [4][kEpilogueWarps]
  int* norm_arrived = reinterpret_cast<int*>(norm_parts + 4 * C::kEpilogueWarps);  // [4]
  static_assert((2 * kStages + 4) * 8 + 8 + 4 * (4 * C::kEpilogueWarps + 4) <= C::kBarrierBytes, "barrier region");

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], C::kEpilogueWarps);
    }
    *abort_flag = 0;
    for (int k = 0; k < 4; ++k) norm_arrived[k] = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
        const GemmTile tile = tiles[t];
        const GemmProblem* p = &problems[tile.problem];
        for (int kb = tile.kb0; kb < tile.kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag)) {
            ok = false;
            break;
          }
          uint8_t* s = stage_base + stage * C::kStageBytes;
          const bool wide = kHalf && tile.cols > kBN;
          mbar_arrive_expect_tx(&full_bar[stage], kHalf && !wide ? kTileBytesA + kTileBytesB : C::kStageBytes);
          const int ak = p->a_k0 + kb * kBK, bk = p->b_k0 + kb * kBK;
          const int ar = p->a_row0 + tile.m0, br = p->b_row0 + tile.n0;
          tma_load_2d(s, p->a_hi, &full_bar[stage], ak, ar);
          tma_load_2d(s + kTileBytesA, p->b_hi, &full_bar[stage], bk, br);
          if (wide) tma_load_2d(s + kTileBytesA + kTileBytesB, p->b_hi, &full_bar[stage], bk, br + kBN);
          if (kSplit) {
            tma_load_2d(s + kTileBytesA + kTileBytesB, p->a_lo, &full_bar[stage], ak, ar);
            tma_load_2d(s + 2 * kTileBytesA + kTileBytesB, p->b_lo, &full_bar[stage], bk, br);
          }
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int it = 0;
      for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++it) {
        const GemmTile tile = tiles[t];
        const int buf = tile.bufs == 1 ? 0 : it & 1, round = tile.bufs == 1 ? it : it >> 1;
        if (!mbar_wait(&acc_empty[buf], (round & 1) ^ 1, abort_flag)) break;
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + buf * C::kAccCols;
        const uint32_t d_cross = d_tmem + (tile.bufs == 1 ? 2 * kBN : kBN);  // half pairs
        // Columns beyond N are not multiplied (in steps of 16); the epilogue does not read them.
        const int live = kHalf ? min(tile.cols, (problems[tile.problem].N - tile.n0 + 15) & ~15) : kBN;
        const uint32_t idesc_half = kIdescHalf | (static_cast<uint32_t>(live >> 3) << 17);
        for (int kb = tile.kb0; kb < tile.kb1; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t s = smem_u32(stage_base + stage * C::kStageBytes);
          const uint64_t a_hi = make_kmajor_sw128_desc(s);
          const uint64_t b_hi = make_kmajor_sw128_desc(s + kTileBytesA);
          if constexpr (kHalf) {
            // A row is [32 fp16 hi | 32 fp16 lo]: K steps of 16 at byte offsets 0 and 32, the lo
            // halves 64 bytes further.  lo is held times 2^11, so its products have their own accumulator.
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const uint64_t hi = static_cast<uint64_t>(k * 2), lo = static_cast<uint64_t>(4 + k * 2);
              const uint32_t first = kb != tile.kb0 || k != 0;
              umma_f16(d_cross, a_hi + lo, b_hi + hi, idesc_half, first);
              umma_f16(d_tmem, a_hi + hi, b_hi + hi, idesc_half, first);
              umma_f16(d_cross, a_hi + hi, b_hi + lo, idesc_half, 1);
            }
            umma_commit(&empty_bar[stage]);
            if (++stage == kStages) {
              stage = 0;
              phase ^= 1;
            }
            continue;
          }
          const uint64_t a_lo = make_kmajor_sw128_desc(s + kTileBytesA + kTileBytesB);
          const uint64_t b_lo = make_kmajor_sw128_desc(s + 2 * kTileBytesA + kTileBytesB);
#pragma unroll
          for (int k = 0; k < kBK / 8; ++k) {
            // Advancing the start address by 32 bytes (encoded >> 4) walks the K steps inside
            // the 128-byte swizzle row.
            const uint64_t koff = static_cast<uint64_t>(k * 2);
            if (kSplit) {
              // Consecutive products share one operand descriptor (b_hi, then a_hi).
              umma_tf32(d_tmem, a_lo + koff, b_hi + koff, kIdesc, kb != tile.kb0 || k != 0);
              umma_tf32(d_tmem, a_hi + koff, b_hi + koff, kIdesc, 1);
              umma_tf32(d_tmem, a_hi + koff, b_lo + koff, kIdesc, 1);
            } else {
              umma_tf32(d_tmem, a_hi + koff, b_hi + koff, kIdesc, kb != tile.kb0 || k != 0);
            }
          }
          umma_commit(&empty_bar[stage]);  // frees the stage once these MMAs have read it
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) umma_commit(&acc_full[buf]);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3;  // TMEM lane quadrant this warp may read
    constexpr int kGroups = C::kColumnGroups;
    const int group = (warp - 2) >> 2;  // of the stripe's chunks this warp takes group, group + kGroups, ...
    float* st = staging + (warp - 2) * 32 * kStagePitch;
    int it = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it) {
      const GemmTile tile = tiles[t];
      const GemmProblem* p = &problems[tile.problem];
      const int M = p->M, N = p->N, flags = p->flags;
      float* __restrict__ Cp = p->c;
      float* __restrict__ Dhi = p->d_hi;
      float* __restrict__ Dlo = p->d_lo;
      const int ldc = p->ldc, ldd = p->ldd;
      const int row0 = tile.m0 + q * 32;
      const bool do_push = kPush && (flags & kFlagPeerPush) && push.num_peers > 0;
      const long long push_offset = p->push_offset;
      const int buf = tile.bufs == 1 ? 0 : it & 1, round = tile.bufs == 1 ? it : it >> 1;
      if (kHalf && beta != 0.f && row0 + lane < M && ((flags & kFlagPackedC) || !(flags & kFlagNoC))) {
        // The old values of C are on their way to the L2 while the products run.
        const int row = row0 + lane;
        const float* crow = (flags & kFlagPackedC) ? Cp + static_cast<long long>(row) * N - (static_cast<long long>(row) * (row + 1)) / 2
                                                   : Cp + static_cast<long long>(row) * ldc;
        for (int c = group; c < tile.cols / 32 && tile.n0 + c * 32 < N; c += kGroups) {
          const int last = min(tile.n0 + c * 32 + 31, N - 1);  // (a row segment may straddle two lines: the first and the last entry)
          const int first = (flags & kFlagPackedC) ? max(tile.n0 + c * 32, row) : tile.n0 + c * 32;
          if (first > last) continue;
          asm volatile("prefetch.global.L2 [%0];" ::"l"(crow + first));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(crow + last));
        }
      }
      // Half pairs: the accumulator will hold (s_a a)(s_b b), with a scale per row of A and of B.  The bound of a row of a
      // split output is the same for every tile of the row, so whoever is here writes it.  All of it is
      // fetched before the wait for the products.
      constexpr int kOwn = kHalf ? 2 * kBN / 32 / kGroups : 1;  // chunks of a stripe that are this warp's
      float inv_a = 1.f, scale_d = 1.f, inv_cols[kOwn];
      if constexpr (kHalf) {
        const int row = min(row0 + lane, M - 1);
        inv_a = pair_inverse_scale(p->a_bound[row / p->a_div]);
        if (kSym && (flags & kFlagSplitOut) && (flags & kFlagFixedScale)) {
          scale_d = pair_scale(p->d_bound[0]);
        } else if ((flags & kFlagSplitOut) && Dlo == nullptr) {
          float bound;
          if (p->d_left != nullptr) {
            bound = p->d_left[row] * p->d_right[0];
            if (p->d_cap != nullptr) bound = fminf(bound, p->d_cap[0]);
            bound *= fabsf(alpha);
            if (group == 0 && row0 + lane < M) p->d_bound[row] = bound;
          } else {
            bound = p->d_bound[row];
          }
          scale_d = pair_scale(bound);
        }
#pragma unroll
        for (int k = 0; k < kOwn; ++k)
          inv_cols[k] = pair_inverse_scale(p->b_bound[min(tile.n0 + (group + k * kGroups) * 32 + lane, N - 1) / p->b_div]);
      }
      if (!mbar_wait(&acc_full[buf], round & 1, abort_flag)) break;
      tc_fence_after_sync();
      const uint32_t acc_tmem = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + buf * C::kAccCols;
      // The 32 columns of chunk c; with half pairs the cross sums, held times 2^11, join the main ones here.
      auto load_chunk = [&](int c, float(&v)[32]) {
        if constexpr (kHalf) {
          float x[32];
          tmem_ld_2x32x32(acc_tmem + c * 32, acc_tmem + (tile.bufs == 1 ? 2 * kBN : kBN) + c * 32, v, x);
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = fmaf(x[j], kPairLoInv, v[j]);
        } else {
          tmem_ld_32x32(acc_tmem + c * 32, v);
        }
      };
      // The accumulator goes back to the MMAs once the warp has loaded its last chunk: with one buffer they wait for it.
      // (Loading each chunk ahead of the stores of the one before spilled 600 bytes: 2123 -> 2475 us in a step's products over
      // 8192 x 8192.)
      bool held = true;
      auto release = [&]() {
        if (!held) return;
        held = false;
        tc_fence_before_sync();
        if (lane == 0) mbar_arrive(&acc_empty[buf]);
      };
      float sq = 0.f, tr = 0.f;
      // Symmetric result (kFlagMirror): only entries on or above the diagonal are taken from the
      // accumulator; every 32 x 32 chunk strictly above the diagonal is also stored transposed and
      // the chunks on the diagonal are symmetrised, so the stored matrix is symmetric bit for bit
      // (an antisymmetric rounding residue would be amplified by the polynomial iterations that
      // consume these products).
      const bool sym = kMode != kGemmHalfPair && (flags & kFlagMirror) != 0;
      const bool diag_tile = sym && tile.n0 == tile.m0;
      const bool parted = kMode == kGemmHalfPair && tile.parts > 1;
      bool finish = row0 < M;  // this warp runs the epilogue of its stripe
      const int chunks = kHalf ? tile.cols / 32 : kBN / 32;
      if (parted && row0 < M) {
        float4* own = stripe_of(tile, tile.part, q) + lane;
        for (int c = group; c < chunks && tile.n0 + c * 32 < N; c += kGroups) {
          if ((flags & kFlagPackedC) && tile.n0 + c * 32 + 31 < row0) continue;
          float v[32];
          load_chunk(c, v);
#pragma unroll
          for (int g = 0; g < 8; ++g) own[(c * 8 + g) * 32] = make_float4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
        }
        release();
        __threadfence();
        __syncwarp();
        int arrived = 0;
        int* counter = tile.counter + q * kGroups + group;
        if (lane == 0) arrived = atomicAdd(counter, 1);
        finish = __shfl_sync(0xffffffffu, arrived, 0) == tile.parts - 1;
        if (finish) {
          if (lane == 0) *counter = 0;
          __threadfence();
        }
      }
      if (finish) {
        // Chunks this warp stores: neither beyond N, nor strictly below the diagonal of a packed result, nor written as
        // the transpose of another.
        auto next_chunk = [&](int c) {
          while (c < chunks && (((flags & kFlagPackedC) && tile.n0 + c * 32 + 31 < row0) || (diag_tile && c < q))) c += kGroups;
          return tile.n0 + c * 32 < N ? c : chunks;
        };
        int after;
        // Exponents of the scales to take out: where no product of two of them leaves the range of fp32, they are
        // multiplied first.
        int a_min = 0, a_max = 0;
        if constexpr (kHalf) {
          const int e = static_cast<int>(__float_as_uint(inv_a) >> 23) - 127;
          a_min = __reduce_min_sync(0xffffffffu, e);
          a_max = __reduce_max_sync(0xffffffffu, e);
        }
#pragma unroll 1
        for (int c = next_chunk(group); c < chunks; c = after) {
          const int col0 = tile.n0 + c * 32;
          after = next_chunk(c + kGroups);
          const bool mirror = sym && (!diag_tile || c > q);
          const bool diag_chunk = diag_tile && c == q;
          float v[32];
          if (kMode == kGemmHalfPair && parted) {
            sum_parts(tile, q, c, lane, v);
          } else {
            load_chunk(c, v);
            if (after >= chunks) release();
          }
          float sq_chunk = 0.f;
          if constexpr (kHalf) {
            float mine = inv_cols[0];
#pragma unroll
            for (int k = 1; k < kOwn; ++k) mine = c == group + k * kGroups ? inv_cols[k] : mine;
            const int e = static_cast<int>(__float_as_uint(mine) >> 23) - 127;
            const bool split_out = !kSym && (flags & kFlagSplitOut);
            if (a_min + __reduce_min_sync(0xffffffffu, e) >= -120 && a_max + __reduce_max_sync(0xffffffffu, e) <= 120) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] *= inv_a * __shfl_sync(0xffffffffu, mine, j);
            } else {  // one after the other, the smaller first
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                const float inv_b = __shfl_sync(0xffffffffu, mine, j);
                v[j] = (v[j] * fminf(inv_a, inv_b)) * fmaxf(inv_a, inv_b);
              }
            }
            if (split_out) {
              // One thread owns the 128-byte chunk of its row: 32 hi, then 32 lo (zero beyond N, which
              // the next product reads as K padding).
              if (row0 + lane < M) {
                const float factor = alpha * scale_d;
                const int cols = N - col0;
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = j < cols ? factor * v[j] : 0.f;
                store_pair_chunk(Dhi + static_cast<long long>(row0 + lane) * ldd + col0, v);
              }
              continue;
            }
            if (kSym && (flags & kFlagSplitOut) && Dlo == nullptr) {
              half_pair_chunk(v, st, Cp, Dhi, M, N, ldc, ldd, flags, row0, col0, lane, alpha, beta, gamma, scale_d, mirror,
                              diag_chunk, sq, tr);
              continue;
            }
          }
          // Fast path: the thread that holds row (row0 + lane) of the accumulator stores its 32
          // consecutive columns itself with 16-byte accesses (C, then the (hi, lo) pair), and
          // stores the transposed copy of a symmetric result one column at a time, where the 32
          // lanes are 32 consecutive addresses.  No staging through shared memory.  It needs a full
          // chunk, 16-byte alignment of every row segment and none of the per-element layouts
          // (packed triangle, peer push, the symmetrised diagonal chunk).
          const bool fast_c = (flags & kFlagNoC) || ((ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(Cp) & 15) == 0);
          const bool fast_d = !(flags & kFlagSplitOut) ||
                              ((ldd & 3) == 0 && ((reinterpret_cast<uintptr_t>(Dhi) | reinterpret_cast<uintptr_t>(Dlo)) & 15) == 0);
          if (col0 + 32 <= N && !(flags & kFlagPackedC) && !do_push && !diag_chunk && fast_c && fast_d) {
            const int row = row0 + lane;
            if (row < M) {
              const bool write_c = !(flags & kFlagNoC);
              if (flags & kFlagSquareAcc) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] *= v[j];
              }
              if (write_c && beta != 0.f) {
                const float4* src = reinterpret_cast<const float4*>(Cp + static_cast<long long>(row) * ldc + col0);
#pragma unroll
                for (int j4 = 0; j4 < 8; ++j4) {
                  const float4 o = src[j4];
                  v[4 * j4 + 0] = alpha * v[4 * j4 + 0] + beta * o.x;
                  v[4 * j4 + 1] = alpha * v[4 * j4 + 1] + beta * o.y;
                  v[4 * j4 + 2] = alpha * v[4 * j4 + 2] + beta * o.z;
                  v[4 * j4 + 3] = alpha * v[4 * j4 + 3] + beta * o.w;
                }
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] *= alpha;
              }
              if (flags & (kFlagAddDiag | kFlagTrace)) {
                const int dj = row - col0;  // position of the diagonal entry in this segment, if any
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                  if (j == dj) {
                    if (flags & kFlagAddDiag) v[j] += gamma;
                    if (flags & kFlagTrace) tr += v[j];
                  }
                }
              }
#pragma unroll
              for (int j = 0; j < 32; ++j) sq_chunk = fmaf(v[j], v[j], sq_chunk);
              if (write_c) {
                float4* dst = reinterpret_cast<float4*>(Cp + static_cast<long long>(row) * ldc + col0);
#pragma unroll
                for (int j4 = 0; j4 < 8; ++j4) dst[j4] = make_float4(v[4 * j4], v[4 * j4 + 1], v[4 * j4 + 2], v[4 * j4 + 3]);
              }
              if (flags & kFlagSplitOut) {
                float4* dh = reinterpret_cast<float4*>(Dhi + static_cast<long long>(row) * ldd + col0);
                float4* dl = reinterpret_cast<float4*>(Dlo + static_cast<long long>(row) * ldd + col0);
#pragma unroll
                for (int j4 = 0; j4 < 8; ++j4) {
                  float h[4], l[4];
#pragma unroll
                  for (int k = 0; k < 4; ++k) {
                    h[k] = tf32_round(v[4 * j4 + k]);
                    l[k] = v[4 * j4 + k] - h[k];
                  }
                  dh[j4] = make_float4(h[0], h[1], h[2], h[3]);
                  dl[j4] = make_float4(l[0], l[1], l[2], l[3]);
                }
              }
              if (mirror) {
                // (row, col0 + j) -> (col0 + j, row): for a fixed j the warp writes 32 consecutive floats
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                  const long long oc = static_cast<long long>(col0 + j) * ldc + row;
                  if (write_c) Cp[oc] = v[j];
                  if (flags & kFlagSplitOut) {
                    const long long od = static_cast<long long>(col0 + j) * ldd + row;
                    const float hi = tf32_round(v[j]);
                    Dhi[od] = hi;
                    Dlo[od] = v[j] - hi;
                  }
                }
                sq_chunk *= 2.f;
              }
            }
            sq += sq_chunk;
            continue;
          }
#pragma unroll
          for (int j = 0; j < 32; ++j) st[lane * kStagePitch + j] = v[j];
          __syncwarp();
          const int col = col0 + lane;
          if (col < N) {
            const int rows = min(32, M - row0);
            const bool packed = (flags & kFlagPackedC) != 0;
            const bool write_c = packed || !(flags & kFlagNoC);
            // All loads of the old values first, then the stores: the loads are independent
            // and overlap instead of each waiting behind the previous store.  Offsets advance
            // incrementally: one row down is +ldc, or +(N - row - 1) in the packed triangle.
            const long long off0 =
                packed ? static_cast<long long>(row0) * N - (static_cast<long long>(row0) * (row0 - 1)) / 2 + (col - row0)
                       : static_cast<long long>(row0) * ldc + col;
            float old[32];
            if (write_c && beta != 0.f) {
              long long o = off0;
#pragma unroll
              for (int rr = 0; rr < 32; ++rr) {
                const int row = row0 + rr;
                const bool live = rr < rows && (!packed || col >= row);
                old[rr] = live ? Cp[o] : 0.f;
                o += packed ? (N - row - 1) : ldc;
              }
            } else {
#pragma unroll
              for (int rr = 0; rr < 32; ++rr) old[rr] = 0.f;
            }
            long long o = off0;
#pragma unroll
            for (int rr = 0; rr < 32; ++rr) {
              const int row = row0 + rr;
              const bool live = rr < rows && (!packed || col >= row);
              if (live) {
                float acc = st[rr * kStagePitch + lane];
                if (flags & kFlagSquareAcc) acc *= acc;
                float val = alpha * acc + beta * old[rr];
                if ((flags & kFlagAddDiag) && row == col) val += gamma;
                if (sym) st[rr * kStagePitch + lane] = val;  // read back transposed below
                if (!diag_chunk) {
                  if ((flags & kFlagTrace) && row == col) tr += val;
                  if (write_c) Cp[o] = val;
                  if (flags & kFlagSplitOut) {
                    const long long od = static_cast<long long>(row) * ldd + col;
                    const float hi = tf32_round(val);
                    Dhi[od] = hi;
                    Dlo[od] = val - hi;
                  }
                  if (kPush && do_push) {
                    // A warp stores 32 consecutive elements of one row into each rank's slot.
                    const long long e = static_cast<long long>(row) * N + col;
                    for (int r = 0; r < push.num_peers; ++r) {
                      void* dst = reinterpret_cast<void*>(push.base[r] + push_offset);
                      if (push.dtype == 1) {
                        static_cast<__nv_bfloat16*>(dst)[e] = __float2bfloat16_rn(val);
                      } else if (push.dtype == 2) {
                        static_cast<__half*>(dst)[e] = __float2half_rn(val);
                      } else {
                        static_cast<float*>(dst)[e] = val;
                      }
                    }
                  }
                  sq_chunk += val * val;
                }
              }
              o += packed ? (N - row - 1) : ldc;
            }
          }
          __syncwarp();
          if (diag_chunk) {
            // Entry (row0 + rr, col0 + lane) takes the value computed for whichever of it and its
            // transpose lies on or above the diagonal.
            if (col < N) {
              const int rows = min(32, M - row0);
              const bool write_c = !(flags & kFlagNoC);
              for (int rr = 0; rr < rows; ++rr) {
                const float val = lane >= rr ? st[rr * kStagePitch + lane] : st[lane * kStagePitch + rr];
                const int row = row0 + rr;
                if ((flags & kFlagTrace) && rr == lane) tr += val;
                if (write_c) Cp[static_cast<long long>(row) * ldc + col] = val;
                if (flags & kFlagSplitOut) {
                  const long long od = static_cast<long long>(row) * ldd + col;
                  const float hi = tf32_round(val);
                  Dhi[od] = hi;
                  Dlo[od] = val - hi;
                }
                sq_chunk += val * val;
              }
            }
            __syncwarp();
          } else if (mirror) {
            // Element (row0 + lane, col0 + j) goes to (col0 + j, row0 + lane): lanes run along the
            // destination row, and the odd staging pitch keeps the column read conflict-free.
            const int rows = min(32, M - row0), cols = min(32, N - col0);
            if (lane < rows) {
              const bool write_c = !(flags & kFlagNoC);
              for (int j = 0; j < cols; ++j) {
                const float val = st[lane * kStagePitch + j];
                const int drow = col0 + j, dcol = row0 + lane;
                if (write_c) Cp[static_cast<long long>(drow) * ldc + dcol] = val;
                if (flags & kFlagSplitOut) {
                  const long long od = static_cast<long long>(drow) * ldd + dcol;
                  const float hi = tf32_round(val);
                  Dhi[od] = hi;
                  Dlo[od] = val - hi;
                }
              }
            }
            __syncwarp();
            sq_chunk *= 2.f;
          }
          sq += sq_chunk;
        }
      }
      release();
      if (flags & kFlagSumSq) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if constexpr (kMode == kGemmHalfPair) {
          // The warps' sums in a fixed order, by the warp that arrives last (none waits; a warp is at most two tiles ahead
          // of another): a problem of one tile adds up the same way in every run.
          if (lane == 0) {
            float* mine = norm_parts + (it & 3) * C::kEpilogueWarps;
            mine[warp - 2] = sq;
            __threadfence_block();
            if (atomicAdd(&norm_arrived[it & 3], 1) == C::kEpilogueWarps - 1) {
              norm_arrived[it & 3] = 0;
              __threadfence_block();
              float total = 0.f;
#pragma unroll
              for (int w = 0; w < C::kEpilogueWarps; ++w) total += static_cast<volatile float*>(mine)[w];
              if (total != 0.f) atomicAdd(p->sumsq, total);
            }
          }
        } else if (lane == 0 && sq != 0.f) {
          atomicAdd(p->sumsq, sq);
        }
      }
      if (flags & kFlagTrace) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tr += __shfl_xor_sync(0xffffffffu, tr, o);
        if (lane == 0 && tr != 0.f) atomicAdd(p->sumsq + 1, tr);
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0) atomicExch(status, kErrPipelineTimeout);
    // Give copies that are still in flight time to land before the CTA's shared memory goes away.
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) {
    }
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

template <int kMode, bool kPush>
void launch_impl(const GemmProblem* problems, const GemmTile* tiles, int num_tiles, float alpha, float beta,
                 float gamma, int* status, int max_ctas, cudaStream_t stream, const PeerPush& push) {
  using C = Cfg<kMode>;
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(grouped_gemm_kernel<kMode, kPush>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    configured = true;
  }
  const int grid = num_tiles < max_ctas ? num_tiles : max_ctas;
  grouped_gemm_kernel<kMode, kPush><<<grid, C::kThreads, C::kSmemBytes, stream>>>(problems, tiles, num_tiles, alpha,
                                                                               beta, gamma, status, push);
}

}  // namespace

void launch_grouped_gemm(const GemmProblem* problems, const GemmTile* tiles, int num_tiles, float alpha, float beta,
                         GemmMode mode, int* status, int max_ctas, cudaStream_t stream, const PeerPush* push, float gamma) {
  if (num_tiles <= 0) return;
  PeerPush none{};
  const PeerPush& pp = push != nullptr ? *push : none;
  const bool pushing = pp.num_peers > 0;
  auto go = [&](auto launch) { launch(problems, tiles, num_tiles, alpha, beta, gamma, status, max_ctas, stream, pp); };
  if (mode == kGemmHalfPair) {
    pushing ? go(launch_impl<kGemmHalfPair, true>) : go(launch_impl<kGemmHalfPair, false>);
  } else if (mode == kGemmHalfPairSym) {
    go(launch_impl<kGemmHalfPairSym, false>);
  } else if (mode == kGemmTf32x3) {
    pushing ? go(launch_impl<kGemmTf32x3, true>) : go(launch_impl<kGemmTf32x3, false>);
  } else {
    pushing ? go(launch_impl<kGemmTf32, true>) : go(launch_impl<kGemmTf32, false>);
  }
}

}  // namespace ob200
