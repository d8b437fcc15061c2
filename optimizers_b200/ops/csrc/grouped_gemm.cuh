// Grouped "TN" GEMM on the 5th-generation tensor cores:  C_g = beta * C_g + alpha * A_g * B_g^T
// for a table of independent problems, where A_g is [M,K] and B_g is [N,K], both K-major.
//
// Operand formats (GemmMode).  kGemmTf32x3: each operand arrives as a (hi, lo) pair of fp32 arrays
// with hi = tf32_round(x), lo = x - hi, and every K step issues three tf32 products
// (hi*hi + hi*lo + lo*hi) into the same fp32 TMEM accumulator, which restores fp32-grade
// accuracy.  kGemmTf32: one tf32 product on the raw fp32 operands.  kGemmHalfPair: the same three
// products at the fp16 rate, twice that of tf32, on interleaved fp16 pairs with a scale per row (half_pair.cuh):
// hi and lo of 32 consecutive K elements share one 128-byte swizzle row, so an operand is one array of
// 4 bytes per element, half of the tf32 pair's.  Both splits carry 11 + 11 significant bits: a tf32 pair at any
// size of the entry, an fp16 pair down to 2^-28 of its row's bound.  lo is stored times 2^11, so the two
// cross products go to an accumulator of their own and join the main one in the epilogue.  The fp16 split
// rounds lo where the tensor core truncates a tf32 lo, and sums 16 products instead of 8 before each (truncating)
// accumulation, so over rows whose entries lie within that range its error is the smaller one.  Measured on one
// B200 (the three products counted): 16 products of 2048^3 in 617 us instead of 1147 (1340 TFLOP/s against 720; cuBLAS
// bf16 reaches 1640), 6 of 768^3 in 31.5 us instead of 47, relative error against fp64 at K = 2048 2.5e-6 instead of 1.4e-5.
//
// Structure (one persistent CTA per SM, 192 threads, 320 with half pairs):
//   warp 0      TMA producer: cp.async.bulk.tensor tiles of 128 rows x 128 bytes, 128-byte swizzle
//   warp 1      MMA issuer: tcgen05.mma 128x128x8 kind::tf32, or 128x128x16 / 128x256x16 kind::f16,
//               accumulators in TMEM, two accumulator buffers so the epilogue of one tile overlaps
//               the next tile's MMAs (half pairs with 256 columns: main and cross accumulators fill the TMEM, one buffer)
//   warps 2..   epilogue (four warps, eight with half pairs): tcgen05.ld, transpose through shared memory, then coalesced global
//               access with the fused options below.
//
// Epilogue options per problem (flags):
//   kFlagPackedC    C is the row-major packed upper triangle of a symmetric N x N matrix; only
//                   entries with col >= row are touched (the tile list then holds only tiles
//                   on or above the diagonal)
//   kFlagSplitOut   additionally write the result as a (hi, lo) tf32 pair into d_hi/d_lo
//                   (row pitch ldd) so it can feed the next GEMM of a chain
//   kFlagSumSq      add the sum of squares of the results to *sumsq (Frobenius norm partials)
//   kFlagNoC        do not write C (only the split / sumsq outputs)
//   kFlagPeerPush   the result is also stored, in the communication dtype, into every rank's gather
//                   buffer over NVLink (fused all-gather of the search directions)
//   kFlagSquareAcc  the accumulator is squared before alpha/beta are applied: with C the running
//                   second moment V this is V <- beta2 V + w (Q_L^T G Q_R)^2 fused into the projection
//   kFlagMirror     the result is symmetric (products of commuting symmetric matrices, Grams): the
//                   tile list holds only tiles on or above the diagonal and every tile strictly
//                   above it is also stored transposed (C, d_hi, d_lo), so the full matrix is an
//                   operand of the next product at half the tensor-core work; sumsq counts such
//                   a tile twice
//   kFlagAddDiag    gamma (a launch scalar) is added to the diagonal entries: C = alpha A B^T +
//                   beta C + gamma I, the polynomial steps of the matrix sign iteration
//   kFlagTrace      add the diagonal entries of the result to sumsq[1] (trace)
#pragma once

#include <cstdint>
#include <cuda.h>

namespace ob200 {

constexpr int kFlagPackedC = 1;
constexpr int kFlagSplitOut = 2;
constexpr int kFlagSumSq = 4;
constexpr int kFlagNoC = 8;
constexpr int kFlagSquareAcc = 16;  // C = beta * C + alpha * acc^2 (second moment in the eigenbasis)
constexpr int kFlagMirror = 64;     // symmetric result: upper tiles computed, mirrored into the lower triangle
constexpr int kFlagAddDiag = 128;   // + gamma on the diagonal
constexpr int kFlagTrace = 256;     // sumsq[1] += trace of the result
constexpr int kFlagPeerPush = 32;   // also store the result, cast to the communication dtype, into the
                                    // problem's slot of every rank's gather buffer (PeerPush): the
                                    // all-gather of the search directions happens tile by tile from
                                    // the epilogue of the GEMM that produces them

constexpr int kFlagFixedScale = 512;  // half-pair split output: one bound for all rows, set by the caller in d_bound[0]; needed
                                      // where the result is more than alpha A B^T

constexpr int kErrPipelineTimeout = 1;  // a bounded mbarrier wait expired

struct alignas(128) GemmProblem {
  // 2-D tensor maps (dim0 = K, contiguous; dim1 = rows) of the arrays the operands are views of.
  // They live in device memory next to the problem table; several problems (the panels of a
  // blocked factorisation) may share one map and differ only in the view origin below.
  const CUtensorMap* a_hi;
  const CUtensorMap* a_lo;
  const CUtensorMap* b_hi;
  const CUtensorMap* b_lo;
  int a_row0, a_k0;  // origin of the A view inside its array (a_k0 a multiple of 4: TMA alignment)
  int b_row0, b_k0;  // a view that does not end where its array ends along K must have K % kBK == 0
  float* c;
  float* d_hi;
  float* d_lo;
  float* sumsq;
  int M, N, K;
  int ldc;  // row pitch of C in elements (full mode); N in packed mode
  int ldd;  // row pitch of d_hi / d_lo
  int flags;
  // kGemmHalfPair: bounds behind the scales of the operands' rows, that of row r at a_bound[r / a_div] (a re-viewed
  // array has several view rows per row it was written with; one bound for all rows has a div beyond any row).
  const float* a_bound;
  const float* b_bound;
  int a_div, b_div;
  // Bounds of the rows of a split output.  d_left null: d_bound[i] is given (RowBoundOp in block_kernels.cuh; kFlagFixedScale:
  // d_bound[0], for every row).  Else they follow from |sum_k a_ik b_jk| <= |a_i|_1 max|b|, or max|a_i| times the largest
  // |b_j|_1, and the epilogue writes them: d_bound[i] = |alpha| min(d_left[i] d_right[0], d_cap[0]), d_cap a bound of the
  // whole result or null.
  const float* d_left;
  const float* d_right;
  const float* d_cap;
  float* d_bound;
  long long push_offset;  // byte offset of the problem's slot inside the gather buffers (kFlagPeerPush)
};

// Destination of kFlagPeerPush stores: the gather buffer of every rank of the group (this rank
// included), all laid out identically.  Plain stores over NVLink; no TMA touches peer memory.
struct PeerPush {
  unsigned long long base[8];
  int num_peers;  // 0: no problem of the launch pushes
  int dtype;      // 0 fp32, 1 bf16, 2 fp16
};

// One work item: an output tile, or with parts > 1 the share [kb0, kb1) of its K blocks.  Every part leaves its
// accumulator at `partial` (part-major, kBM x cols floats each); of each 32-row stripe and half of its 32-column chunks the
// warp that arrives last at its counter adds the parts up in their order, so that the result does not depend on the
// arrival, and runs the epilogue on the sum.  No part waits for another.
struct alignas(16) GemmTile {
  int problem;
  int m0;  // first row of the tile
  int n0;  // first column of the tile
  int cols;  // 128, or 256 (half pairs only)
  int kb0, kb1;
  int part, parts;
  float* partial;
  int* counter;  // [kCountersPerTile], zero between launches
  int bufs;      // accumulator buffers in use, the same for all tiles of a launch: 1 where a tile has 256 columns
  int pad_[3];
};

// kGemmHalfPairSym: kGemmHalfPair with the epilogues of the symmetric iterations (split outputs with a given bound,
// mirrored, with beta, diagonal, norm and trace); an instantiation of its own, so that their registers do
// not weigh on the step's products.
enum GemmMode : int { kGemmTf32 = 0, kGemmTf32x3 = 1, kGemmHalfPair = 2, kGemmHalfPairSym = 3 };

constexpr int kCountersPerTile = 8;  // one per 32-row stripe and epilogue warp of it

constexpr int kBM = 128;
constexpr int kBN = 128;
constexpr int kBK = 32;  // fp32 elements (or fp16 pairs) = 128 bytes = one swizzle row

// Host-side launch.  `status` is a device int the kernel writes a non-zero error code to.
void launch_grouped_gemm(const GemmProblem* problems, const GemmTile* tiles, int num_tiles, float alpha, float beta,
                         GemmMode mode, int* status, int max_ctas, cudaStream_t stream, const PeerPush* push = nullptr,
                         float gamma = 0.f);

}  // namespace ob200
