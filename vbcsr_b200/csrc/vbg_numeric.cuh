// Numeric phase of the thresholded SpGEMM on the FP64 tensor cores
// (vbg_numeric.cu), called by vbg_spgemm.cu.
#pragma once

#include "vbg_internal.cuh"

namespace vbg {

// Pair gates.  kGateSum is the plain product (symbolic: keep j iff
// sum_k |A_ik||B_kj| > threshold; numeric: skip a pair below threshold /
// max(1, n_A)).  The others are the fused triple products' per-row gates
// (ops/spmm/rarh.hpp, rhar.hpp, square_polynomial.hpp): a pair
// (i,k)(k,j) reaches C's row only when |L_ik||R_kj| >= eps, and every column
// a pair reaches is kept by the symbolic phase:
//   kGateStage1  eps = thr / (2 max(1, n_L) |R row k| max|A|)   (T = L B)
//   kGateStage2  eps = thr / (2 n_L), |L_ik| the stage-one bound  (C = T A)
//   kGatePoly    eps = thr / max(1, n_L), 0 for an all-zero A      (A A)
// with n_L the left operand's blocks in row i; every eps is 0 for thr <= 0.
constexpr int kGateSum = 0;
constexpr int kGateStage1 = 1;
constexpr int kGateStage2 = 2;
constexpr int kGatePoly = 3;

__host__ __device__ inline double gate_eps(int mode, double thr, double amax, int nl, int nb) {
  if (mode == kGateStage1)
    return (thr > 0.0 && amax > 0.0 && nb > 0) ? thr / (2.0 * (double)(nl > 1 ? nl : 1) * (double)nb * amax) : 0.0;
  if (mode == kGateStage2) return (thr > 0.0 && nl > 0) ? thr / (2.0 * (double)nl) : 0.0;
  if (mode == kGatePoly) return (thr > 0.0 && amax > 0.0) ? thr / (double)(nl > 1 ? nl : 1) : 0.0;
  return thr / (double)(nl > 1 ? nl : 1);
}

// What decides which pairs a product keeps and what it leaves.
struct NumericGate {
  int mode = kGateSum;
  const double* amax = nullptr;  // gated modes: the largest block norm of A (device)
  double thr = 0.0;
  int drop = 1;                  // keep flags from the finished blocks' norms (else every block is kept)
  double* bound_out = nullptr;   // per C slot: the sum of the norms of its kept pairs (nullptr: not wanted)
};

// Merged rows of two block rows 2 p and 2 p + 1 of a pattern: entries
// {block column, slot in the first row or -1, slot in the second or -1, 0},
// columns ascending, from row_ptr[2 p] on; cnt[p] of them.
struct RowPairs {
  DevBuf list, cnt;  // used on the stream of the operation only
  explicit RowPairs(cudaStream_t s) : list(s), cnt(s) {}
};
// stats (device, may be nullptr): {most entries of a pair, most values of a
// pair's two rows} as maxima over the pairs, combined with what is there.
int merge_row_pairs(const vbg_matrix* m, RowPairs& out, int* stats, cudaStream_t s);

// C's values, keep flags, pair counts and bounds for C's pattern (its rows
// sorted).  A, B: blocks of at most 8 x 8, no block column twice in a row,
// B's column view built.  max_k, max_vals: merge_row_pairs' statistics of A;
// pairs: block pairs (i, k)(k, j) whose C block may exist.
// kNumericNotFit when a pair of A's rows does not fit shared memory (nothing
// launched).
constexpr int kNumericNotFit = 1;
int numeric_pairs(const vbg_matrix* A, const vbg_matrix* B, vbg_matrix* C, const RowPairs& ka, int max_k,
                  int max_vals, double pairs, const double* normsA, const double* normsB, const NumericGate& gate,
                  unsigned char* keep, unsigned long long* products, cudaStream_t s);

}  // namespace vbg
