// Arguments of the sparse apply kernels and the reductions they share
// (vbg_apply.cu, vbg_mma.cu).
#pragma once

#include "vbg_internal.cuh"

namespace vbg {

struct ApplyArgs {
  int n_rows;                // output block rows
  const int* order;          // visiting order of output rows (nullptr = natural)
  const int* ptr;            // entry range per output row (row_ptr or csc_ptr)
  const int* ent_slot;       // adjoint: slot of each entry (forward: entry == slot)
  const int* ent_src;        // source block of each entry (col_ind or csc_row)
  const int* bsz;
  const int64_t* scal_off;
  const int64_t* blk_off;
  const int2* slot_meta;     // forward: per slot {first X row of the block column, rows << 8 | cols}
  const int64_t* koff;       // pipelined kernel: per-slot offsets of the kernel-layout values
  const int4* spans;         // pipelined kernel: spans, FP32 layout offsets, each block row's span range
  const int64_t* span_koff32;
  const int* row_sptr;
  int ld;                    // leading dimension of X/Y in elements (1 = vector)
  // epilogue  Y = alpha * (A X) + beta * X + gamma * Xprev
  double alpha, beta, gamma;
  const void* X;
  const void* Xprev;
  void* Y;
  const void* dotw;          // dot partner for dots[0] (nullptr -> X)
  void* acc;                 // acc += acc_coef * Y (nullptr -> none)
  double cre, cim;
  int want_dots;
  double* row_dots;          // with want_dots: per block row (d0, d1) here instead of the grid reduction
  double* partials;
  unsigned* counter;
  double* dots_out;
  int max_ctas;              // CTAs `partials` has room for (0: max_total_ctas())
  // vector apply: ranges each CTA prefetches its share of into L2 at start
  // (16-byte aligned; set when the whole working set fits L2)
  int npf;
  const void* pf_ptr[4];
  long long pf_bytes[4];
  // scalar-row vector apply: per scalar row {first slot, count << 8 | row in block}, scalar rows
  const int2* srow;
  int64_t n_scal;
};

__device__ __forceinline__ double shfl_xor_s(double v, int off) { return __shfl_xor_sync(0xffffffffu, v, off); }
__device__ __forceinline__ float shfl_xor_s(float v, int off) { return __shfl_xor_sync(0xffffffffu, v, off); }
__device__ __forceinline__ cplx shfl_xor_s(cplx v, int off) {
  return {__shfl_xor_sync(0xffffffffu, v.re, off), __shfl_xor_sync(0xffffffffu, v.im, off)};
}
__device__ __forceinline__ double add_s(double a, double b) { return a + b; }
__device__ __forceinline__ float add_s(float a, float b) { return a + b; }
__device__ __forceinline__ cplx add_s(cplx a, cplx b) { return {a.re + b.re, a.im + b.im}; }

// Fixed-order two-value reduction across the grid: per-CTA partials, then
// the last CTA to finish sums them in a fixed tree and resets the counter.
// Blocks have at most 1024 threads.
static __device__ void grid_reduce2(double d0, double d1, double* partials, unsigned* counter, double* out, int part_base,
                             int total) {
  __shared__ double red[32][2];
  __shared__ bool is_last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    d0 += __shfl_xor_sync(0xffffffffu, d0, off);
    d1 += __shfl_xor_sync(0xffffffffu, d1, off);
  }
  if (lane == 0) {
    red[warp][0] = d0;
    red[warp][1] = d1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double s0 = 0.0, s1 = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      s0 += red[w][0];
      s1 += red[w][1];
    }
    partials[2 * (part_base + blockIdx.x)] = s0;
    partials[2 * (part_base + blockIdx.x) + 1] = s1;
    __threadfence();
    const unsigned prev = atomicAdd(counter, 1u);
    is_last = (prev == (unsigned)total - 1);
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  double s0 = 0.0, s1 = 0.0;
  for (int b = threadIdx.x; b < total; b += blockDim.x) {
    s0 += __ldcg(partials + 2 * b);
    s1 += __ldcg(partials + 2 * b + 1);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, off);
    s1 += __shfl_xor_sync(0xffffffffu, s1, off);
  }
  __syncthreads();
  if (lane == 0) {
    red[warp][0] = s0;
    red[warp][1] = s1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t0 = 0.0, t1 = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      t0 += red[w][0];
      t1 += red[w][1];
    }
    out[0] = t0;
    out[1] = t1;
    *counter = 0u;
  }
}

// Per-row dot output (batched recurrences): sums this row's lane partials
// over the warp and writes them; the caller's accumulators are untouched.
__device__ __forceinline__ void write_row_dots(double* row_dots, int row, double r0, double r1) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    r0 += __shfl_xor_sync(0xffffffffu, r0, off);
    r1 += __shfl_xor_sync(0xffffffffu, r1, off);
  }
  if ((threadIdx.x & 31) == 0) {
    row_dots[2 * row] = r0;
    row_dots[2 * row + 1] = r1;
  }
}

// Largest number of CTAs one apply (all its launches together) can use.
inline int max_total_ctas() { return sm_count() * 8 * 10; }

// A launch that reduces its dots through `partials` must fit them: `total`
// CTAs of this apply against the room the caller gave (a.max_ctas), else the
// library's scratch (max_total_ctas()).
inline int check_dot_ctas(const ApplyArgs& a, int total) {
  if (!a.want_dots || a.row_dots) return 0;
  const int cap = a.max_ctas > 0 ? a.max_ctas : max_total_ctas();
  if (total <= cap) return 0;
  return fail(a.max_ctas > 0 ? VBG_E_ARG : VBG_E_STATE,
              "this launch needs " + std::to_string(total) + " CTA partial sums; the dot scratch holds " +
                  std::to_string(cap));
}

constexpr int kSplitWantWarps = 24;
// Warps that share a task: the fewest of 1, 2, 4, 8 that give every SM
// kSplitWantWarps warps (a warp alone walks its row's entries two at a time, so
// a matrix of few rows otherwise waits on one row's loads), while each still
// gets two entries of an average row.
inline int row_split(const vbg_matrix* m, int64_t ntasks) {
  const int64_t want = (int64_t)sm_count() * kSplitWantWarps;
  int s = 1;
  while (s < 8 && ntasks * s < want && m->nnzb >= 4 * (int64_t)s * m->n) s *= 2;
  return s;
}

// The row-wise multivector apply on the FP64 tensor cores (vbg_mma.cu), FP64
// and complex values.
int launch_mma(const vbg_matrix* m, bool adj, const ApplyArgs& a, cudaStream_t s);

}  // namespace vbg
