// Numeric phase of the thresholded SpGEMM, FP64 tensor-core form (blocks of at
// most 8 x 8, real and complex): C_ij = sum over k of A_ik B_kj, pairs skipped
// when |A_ik| |B_kj| is below the row's gate (ops/spmm/vbcsr.hpp:372,386 of
// the reference), the finished blocks' norms giving the filter's keep flags.
//
// A CTA computes two consecutive block rows of C.  Their A rows are merged
// into one list of inner block columns k beforehand (merge_row_pairs), and so
// are C's two rows; the CTA keeps the A values of both rows and the list in
// shared memory.  A warp takes J of the merged C columns at a time: for each
// it walks B's column (32 entries a round: row, norm and value offset,
// coalesced), finds k in the list (a window table, or a binary search when
// the list's columns span more than kWin), tests the gate for both rows and
// notes the offset and the kept rows in a table over (k, column).  Then it
// multiplies what was kept, A's fragments of the two rows from shared memory
// and B's from L2, two m8n8k4 steps a block product: all J columns in one
// pass over k when most pairs are kept, else a column at a time over its own.
//
// What bounds it: B's fragments from L2 (each serves both rows) and the
// instructions around the tensor steps.  One C block per warp and pass, as it
// was before, loaded both fragments for every pair, kept a list entry with
// two 64-bit offsets per pair, and ran one launch per block size in series (52
// instructions a pair, 1.93 ms on 12000 rows of 4-8, 29 blocks a row, 8.3 M
// pairs).  Warp instructions a kept pair now: 34 in the dense form (3000 rows of
// 121 full blocks of 6, 43 M pairs: 2.67 ms, tensor pipe active 45 %), 82 in the
// sparse form on the 8.3 M pairs (1.38 ms, 17 %), whose short lists pay for the
// walk of B's columns.
#include <algorithm>
#include <type_traits>

#include "vbg_numeric.cuh"

namespace vbg {

constexpr int kWin = 1024;  // window table entries
constexpr size_t kPairsSmem2 = 113 * 1024;  // two CTAs per SM
constexpr size_t kPairsSmem1 = 226 * 1024;  // one CTA per SM

// A warp per row pair.  Both rows are sorted and hold distinct columns: an
// entry's place in the union is its own index plus the other row's entries
// below it, less the columns both hold below it.
__global__ void merge_row_pairs_kernel(int n, const int* __restrict__ rp, const int* __restrict__ ci,
                                       const int64_t* __restrict__ off, int4* __restrict__ list,
                                       int* __restrict__ cnt, int* __restrict__ stats) {
  const int lane = threadIdx.x & 31;
  const int np = (n + 1) / 2;
  const unsigned below = (1u << lane) - 1u;
  for (int p = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); p < np; p += gridDim.x * (blockDim.x >> 5)) {
    const int s0 = rp[2 * p], s1 = rp[2 * p + 1], s2 = 2 * p + 1 < n ? rp[2 * p + 2] : s1;
    auto find = [&](int lo, int hi, int c) {  // first slot in [lo, hi) with column >= c
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (ci[mid] < c) lo = mid + 1;
        else hi = mid;
      }
      return lo;
    };
    int both = 0;
    for (int b = s0; b < s1; b += 32) {
      const int s = b + lane;
      const bool on = s < s1;
      const int c = on ? ci[s] : 0;
      const int o = on ? find(s1, s2, c) : s2;
      const bool hit = on && o < s2 && ci[o] == c;
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (on) list[s0 + (s - s0) + (o - s1) - both - __popc(m & below)] = make_int4(c, s, hit ? o : -1, 0);
      both += __popc(m);
    }
    int seen = 0;
    for (int b = s1; b < s2; b += 32) {
      const int s = b + lane;
      const bool on = s < s2;
      const int c = on ? ci[s] : 0;
      const int o = on ? find(s0, s1, c) : s1;
      const bool hit = on && o < s1 && ci[o] == c;
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (on && !hit) list[s0 + (s - s1) + (o - s0) - seen - __popc(m & below)] = make_int4(c, -1, s, 0);
      seen += __popc(m);
    }
    if (lane == 0) {
      const int k = (s2 - s0) - both;
      cnt[p] = k;
      if (stats) {
        atomicMax(stats, k);
        atomicMax(stats + 1, (int)min((int64_t)INT32_MAX, off[s2] - off[s0]));
      }
    }
  }
}

int merge_row_pairs(const vbg_matrix* m, RowPairs& out, int* stats, cudaStream_t s) {
  const int np = (m->n + 1) / 2;
  int rc;
  if ((rc = out.list.ensure(std::max<int64_t>(m->nnzb, 1) * sizeof(int4), s))) return rc;
  if ((rc = out.cnt.ensure(std::max(np, 1) * sizeof(int), s))) return rc;
  if (!np) return 0;
  const int grid = std::max(1, std::min((np + 7) / 8, sm_count() * 16));
  merge_row_pairs_kernel<<<grid, 256, 0, s>>>(m->n, m->row_ptr.as<int>(), m->col_ind.as<int>(),
                                              m->blk_off.as<int64_t>(), out.list.as<int4>(), out.cnt.as<int>(), stats);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

// B's column view as the walk reads it: {norm, value offset} of every entry.
struct alignas(16) ColRec {
  double norm;
  long long off;
};
__global__ void column_records_kernel(int64_t nnzb, const int* __restrict__ slot, const double* __restrict__ norms,
                                      const int64_t* __restrict__ off, ColRec* __restrict__ rec) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nnzb; t += (int64_t)gridDim.x * blockDim.x) {
    const int s = slot[t];
    rec[t] = {norms[s], (long long)off[s]};
  }
}

struct PairsArgs {
  int n;
  const int4* ka;      // merged A rows
  const int* ka_cnt;
  const int* a_rp;
  const int64_t* a_off;
  const double* nA;
  const int4* cj;      // merged C rows
  const int* cj_cnt;
  const int* c_rp;
  const int64_t* c_off;
  const int* bt_ptr;
  const int* bt_row;
  const ColRec* bt_rec;
  const int* b_rp;
  const int* bsz;
  NumericGate gate;
  unsigned char* keep;
  unsigned long long* products;
  int kc;              // list entries shared memory has room for
  int vc;              // and A values
};

// Shared memory: A values (vc) | norms of both rows (2 kc doubles) | records
// {A offsets in the first and second row, inner size + 16 if the first row
// holds k + 32 if the second does, 0} (kc int4) | offset tables of the warps
// (kc J ints each) | columns (kc ints) | kept-row bits of the warps (kc bytes
// each).  kc is a multiple of 16.
__host__ __device__ inline size_t pairs_smem(int kc, int vc, int es, int J, int warps) {
  return ((size_t)vc * es + 15) / 16 * 16 + (size_t)kc * (16 + 16 + 4ull * J * warps + 4 + warps);
}

template <typename T> struct PairsJ { static constexpr int v = 4; };
template <> struct PairsJ<cplx> { static constexpr int v = 2; };

// One operand fragment half of a lane.
template <typename T>
__device__ __forceinline__ T frag_or_zero(bool on, const T* p) {
  return on ? *p : zero_s<T>();
}
template <typename T>
__device__ __forceinline__ T frag_or_zero_ldg(bool on, const T* p) {
  if constexpr (std::is_same<T, cplx>::value) {
    if (!on) return zero_s<T>();
    const double2 v = __ldg(reinterpret_cast<const double2*>(p));
    return {v.x, v.y};
  } else {
    return on ? __ldg(p) : 0.0;
  }
}
// acc: this lane's two elements of a C tile.
__device__ __forceinline__ void pair_mma(double (&acc)[2], double a, double b) { dmma_884(acc[0], acc[1], a, b); }
__device__ __forceinline__ void pair_mma(cplx (&acc)[2], cplx a, cplx b) {
  dmma_884(acc[0].re, acc[1].re, a.re, b.re);
  dmma_884(acc[0].im, acc[1].im, a.re, b.im);
  dmma_884(acc[0].re, acc[1].re, -a.im, b.im);
  dmma_884(acc[0].im, acc[1].im, a.im, b.re);
}
__device__ __forceinline__ double sq_abs(double v) { return __dmul_rn(v, v); }
__device__ __forceinline__ double sq_abs(cplx v) { return fma(v.re, v.re, __dmul_rn(v.im, v.im)); }

// CTAs per SM and pairs in flight of the sparse form.  It is bound by the
// latency of its short loops, so warps count for more than pairs in flight:
// for whole products of 12000 rows (real) and a 60 x 60 lattice (complex),
// two CTAs of four or two pairs took 2272 and 1173 us, three of two 1952,
// four of one 1072.
template <typename T>
constexpr int kSparseCtas = std::is_same<T, cplx>::value ? 4 : 3;
template <typename T>
constexpr int kSparsePairs = std::is_same<T, cplx>::value ? 1 : 2;

template <typename T, bool GATED, bool DENSE>
__global__ void __launch_bounds__(DENSE ? 512 : 256, DENSE ? 1 : kSparseCtas<T>)
    numeric_pairs_kernel(PairsArgs a, const T* __restrict__ A, const T* __restrict__ B, T* __restrict__ C) {
  constexpr int J = PairsJ<T>::v;
  extern __shared__ __align__(16) unsigned char pairs_raw[];
  __shared__ short wtab[kWin];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int kc = a.kc;
  T* sA = reinterpret_cast<T*>(pairs_raw);
  double* kn0 = reinterpret_cast<double*>(pairs_raw + ((size_t)a.vc * sizeof(T) + 15) / 16 * 16);
  double* kn1 = kn0 + kc;
  int4* krec = reinterpret_cast<int4*>(kn1 + kc);
  int* tab_all = reinterpret_cast<int*>(krec + kc);
  int* tab = tab_all + (size_t)warp * kc * J;
  int* kcol = tab_all + (size_t)warps * kc * J;
  unsigned char* bits = reinterpret_cast<unsigned char*>(kcol + kc) + (size_t)warp * kc;

  const int i0 = 2 * blockIdx.x;
  const bool second = i0 + 1 < a.n;
  const int s0 = a.a_rp[i0], s1 = a.a_rp[i0 + 1], s2 = second ? a.a_rp[i0 + 2] : s1;
  const int64_t av0 = a.a_off[s0];
  const int nv = (int)(a.a_off[s2] - av0);
  const int nk = a.ka_cnt[blockIdx.x], nc = a.cj_cnt[blockIdx.x];
  if (nc == 0) return;
  const double thr = a.gate.thr;
  const int mode = GATED ? a.gate.mode : kGateSum;
  const double amax = GATED ? *a.gate.amax : 0.0;
  const double eps0 = gate_eps(mode, thr, amax, s1 - s0, 0), eps1 = gate_eps(mode, thr, amax, s2 - s1, 0);
  for (int e = threadIdx.x; e < nv; e += blockDim.x) sA[e] = A[av0 + e];
  const int4* kl = a.ka + s0;
  const int kmin = nk ? kl[0].x : 0, span = nk ? kl[nk - 1].x - kmin + 1 : 0;
  if (span <= kWin)
    for (int t = threadIdx.x; t < span; t += blockDim.x) wtab[t] = -1;
  for (int t = threadIdx.x; t < nk; t += blockDim.x) {
    const int4 e = kl[t];
    kcol[t] = e.x;
    kn0[t] = e.y >= 0 ? a.nA[e.y] : 0.0;
    kn1[t] = e.z >= 0 ? a.nA[e.z] : 0.0;
    krec[t] = make_int4(e.y >= 0 ? (int)(a.a_off[e.y] - av0) : 0, e.z >= 0 ? (int)(a.a_off[e.z] - av0) : 0,
                        a.bsz[e.x] | (e.y >= 0 ? 16 : 0) | (e.z >= 0 ? 32 : 0), 0);
  }
  __syncthreads();
  if (span <= kWin)
    for (int t = threadIdx.x; t < nk; t += blockDim.x) wtab[kcol[t] - kmin] = (short)t;
  __syncthreads();
  const int r0 = a.bsz[i0], r1 = second ? a.bsz[i0 + 1] : 1;
  // this lane's row in the A blocks: rows past the block repeat its last one
  // (their results are not stored)
  const int ar0 = min(g, r0 - 1), ar1 = min(g, r1 - 1);
  const int4* cl = a.cj + a.c_rp[i0];
  unsigned prods = 0;

  for (int grp = warp * J; grp < nc; grp += warps * J) {
    const int gn = min(J, nc - grp);
    int4 ce = make_int4(-1, -1, -1, 0);
    if (lane < gn) ce = cl[grp + lane];
    for (int t = lane; t < nk; t += 32) bits[t] = 0;
    // lane c: column c's width and, gated, the sums of its kept pair norms
    const int lcc = lane < gn ? a.bsz[ce.x] : 1;
    double lsum0 = 0.0, lsum1 = 0.0;
    __syncwarp();
#pragma unroll 1
    for (int c = 0; c < gn; ++c) {
      const int j = __shfl_sync(0xffffffffu, ce.x, c);
      const bool want0 = __shfl_sync(0xffffffffu, ce.y, c) >= 0, want1 = __shfl_sync(0xffffffffu, ce.z, c) >= 0;
      double bsum0 = 0.0, bsum1 = 0.0;
      const int q0 = a.bt_ptr[j], q1 = a.bt_ptr[j + 1];
      for (int q = q0 + lane; q < q1; q += 32) {
        const int k = a.bt_row[q];
        const ColRec rec = a.bt_rec[q];
        int idx = -1;
        if (span <= kWin) {
          const unsigned d = (unsigned)(k - kmin);
          if (d < (unsigned)span) idx = wtab[d];
        } else {
          int lo = 0, hi = nk;
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (kcol[mid] < k) lo = mid + 1;
            else hi = mid;
          }
          if (lo < nk && kcol[lo] == k) idx = lo;
        }
        if (idx < 0) continue;
        double e0 = eps0, e1 = eps1;
        if (GATED && mode == kGateStage1) {
          const int nb = a.b_rp[k + 1] - a.b_rp[k];
          e0 = gate_eps(kGateStage1, thr, amax, s1 - s0, nb);
          e1 = gate_eps(kGateStage1, thr, amax, s2 - s1, nb);
        }
        const double p0 = kn0[idx] * rec.norm, p1 = kn1[idx] * rec.norm;
        const unsigned has = (unsigned)krec[idx].z;
        const bool on0 = want0 && (has & 16u) && !(p0 < e0), on1 = want1 && (has & 32u) && !(p1 < e1);
        if (on0 || on1) {
          tab[idx * J + c] = (int)rec.off;
          bits[idx] |= (unsigned char)((on0 ? 1u << c : 0u) | (on1 ? 16u << c : 0u));
          prods += (on0 ? 1u : 0u) + (on1 ? 1u : 0u);
          if (GATED) {
            if (on0) bsum0 += p0;
            if (on1) bsum1 += p1;
          }
        }
      }
      __syncwarp();
      if (GATED) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          bsum0 += __shfl_xor_sync(0xffffffffu, bsum0, off);
          bsum1 += __shfl_xor_sync(0xffffffffu, bsum1, off);
        }
        if (lane == c) {
          lsum0 = bsum0;
          lsum1 = bsum1;
        }
      }
    }
    // the finished blocks, their norms and keep flags
    auto finish = [&](const T(&acc)[2], int p, int r, int c, double bsum) {
      T* cp = C + a.c_off[p];
      const int u = 2 * t4;
      double sq = 0.0;
      if (g < r) {
        if (u < c) {
          cp[g * c + u] = acc[0];
          sq = sq_abs(acc[0]);
        }
        if (u + 1 < c) {
          cp[g * c + u + 1] = acc[1];
          sq = __dadd_rn(sq, sq_abs(acc[1]));
        }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
      if (GATED && a.gate.bound_out && lane == 0) a.gate.bound_out[p] = bsum;
      if (lane == 0) a.keep[p] = ((GATED && !a.gate.drop) || thr <= 0.0 || sqrt(sq) >= thr) ? 1 : 0;
    };
    if constexpr (DENSE) {
      // columns past the block: as the rows
      int cc[J], bi[J];
#pragma unroll
      for (int c = 0; c < J; ++c) {
        cc[c] = __shfl_sync(0xffffffffu, lcc, c);
        bi[c] = t4 * cc[c] + min(g, cc[c] - 1);
      }
      T acc0[J][2], acc1[J][2];
#pragma unroll
      for (int c = 0; c < J; ++c) acc0[c][0] = acc0[c][1] = acc1[c][0] = acc1[c][1] = zero_s<T>();
      constexpr unsigned kFull = (1u << J) - 1u;
      for (int t = 0; t < nk; t += 2) {
        unsigned m[2];
        m[0] = bits[t];
        m[1] = t + 1 < nk ? bits[t + 1] : 0u;
        if ((m[0] | m[1]) == 0u) continue;
        T fa0[2][2], fa1[2][2], fb[2][J][2];
        int in[2];
        // all operands of two inner block columns, then their products
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          in[u] = 0;
          if (m[u] == 0u) continue;
          const int4 kr = krec[t + u];
          in[u] = kr.z & 15;
          const bool h0 = t4 < in[u], h1 = t4 + 4 < in[u];
          const int* to = tab + (t + u) * J;
#pragma unroll
          for (int c = 0; c < J; ++c)
            if ((m[u] >> c) & 0x11u) {
              const T* bp = B + to[c] + bi[c];
              fb[u][c][0] = frag_or_zero_ldg(h0, bp);
              fb[u][c][1] = frag_or_zero_ldg(h1, bp + 4 * cc[c]);
            }
          if (m[u] & 0xfu) {
            const T* ap = sA + kr.x + ar0 * in[u] + t4;
            fa0[u][0] = frag_or_zero(h0, ap);
            fa0[u][1] = frag_or_zero(h1, ap + 4);
          }
          if (m[u] & 0xf0u) {
            const T* ap = sA + kr.y + ar1 * in[u] + t4;
            fa1[u][0] = frag_or_zero(h0, ap);
            fa1[u][1] = frag_or_zero(h1, ap + 4);
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (m[u] == (kFull | (kFull << 4))) {
#pragma unroll
            for (int c = 0; c < J; ++c) {
              pair_mma(acc0[c], fa0[u][0], fb[u][c][0]);
              pair_mma(acc1[c], fa1[u][0], fb[u][c][0]);
            }
            if (in[u] > 4) {
#pragma unroll
              for (int c = 0; c < J; ++c) {
                pair_mma(acc0[c], fa0[u][1], fb[u][c][1]);
                pair_mma(acc1[c], fa1[u][1], fb[u][c][1]);
              }
            }
          } else {
#pragma unroll
            for (int c = 0; c < J; ++c) {
              if ((m[u] >> c) & 1u) {
                pair_mma(acc0[c], fa0[u][0], fb[u][c][0]);
                if (in[u] > 4) pair_mma(acc0[c], fa0[u][1], fb[u][c][1]);
              }
              if ((m[u] >> c) & 16u) {
                pair_mma(acc1[c], fa1[u][0], fb[u][c][0]);
                if (in[u] > 4) pair_mma(acc1[c], fa1[u][1], fb[u][c][1]);
              }
            }
          }
        }
      }
#pragma unroll
      for (int c = 0; c < J; ++c) {
        const int p0 = __shfl_sync(0xffffffffu, ce.y, c), p1 = __shfl_sync(0xffffffffu, ce.z, c);
        const double b0 = GATED ? __shfl_sync(0xffffffffu, lsum0, c) : 0.0;
        const double b1 = GATED ? __shfl_sync(0xffffffffu, lsum1, c) : 0.0;
        if (p0 >= 0) finish(acc0[c], p0, r0, cc[c], b0);
        if (p1 >= 0) finish(acc1[c], p1, r1, cc[c], b1);
      }
    } else {
#pragma unroll 1
      for (int c = 0; c < gn; ++c) {
        const int cc = __shfl_sync(0xffffffffu, lcc, c), bi = t4 * cc + min(g, cc - 1);
        T acc0[2] = {zero_s<T>(), zero_s<T>()}, acc1[2] = {zero_s<T>(), zero_s<T>()};
        for (int kb = 0; kb < nk; kb += 32) {
          const unsigned m = kb + lane < nk ? (unsigned)bits[kb + lane] >> c : 0u;
          const unsigned w0 = __ballot_sync(0xffffffffu, m & 1u), w1 = __ballot_sync(0xffffffffu, m & 16u);
          for (unsigned w = w0 | w1; w;) {
            constexpr int U = kSparsePairs<T>;
            T fa0[U][2], fa1[U][2], fb[U][2];
            int in[U];
            unsigned at[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              at[u] = w & (0u - w);  // the lowest kept k, as a bit (0: none left)
              w ^= at[u];
              in[u] = 0;
              if (at[u] == 0u) continue;
              const int t = kb + __ffs(at[u]) - 1;
              const int4 kr = krec[t];
              in[u] = kr.z & 15;
              const bool h0 = t4 < in[u], h1 = t4 + 4 < in[u];
              const T* bp = B + tab[t * J + c] + bi;
              fb[u][0] = frag_or_zero_ldg(h0, bp);
              fb[u][1] = frag_or_zero_ldg(h1, bp + 4 * cc);
              const T *p0 = sA + kr.x + ar0 * in[u] + t4, *p1 = sA + kr.y + ar1 * in[u] + t4;
              fa0[u][0] = frag_or_zero(h0, p0);
              fa0[u][1] = frag_or_zero(h1, p0 + 4);
              fa1[u][0] = frag_or_zero(h0, p1);
              fa1[u][1] = frag_or_zero(h1, p1 + 4);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
              if (at[u] & w0) {
                pair_mma(acc0, fa0[u][0], fb[u][0]);
                if (in[u] > 4) pair_mma(acc0, fa0[u][1], fb[u][1]);
              }
              if (at[u] & w1) {
                pair_mma(acc1, fa1[u][0], fb[u][0]);
                if (in[u] > 4) pair_mma(acc1, fa1[u][1], fb[u][1]);
              }
            }
          }
        }
        const int p0 = __shfl_sync(0xffffffffu, ce.y, c), p1 = __shfl_sync(0xffffffffu, ce.z, c);
        const double b0 = GATED ? __shfl_sync(0xffffffffu, lsum0, c) : 0.0;
        const double b1 = GATED ? __shfl_sync(0xffffffffu, lsum1, c) : 0.0;
        if (p0 >= 0) finish(acc0, p0, r0, cc, b0);
        if (p1 >= 0) finish(acc1, p1, r1, cc, b1);
      }
    }
    __syncwarp();  // the next columns rewrite the tables
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) prods += __shfl_xor_sync(0xffffffffu, prods, off);
  if (lane == 0 && prods) atomicAdd(a.products, (unsigned long long)prods);
}

template <typename T, bool GATED, bool DENSE>
static int launch_pairs_k(const PairsArgs& a, int warps, size_t smem, const T* A, const T* B, T* C, cudaStream_t s) {
  static bool attr[kMaxDevices] = {};
  const int dev = current_device();
  if (!attr[dev]) {
    VBG_CUDA(cudaFuncSetAttribute(numeric_pairs_kernel<T, GATED, DENSE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kPairsSmem1 - kWin * (int)sizeof(short)));
    attr[dev] = true;
  }
  numeric_pairs_kernel<T, GATED, DENSE><<<(a.n + 1) / 2, warps * 32, smem, s>>>(a, A, B, C);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

template <typename T>
static int launch_pairs(const PairsArgs& a, bool gated, bool dense, int warps, size_t smem, const vbg_matrix* A,
                        const vbg_matrix* B, vbg_matrix* C, cudaStream_t s) {
  const T *va = A->vals.as<T>(), *vb = B->vals.as<T>();
  T* vc = C->vals.as<T>();
  if (gated)
    return dense ? launch_pairs_k<T, true, true>(a, warps, smem, va, vb, vc, s)
                 : launch_pairs_k<T, true, false>(a, warps, smem, va, vb, vc, s);
  return dense ? launch_pairs_k<T, false, true>(a, warps, smem, va, vb, vc, s)
               : launch_pairs_k<T, false, false>(a, warps, smem, va, vb, vc, s);
}

// The share of C's blocks' inner columns that hold a pair from which a pass
// over all of them with J products each (DENSE) beats running through every
// C column's own pairs.  Whole products, us, dense / sparse form, blocks of 4-8:
// share 0.26 (31 of 65 columns of a band) 1716 / 1333, complex 2502 / 2206; 0.33
// 2170 / 1736 and 3414 / 3621; 0.41 1004 / 888 and 1563 / 1680; random rows of
// 160 blocks at 0.5 682 / 663 and 705 / 940, at 0.7 714 / 911 and 983 / 1388.
// Full bands of blocks of 6 (share 0.5): 65 blocks a row 1376 / 1247, 121 3238 /
// 3503, 201 8421 / 14374; complex 49 1579 / 1503, 65 2460 / 2594, 121 7191 /
// 10827: the longer the rows, the fewer CTAs of the sparse form share an SM.
constexpr double kDenseShare = 0.45;

int numeric_pairs(const vbg_matrix* A, const vbg_matrix* B, vbg_matrix* C, const RowPairs& ka, int max_k,
                  int max_vals, double pairs, const double* normsA, const double* normsB, const NumericGate& gate,
                  unsigned char* keep, unsigned long long* products, cudaStream_t s) {
  const bool cx = C->dtype == VBG_C128;
  const int es = cx ? 16 : 8, J = cx ? PairsJ<cplx>::v : PairsJ<double>::v;
  const int kc = std::max(16, (max_k + 15) / 16 * 16);
  // offsets into B and indexes into the list are 32 and 16 bits wide
  if (B->nnz >= (int64_t)INT32_MAX || kc > 32767 || max_vals == INT32_MAX) return kNumericNotFit;
  const size_t fixed = kWin * sizeof(short) + 1024;  // the window table and the system's share
  // eight warps; the dense form sixteen where two CTAs of eight do not share an
  // SM but one of sixteen fits (their tables grow with the warps); one CTA of
  // eight an SM only over four rounds of them, else the item kernel's warps fill
  // the SMs better (real blocks of 6, 261 full blocks a row, 3000 rows: 21 ms
  // against 28; 300 x 300 full: 6.3 against 4.2)
  const bool dense = pairs * A->n >= kDenseShare * (double)C->nnzb * (double)A->nnzb;
  int warps = 8;
  size_t smem = pairs_smem(kc, max_vals, es, J, warps);
  if (dense && smem + fixed > kPairsSmem2) {
    const size_t more = pairs_smem(kc, max_vals, es, J, 16);
    if (more + fixed <= kPairsSmem1) {
      warps = 16;
      smem = more;
    } else if (A->n < 8 * sm_count()) {
      return kNumericNotFit;
    }
  }
  if (smem + fixed > kPairsSmem1) return kNumericNotFit;
  RowPairs cj(s);
  int rc;
  if (!A->n) return 0;
  if ((rc = merge_row_pairs(C, cj, nullptr, s))) return rc;
  DevBuf rec(s);
  if ((rc = rec.ensure(std::max<int64_t>(B->nnzb, 1) * sizeof(ColRec)))) return rc;
  if (B->nnzb) {
    const int g = (int)std::min<int64_t>((B->nnzb + 255) / 256, (int64_t)sm_count() * 16);
    column_records_kernel<<<g, 256, 0, s>>>(B->nnzb, B->csc_slot.as<int>(), normsB, B->blk_off.as<int64_t>(),
                                            rec.as<ColRec>());
    VBG_CUDA(cudaGetLastError());
  }
  PairsArgs a{};
  a.n = A->n;
  a.ka = ka.list.as<int4>();
  a.ka_cnt = ka.cnt.as<int>();
  a.a_rp = A->row_ptr.as<int>();
  a.a_off = A->blk_off.as<int64_t>();
  a.nA = normsA;
  a.cj = cj.list.as<int4>();
  a.cj_cnt = cj.cnt.as<int>();
  a.c_rp = C->row_ptr.as<int>();
  a.c_off = C->blk_off.as<int64_t>();
  a.bt_ptr = B->csc_ptr.as<int>();
  a.bt_row = B->csc_row.as<int>();
  a.bt_rec = rec.as<ColRec>();
  a.b_rp = B->row_ptr.as<int>();
  a.bsz = A->bsz.as<int>();
  a.gate = gate;
  a.keep = keep;
  a.products = products;
  a.kc = kc;
  a.vc = max_vals;
  const bool gated = gate.mode != kGateSum || gate.bound_out || !gate.drop;
  return cx ? launch_pairs<cplx>(a, gated, dense, warps, smem, A, B, C, s)
            : launch_pairs<double>(a, gated, dense, warps, smem, A, B, C, s);
}

}  // namespace vbg
