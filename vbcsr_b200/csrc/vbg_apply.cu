// Sparse apply kernels: y = A x, Y = A X, their adjoints, the fused Chebyshev
// step (recurrence update + moment dot products in one pass) and the KPM
// moment loop built on it.
//
// Reference behaviour replaced:
//   BlockSpMat::mult / mult_dense / mult_adjoint / mult_dense_adjoint
//     vbcsr/core/block_csr.hpp:985-1050
//   row-direct apply  vbcsr/core/detail/kernels/vbcsr_apply.hpp:193-244 (mult),
//     :277-340 (mult_dense), :342-424 (adjoint)
//   per-block kernels rm_gemv / rm_gemm
//     vbcsr/core/detail/kernels/rowmajor_kernels.hpp:45-185,552-600
//   Chebyshev loop bodies examples/ex08_graphene_dos.py:99-114,
//     examples/inp_nanocrystal_dos/kpm.py:40-74, vbcsr/utils.py:71-126
//
// Layout: one warp per output block row.  For a plain vector the 32 lanes are
// split into (block, row-within-block) pairs, each lane reducing one r x c
// block row against its x strip; for a multivector the lanes cover the padded
// row of X (16-byte vectors per lane: 2 FP64, 4 FP32 or 1 complex) and lane
// groups split the row's blocks when the row is narrower than a warp.  Rows
// are visited in block-size-class order and the block size r is a
// compile-time constant inside each class body.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <numeric>
#include <type_traits>

#include "vbg_internal.cuh"
#include "vbg_args.cuh"

namespace vbg {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;

template <typename T> struct VT;
template <> struct VT<double> { using raw = double2; static constexpr int E = 2; };
template <> struct VT<float> { using raw = float4; static constexpr int E = 4; };
template <> struct VT<cplx> { using raw = double2; static constexpr int E = 1; };

template <typename T>
struct Vec {
  T v[VT<T>::E];
};

template <typename T>
__device__ __forceinline__ Vec<T> load_vec(const T* base, int64_t vidx) {
  typename VT<T>::raw r = reinterpret_cast<const typename VT<T>::raw*>(base)[vidx];
  Vec<T> out;
  memcpy(&out, &r, sizeof(r));
  return out;
}
template <typename T>
__device__ __forceinline__ void store_vec(T* base, int64_t vidx, const Vec<T>& v) {
  typename VT<T>::raw r;
  memcpy(&r, &v, sizeof(r));
  reinterpret_cast<typename VT<T>::raw*>(base)[vidx] = r;
}

// Epilogue for one output element.
template <typename T>
__device__ __forceinline__ T epi_value(const ApplyArgs& a, T sum, int64_t gi) {
  T y = scal_r(a.alpha, sum);
  if (a.beta != 0.0) y = axpy_r(a.beta, static_cast<const T*>(a.X)[gi], y);
  if (a.gamma != 0.0) y = axpy_r(a.gamma, static_cast<const T*>(a.Xprev)[gi], y);
  return y;
}

template <typename T>
__device__ __forceinline__ void epi_finish(const ApplyArgs& a, T y, int64_t gi, double& d0, double& d1) {
  if (a.want_dots) {
    const T xd = a.dotw ? static_cast<const T*>(a.dotw)[gi] : static_cast<const T*>(a.X)[gi];
    d0 += re_dot(xd, y);
    d1 += re_dot(y, y);
  }
  if (a.acc) {
    T* ac = static_cast<T*>(a.acc);
    ac[gi] = cmad(a.cre, a.cim, y, ac[gi]);
  }
}

// ------------------------------------------------------------ vector rows
// Sums the G = 32 / R lane groups' partial rows of one block row and runs the
// epilogue on its R outputs.
template <typename T, int R>
__device__ __forceinline__ void vec_row_finish(const ApplyArgs& a, int row, int lane, T acc, T* wred, double& d0,
                                               double& d1) {
  constexpr int G = 32 / R;
  wred[lane] = acc;
  __syncwarp();
  if (lane < R) {
    T sum = wred[lane];
#pragma unroll
    for (int b = 1; b < G; ++b) sum = add_s(sum, wred[lane + b * R]);
    const int64_t gi = a.scal_off[row] + lane;
    const T y = epi_value(a, sum, gi);
    static_cast<T*>(a.Y)[gi] = y;
    epi_finish(a, y, gi, d0, d1);
  }
  __syncwarp();
}

// Lane l handles block (l / R) of each chunk of G = 32 / R blocks and the
// block row (l % R) inside it.
template <typename T, int R, bool ADJ>
__device__ __forceinline__ void vec_row(const ApplyArgs& a, const T* __restrict__ vals, int row, int lane,
                                        T* wred, double& d0, double& d1) {
  constexpr int G = 32 / R;
  const int bl = lane / R;
  const int o = lane - bl * R;
  const int e0 = a.ptr[row], e1 = a.ptr[row + 1];
  const T* __restrict__ x = static_cast<const T*>(a.X);
  T acc = zero_s<T>();
  if (bl < G) {
    for (int e = e0 + bl; e < e1; e += G) {
      const int src = a.ent_src[e];
      const int s = ADJ ? a.ent_slot[e] : e;
      const int inner = a.bsz[src];
      const T* xp = x + a.scal_off[src];
      const T* ap = vals + a.blk_off[s] + (ADJ ? o : o * inner);
#pragma unroll 4
      for (int q = 0; q < inner; ++q) {
        T av = ap[ADJ ? q * R : q];
        if (ADJ) av = conj_s(av);
        acc = fma_s(av, xp[q], acc);
      }
    }
  }
  vec_row_finish<T, R>(a, row, lane, acc, wred, d0, d1);
}

// Rows wider than 8 (outputs of one block row, or of one block column for
// the adjoint), a warp per row: lane l = 8 rs + qs.  Forward, lane (rs, qs)
// takes rows 4 v + rs and columns qs (mod 8) of every block, so the eight qs
// lanes read a row's values side by side; the adjoint, where the outputs run
// along a block's rows, takes outputs 8 v + qs and reads rows rs (mod 4).
// Each X element is loaded once per lane for up to 32 outputs, and the eight
// value loads of a round are independent.  What bounds it is the stream of
// values; one lane per output row, as this was before, read a value per lane
// at a stride of a whole block row (4000 rows of 9-20 complex, 168 MB:
// forward 86 us, adjoint 166 us; the two together 250 us, now 126).
// Entries sub, sub + split, ... of the row; returns this lane's output
// o0 + lane's partial sum (forward: outputs permuted, see wide_out).
template <bool ADJ>
__device__ __forceinline__ int wide_out(int lane) {
  return ADJ ? lane : 4 * (lane & 7) + (lane >> 3);
}

template <typename T, bool ADJ>
__device__ __forceinline__ T vec_wide_sum(const ApplyArgs& a, const T* __restrict__ vals, int e0, int e1, int r,
                                          int o0, int lane, int sub, int split) {
  const T* __restrict__ x = static_cast<const T*>(a.X);
  const int qs = lane & 7, rs = lane >> 3;
  constexpr int V = ADJ ? 4 : 8;
  T acc[V];
#pragma unroll
  for (int v = 0; v < V; ++v) acc[v] = zero_s<T>();
  for (int base = e0 + sub; base < e1; base += 32 * split) {
    const int cnt = min(32, (e1 - base + split - 1) / split);
    long long xo = 0, vo = 0;
    int in = 0;
    if (lane < cnt) {
      const int e = base + lane * split;
      if (!ADJ && a.slot_meta) {
        const int2 mt = __ldg(a.slot_meta + e);
        xo = mt.x;
        in = mt.y & 0xff;
        vo = __ldg(a.blk_off + e);
      } else {
        const int src = __ldg(a.ent_src + e);
        xo = a.scal_off[src];
        in = a.bsz[src];
        vo = a.blk_off[ADJ ? __ldg(a.ent_slot + e) : e];
      }
    }
    for (int j = 0; j < cnt; ++j) {
      const T* __restrict__ xp = x + __shfl_sync(0xffffffffu, xo, j);
      const T* __restrict__ vp = vals + __shfl_sync(0xffffffffu, vo, j);
      const int inner = __shfl_sync(0xffffffffu, in, j);
      if constexpr (!ADJ) {
        for (int q0 = 0; q0 < inner; q0 += 8) {
          const int q = q0 + qs;
          const bool kv = q < inner;
          const T xv = kv ? xp[q] : zero_s<T>();
          T av[V];
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const int o = o0 + 4 * v + rs;
            av[v] = kv && o < r ? vp[(int64_t)o * inner + q] : zero_s<T>();
          }
#pragma unroll
          for (int v = 0; v < V; ++v) acc[v] = fma_s(av[v], xv, acc[v]);
        }
      } else {
        for (int q0 = 0; q0 < inner; q0 += 8) {
          T av[2][V], xv[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int q = q0 + 4 * h + rs;
            const bool kv = q < inner;
            xv[h] = kv ? xp[q] : zero_s<T>();
#pragma unroll
            for (int v = 0; v < V; ++v) {
              const int o = o0 + 8 * v + qs;
              av[h][v] = kv && o < r ? vp[(int64_t)q * r + o] : zero_s<T>();
            }
          }
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int v = 0; v < V; ++v) acc[v] = fma_s(conj_s(av[h][v]), xv[h], acc[v]);
        }
      }
    }
  }
  // the lanes of an output meet by butterflies; each lane keeps its own output
  T mine = zero_s<T>();
#pragma unroll
  for (int v = 0; v < V; ++v) {
    if (o0 + v * (32 / V) >= r) break;
#pragma unroll
    for (int off = ADJ ? 8 : 1; off < (ADJ ? 32 : 8); off <<= 1) acc[v] = add_s(acc[v], shfl_xor_s(acc[v], off));
    if ((ADJ ? rs : qs) == v) mine = acc[v];
  }
  return mine;
}

template <typename T>
__device__ __forceinline__ void vec_wide_finish(const ApplyArgs& a, T sum, int64_t gi, double& d0, double& d1) {
  const T y = epi_value(a, sum, gi);
  static_cast<T*>(a.Y)[gi] = y;
  epi_finish(a, y, gi, d0, d1);
}

template <typename T, bool ADJ>
__device__ void vec_row_wide(const ApplyArgs& a, const T* __restrict__ vals, int row, int lane, double& d0,
                             double& d1) {
  const int r = a.bsz[row];
  const int e0 = a.ptr[row], e1 = a.ptr[row + 1];
  if constexpr (std::is_same<T, float>::value && !ADJ) {
    // a lane per output row: at 4 bytes a value a row's lines stay in L1 from
    // one column to the next, and the lanes along the rows were slower (5000
    // rows of sizes 2-12: 32 us a step against 17, of 9-16: 29 against 24)
    const T* __restrict__ x = static_cast<const T*>(a.X);
    for (int o = lane; o < r; o += 32) {
      T acc = zero_s<T>();
      for (int e = e0; e < e1; ++e) {
        const int src = a.ent_src[e], inner = a.bsz[src];
        const T* __restrict__ xp = x + a.scal_off[src];
        const T* __restrict__ ap = vals + a.blk_off[e] + (int64_t)o * inner;
        for (int q = 0; q < inner; ++q) acc = fma_s(ap[q], xp[q], acc);
      }
      vec_wide_finish(a, acc, a.scal_off[row] + o, d0, d1);
    }
    return;
  }
  for (int o0 = 0; o0 < r; o0 += 32) {
    const T sum = vec_wide_sum<T, ADJ>(a, vals, e0, e1, r, o0, lane, 0, 1);
    const int o = o0 + wide_out<ADJ>(lane);
    if (o < r) vec_wide_finish(a, sum, a.scal_off[row] + o, d0, d1);
  }
}

// Forward vector rows from the per-slot records: lane j of the warp loads
// slot j's {first X row, shape} and value offset for up to 32 of the row's
// blocks at once, so a block costs one level of dependent loads instead of
// three (column index, then the column's offset and size, then values and X).
// The blocks are then handed out by shuffles, G = 32 / R at a time, lane l
// taking block (l / R) and its row (l % R); the value and X loads of two such
// rounds are issued before their multiply-adds.  The records hold 32-bit X
// offsets and 8-bit block sizes, so the caller takes this path for N < 2^31
// and blocks of at most 255 only.  CH columns of a block row are loaded
// before their multiply-adds (fewer for complex values, whose staging
// registers would otherwise set the kernel's occupancy).
template <typename T, int R, int CH = 8>
__device__ __forceinline__ void vec_row_meta(const ApplyArgs& a, const T* __restrict__ vals, int row, int lane,
                                             T* wred, double& d0, double& d1) {
  constexpr int G = 32 / R;
  const int bl = lane / R;
  const int o = lane - bl * R;
  const int e0 = a.ptr[row], e1 = a.ptr[row + 1];
  const T* __restrict__ x = static_cast<const T*>(a.X);
  T acc = zero_s<T>();
  for (int base = e0; base < e1; base += 32) {
    const int cnt = min(32, e1 - base);
    int xo = 0, cs = 0;
    long long vo = 0;
    if (lane < cnt) {
      const int2 mt = __ldg(a.slot_meta + base + lane);
      xo = mt.x;
      cs = mt.y & 0xff;
      vo = __ldg(a.blk_off + base + lane);
    }
    for (int j0 = 0; j0 < cnt; j0 += G) {
      const int j = j0 + bl;
      const int jx = __shfl_sync(0xffffffffu, xo, j & 31);
      const int jc = __shfl_sync(0xffffffffu, cs, j & 31);
      const long long jv = __shfl_sync(0xffffffffu, vo, j & 31);
      if (bl < G && j < cnt) {
        const T* __restrict__ ap = vals + jv + (long long)o * jc;
        const T* __restrict__ xp = x + (unsigned)jx;
        for (int q0 = 0; q0 < jc; q0 += CH) {  // block columns wider than CH take several rounds
          T av[CH], xv[CH];
#pragma unroll
          for (int q = 0; q < CH; ++q) {
            av[q] = q0 + q < jc ? ap[q0 + q] : zero_s<T>();
            xv[q] = q0 + q < jc ? xp[q0 + q] : zero_s<T>();
          }
#pragma unroll
          for (int q = 0; q < CH; ++q) acc = fma_s(av[q], xv[q], acc);
        }
      }
    }
  }
  vec_row_finish<T, R>(a, row, lane, acc, wred, d0, d1);
}

template <typename T, int CH = 8>
__device__ __forceinline__ bool dispatch_vec_row_meta(const ApplyArgs& a, const T* __restrict__ vals, int row,
                                                      int lane, T* wred, double& d0, double& d1) {
  switch (a.bsz[row]) {
    case 1: vec_row_meta<T, 1, CH>(a, vals, row, lane, wred, d0, d1); return true;
    case 2: vec_row_meta<T, 2, CH>(a, vals, row, lane, wred, d0, d1); return true;
    case 3: vec_row_meta<T, 3, CH>(a, vals, row, lane, wred, d0, d1); return true;
    case 4: vec_row_meta<T, 4, CH>(a, vals, row, lane, wred, d0, d1); return true;
    case 5: vec_row_meta<T, 5, CH>(a, vals, row, lane, wred, d0, d1); return true;
    case 6: vec_row_meta<T, 6, CH>(a, vals, row, lane, wred, d0, d1); return true;
    case 7: vec_row_meta<T, 7, CH>(a, vals, row, lane, wred, d0, d1); return true;
    case 8: vec_row_meta<T, 8, CH>(a, vals, row, lane, wred, d0, d1); return true;
    default: return false;
  }
}

// ------------------------------------------------------- multivector rows
// lanes [grp*LPR, grp*LPR + LPR) cover 16-byte vectors of the padded X row;
// the G lane groups take every G-th block of the row and are summed by
// butterfly shuffles at the end.  RM output rows per pass (R <= 8 exact).
template <typename T, int RM, bool ADJ>
__device__ __forceinline__ void mv_rows(const ApplyArgs& a, const T* __restrict__ vals, int row, int lane, int lpr,
                                        int G, int o0, int rcount, int rfull, double& d0, double& d1) {
  constexpr int E = VT<T>::E;
  const int grp = lane / lpr;
  const int vl = lane - grp * lpr;
  const int nvec = a.ld / E;
  const int e0 = a.ptr[row], e1 = a.ptr[row + 1];
  const T* __restrict__ X = static_cast<const T*>(a.X);
  for (int v0 = 0; v0 < nvec; v0 += lpr) {
    const int vi = v0 + vl;
    const bool valid = grp < G && vi < nvec;
    Vec<T> acc[RM];
#pragma unroll
    for (int o = 0; o < RM; ++o)
#pragma unroll
      for (int u = 0; u < E; ++u) acc[o].v[u] = zero_s<T>();
    if (valid) {
      for (int e = e0 + grp; e < e1; e += G) {
        const int src = a.ent_src[e];
        const int inner = a.bsz[src];
        const int64_t xrow0 = a.scal_off[src];
        const T* ab = vals + a.blk_off[ADJ ? a.ent_slot[e] : e];
        for (int q = 0; q < inner; ++q) {
          const Vec<T> xv = load_vec(X, (xrow0 + q) * nvec + vi);
#pragma unroll
          for (int o = 0; o < RM; ++o) {
            if (o < rcount) {
              T av = ab[ADJ ? (int64_t)q * rfull + o0 + o : (int64_t)(o0 + o) * inner + q];
              if (ADJ) av = conj_s(av);
#pragma unroll
              for (int u = 0; u < E; ++u) acc[o].v[u] = fma_s(av, xv.v[u], acc[o].v[u]);
            }
          }
        }
      }
    }
    if (G > 1) {
      for (int off = lpr; off < G * lpr; off <<= 1) {
#pragma unroll
        for (int o = 0; o < RM; ++o)
#pragma unroll
          for (int u = 0; u < E; ++u) acc[o].v[u] = add_s(acc[o].v[u], shfl_xor_s(acc[o].v[u], off));
      }
    }
    if (grp == 0 && vi < nvec) {
#pragma unroll
      for (int o = 0; o < RM; ++o) {
        if (o < rcount) {
          const int64_t grow = a.scal_off[row] + o0 + o;
          const int64_t vidx = grow * nvec + vi;
          Vec<T> y;
          if (a.beta == 0.0 && a.gamma == 0.0 && !a.want_dots && !a.acc) {
#pragma unroll
            for (int u = 0; u < E; ++u) y.v[u] = scal_r(a.alpha, acc[o].v[u]);
          } else {
            Vec<T> xs, xp, xd, ac;
            if (a.beta != 0.0 || (a.want_dots && !a.dotw)) xs = load_vec(X, vidx);
            if (a.gamma != 0.0) xp = load_vec(static_cast<const T*>(a.Xprev), vidx);
            if (a.want_dots) xd = a.dotw ? load_vec(static_cast<const T*>(a.dotw), vidx) : xs;
            if (a.acc) ac = load_vec(static_cast<const T*>(a.acc), vidx);
#pragma unroll
            for (int u = 0; u < E; ++u) {
              T yy = scal_r(a.alpha, acc[o].v[u]);
              if (a.beta != 0.0) yy = axpy_r(a.beta, xs.v[u], yy);
              if (a.gamma != 0.0) yy = axpy_r(a.gamma, xp.v[u], yy);
              y.v[u] = yy;
              if (a.want_dots) {
                d0 += re_dot(xd.v[u], yy);
                d1 += re_dot(yy, yy);
              }
              if (a.acc) ac.v[u] = cmad(a.cre, a.cim, yy, ac.v[u]);
            }
            if (a.acc) store_vec(static_cast<T*>(a.acc), vidx, ac);
          }
          store_vec(static_cast<T*>(a.Y), vidx, y);
        }
      }
    }
  }
}

template <typename T, bool ADJ>
__device__ __forceinline__ void dispatch_vec_row(const ApplyArgs& a, const T* __restrict__ vals, int row, int lane,
                                                 T* wred, double& d0, double& d1) {
  switch (a.bsz[row]) {
    case 1: vec_row<T, 1, ADJ>(a, vals, row, lane, wred, d0, d1); break;
    case 2: vec_row<T, 2, ADJ>(a, vals, row, lane, wred, d0, d1); break;
    case 3: vec_row<T, 3, ADJ>(a, vals, row, lane, wred, d0, d1); break;
    case 4: vec_row<T, 4, ADJ>(a, vals, row, lane, wred, d0, d1); break;
    case 5: vec_row<T, 5, ADJ>(a, vals, row, lane, wred, d0, d1); break;
    case 6: vec_row<T, 6, ADJ>(a, vals, row, lane, wred, d0, d1); break;
    case 7: vec_row<T, 7, ADJ>(a, vals, row, lane, wred, d0, d1); break;
    case 8: vec_row<T, 8, ADJ>(a, vals, row, lane, wred, d0, d1); break;
    default: vec_row_wide<T, ADJ>(a, vals, row, lane, d0, d1); break;
  }
}

// This CTA's share of [p, p + bytes) prefetched into L2 by bulk prefetches
// (16-byte units, 64 KiB per instruction; a tail under 16 bytes is left to
// the loads).  p is 16-byte aligned.
__device__ __forceinline__ void prefetch_share_l2(const void* p, long long bytes) {
  const long long units = bytes >> 4;
  const long long per = (units + gridDim.x - 1) / gridDim.x;
  long long u = per * blockIdx.x;
  const long long u1 = min(units, u + per);
  const char* c = static_cast<const char*>(p);
  for (; u < u1; u += 4096) {
    const unsigned n = static_cast<unsigned>(min(u1 - u, 4096ll) << 4);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(c + (u << 4)), "r"(n) : "memory");
  }
}

// Plain vectors: one launch over all rows, block size dispatched per warp.
// For a working set that fits L2 every CTA first asks L2 for its share of
// the values, the slot records and X, so the warps' dependent loads (row
// range, then records, then values and X) meet L2 instead of HBM latency.
template <typename T, bool ADJ>
__global__ void __launch_bounds__(kThreads) apply_vec_kernel(ApplyArgs a, const T* __restrict__ vals, int part_base,
                                                             int total) {
  __shared__ T wred_all[kThreads];
  if (a.npf && threadIdx.x == 0)
    for (int r = 0; r < a.npf; ++r) prefetch_share_l2(a.pf_ptr[r], a.pf_bytes[r]);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T* wred = wred_all + warp * 32;
  double d0 = 0.0, d1 = 0.0;
  for (int w = blockIdx.x * kWarps + warp; w < a.n_rows; w += gridDim.x * kWarps) {
    // with the slot records, rows in their own order (one warp per row:
    // grouping by size buys nothing here and costs a dependent load)
    const bool meta = !ADJ && a.slot_meta;
    if (meta && dispatch_vec_row_meta<T>(a, vals, w, lane, wred, d0, d1)) continue;
    const int row = (meta || !a.order) ? w : a.order[w];
    dispatch_vec_row<T, ADJ>(a, vals, row, lane, wred, d0, d1);
  }
  if (a.want_dots) grid_reduce2(d0, d1, a.partials, a.counter, a.dots_out, part_base, total);
}

// Vectors on matrices whose blocks are all over 8: a kernel of its own (its
// registers are not set by the narrow rows' paths), `split` warps of the CTA
// per block row when there are too few rows to fill the SMs.
template <typename T, bool ADJ>
__global__ void __launch_bounds__(kThreads, 2) apply_vec_wide_kernel(ApplyArgs a, const T* __restrict__ vals,
                                                                     int max_bs, int split, int part_base,
                                                                     int total) {
  __shared__ T red[kThreads];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per_cta = kWarps / split, sub = warp % split;
  double d0 = 0.0, d1 = 0.0;
  for (int wb = blockIdx.x * per_cta; wb < a.n_rows; wb += gridDim.x * per_cta) {  // CTA-uniform
    const int row = wb + warp / split;
    const bool on = row < a.n_rows;
    const int r = on ? a.bsz[row] : 0;
    const int e0 = on ? a.ptr[row] : 0, e1 = on ? a.ptr[row + 1] : 0;
    // the CTA's rows may differ in size: every warp takes the barriers of
    // the matrix's largest block
    for (int o0 = 0; o0 < max_bs; o0 += 32) {
      T sum = zero_s<T>();
      if (o0 < r) sum = vec_wide_sum<T, ADJ>(a, vals, e0, e1, r, o0, lane, sub, split);
      if (split > 1) {
        red[threadIdx.x] = sum;
        __syncthreads();
        if (sub == 0)
          for (int w = 1; w < split; ++w) sum = add_s(sum, red[threadIdx.x + 32 * w]);
        __syncthreads();
      }
      const int o = o0 + wide_out<ADJ>(lane);
      if (sub == 0 && o < r) vec_wide_finish(a, sum, a.scal_off[row] + o, d0, d1);
    }
  }
  if (a.want_dots) grid_reduce2(d0, d1, a.partials, a.counter, a.dots_out, part_base, total);
}

// Multivectors the staged applies do not take, FP32 and (lane_rows) small FP64
// and complex blocks: one launch per block-size class; rows [w0, w1) of the
// class-ordered row list all have block size R (R == 0: any size > 8).
template <typename T, int R, bool ADJ>
__global__ void __launch_bounds__(kThreads) apply_mv_kernel(ApplyArgs a, const T* __restrict__ vals, int w0, int w1,
                                                            int lpr, int G, int part_base, int total) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double d0 = 0.0, d1 = 0.0;
  for (int w = w0 + blockIdx.x * kWarps + warp; w < w1; w += gridDim.x * kWarps) {
    const int row = a.order[w];
    double r0 = 0.0, r1 = 0.0;
    if constexpr (R > 0) {
      mv_rows<T, R, ADJ>(a, vals, row, lane, lpr, G, 0, R, R, r0, r1);
    } else {
      const int r = a.bsz[row];
      for (int o0 = 0; o0 < r; o0 += 8)
        mv_rows<T, 8, ADJ>(a, vals, row, lane, lpr, G, o0, min(8, r - o0), r, r0, r1);
    }
    if (a.want_dots) {
      if (a.row_dots) {
        write_row_dots(a.row_dots, row, r0, r1);
      } else {
        d0 += r0;
        d1 += r1;
      }
    }
  }
  if (a.want_dots && !a.row_dots) grid_reduce2(d0, d1, a.partials, a.counter, a.dots_out, part_base, total);
}

// ------------------------------------------------ pipelined multivector apply
#include "vbg_pipe.cuh"
#include "vbg_tile.cuh"
#include "vbg_dtile.cuh"
#include "vbg_chain.cuh"
#include "vbg_resident.cuh"
// Forward vectors on matrices whose blocks are all at most 8 x 8, every row
// from the slot records (vec_row_meta): a kernel of its own so that its
// register budget is not set by the general row paths: with 36 warps per
// SM every block row of a 5000-row matrix has its warp resident at once
// instead of some warps taking a second row after the first.  FP64 rows
// stage six columns at a time and complex rows four (kMetaCh), which keeps
// them inside this budget without spills.
constexpr int kMetaWarps = 4;  // warps of a record-driven vector CTA
template <typename T>
constexpr int kMetaCtas = 9;  // CTAs per SM
template <typename T>
constexpr int kMetaCh = std::is_same<T, cplx>::value ? 4 : std::is_same<T, double>::value ? 6 : 8;
template <typename T>
__global__ void __launch_bounds__(kMetaWarps * 32, kMetaCtas<T>) apply_vec_meta_kernel(ApplyArgs a,
                                                                                       const T* __restrict__ vals,
                                                                                       int part_base, int total) {
  __shared__ T wred_all[kMetaWarps * 32];
  if (a.npf && threadIdx.x == 0)
    for (int r = 0; r < a.npf; ++r) prefetch_share_l2(a.pf_ptr[r], a.pf_bytes[r]);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T* wred = wred_all + warp * 32;
  double d0 = 0.0, d1 = 0.0;
  for (int w = blockIdx.x * kMetaWarps + warp; w < a.n_rows; w += gridDim.x * kMetaWarps)
    (void)dispatch_vec_row_meta<T, kMetaCh<T>>(a, vals, w, lane, wred, d0, d1);
  if (a.want_dots) grid_reduce2(d0, d1, a.partials, a.counter, a.dots_out, part_base, total);
}

template <typename T>
static int vec_meta_max_grid() {
  static int cached[kMaxDevices] = {};
  const int dev = current_device();
  if (!cached[dev]) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, apply_vec_meta_kernel<T>, kMetaWarps * 32, 0) !=
            cudaSuccess ||
        per_sm < 1)
      per_sm = 1;
    cached[dev] = per_sm * sm_count();
  }
  return cached[dev];
}

// Adjoint vectors on matrices whose blocks are all at most 8 x 8: lane
// l = 8 rs + qs takes output qs and rows rs and 4 + rs of every block of its
// block column, as for the wide blocks, so a warp reads a block's values in
// two loads of up to 256 consecutive bytes and each X element once, several
// blocks in flight; a lane per (block, output) read them at a stride of a
// block row.  5000 rows of 4-8, 13 blocks a column: 14.4 us, now 10.3.
// `split` warps of the CTA share a block column when there are too few to
// fill the SMs (row_split).  (Forward, the record-driven kernel's lanes
// already run along the values: 10.2 us against 12.3 this way.)
constexpr int kVecAdjWarps = 4;
// Blocks in flight per warp, CTAs per SM (36 warps for real values, 28 for
// complex ones: what their registers allow without spills).
template <typename T>
constexpr int kVecAdjBlocks = std::is_same<T, cplx>::value ? 2 : 3;
template <typename T>
constexpr int kVecAdjCtas = std::is_same<T, cplx>::value ? 7 : 9;

template <typename T>
__device__ __forceinline__ T vec_adj_sum(const ApplyArgs& a, const T* __restrict__ vals, int e0, int e1, int r,
                                         int lane, int sub, int split) {
  const T* __restrict__ x = static_cast<const T*>(a.X);
  const int qs = lane & 7, rs = lane >> 3;
  constexpr int U = kVecAdjBlocks<T>;
  T acc = zero_s<T>();
  for (int base = e0 + sub; base < e1; base += 32 * split) {
    const int cnt = min(32, (e1 - base + split - 1) / split);
    int xo = 0, in = 0;
    long long vo = 0;
    if (lane < cnt) {
      const int e = base + lane * split;
      const int src = __ldg(a.ent_src + e);
      xo = (int)a.scal_off[src];
      in = a.bsz[src];
      vo = a.blk_off[__ldg(a.ent_slot + e)];
    }
    for (int j = 0; j < cnt; j += U) {
      T x0[U], x1[U], v0[U], v1[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const T* __restrict__ xp = x + (unsigned)__shfl_sync(0xffffffffu, xo, (j + u) & 31);
        const T* __restrict__ vp = vals + __shfl_sync(0xffffffffu, vo, (j + u) & 31);
        // past the last block: inner size 0
        const int n = j + u < cnt ? __shfl_sync(0xffffffffu, in, (j + u) & 31) : 0;
        const bool k0 = rs < n, k1 = rs + 4 < n;
        x0[u] = k0 ? xp[rs] : zero_s<T>();
        x1[u] = k1 ? xp[rs + 4] : zero_s<T>();
        v0[u] = k0 && qs < r ? vp[rs * r + qs] : zero_s<T>();
        v1[u] = k1 && qs < r ? vp[(rs + 4) * r + qs] : zero_s<T>();
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        acc = fma_s(conj_s(v0[u]), x0[u], acc);
        acc = fma_s(conj_s(v1[u]), x1[u], acc);
      }
    }
  }
  acc = add_s(acc, shfl_xor_s(acc, 8));
  return add_s(acc, shfl_xor_s(acc, 16));
}

template <typename T>
__global__ void __launch_bounds__(kVecAdjWarps * 32, kVecAdjCtas<T>)
    apply_vec_adj_kernel(ApplyArgs a, const T* __restrict__ vals, int split, int part_base, int total) {
  __shared__ T red[kVecAdjWarps * 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per_cta = kVecAdjWarps / split, sub = warp % split;
  double d0 = 0.0, d1 = 0.0;
  for (int wb = blockIdx.x * per_cta; wb < a.n_rows; wb += gridDim.x * per_cta) {  // CTA-uniform
    const int row = wb + warp / split;
    const bool on = row < a.n_rows;
    const int r = on ? a.bsz[row] : 0;
    T sum = vec_adj_sum<T>(a, vals, on ? a.ptr[row] : 0, on ? a.ptr[row + 1] : 0, r, lane, sub, split);
    if (split > 1) {
      red[threadIdx.x] = sum;
      __syncthreads();
      if (sub == 0)
        for (int w = 1; w < split; ++w) sum = add_s(sum, red[threadIdx.x + 32 * w]);
      __syncthreads();
    }
    if (sub == 0 && lane < r) vec_wide_finish(a, sum, a.scal_off[row] + lane, d0, d1);
  }
  if (a.want_dots) grid_reduce2(d0, d1, a.partials, a.counter, a.dots_out, part_base, total);
}

template <typename T>
static int launch_vec_adj(const vbg_matrix* m, const ApplyArgs& a, const T* vals, cudaStream_t s) {
  static int resident[kMaxDevices] = {};
  const int dev = current_device();
  if (!resident[dev]) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, apply_vec_adj_kernel<T>, kVecAdjWarps * 32, 0) !=
            cudaSuccess ||
        per_sm < 1)
      per_sm = 1;
    resident[dev] = per_sm * sm_count();
  }
  const int split = std::min(row_split(m, m->n), kVecAdjWarps), wpc = kVecAdjWarps / split;
  const int grid = std::max(1, std::min((a.n_rows + wpc - 1) / wpc, resident[dev]));
  if (int rc = check_dot_ctas(a, grid)) return rc;
  apply_vec_adj_kernel<T><<<grid, kVecAdjWarps * 32, 0, s>>>(a, vals, split, 0, grid);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

template <typename T, bool ADJ>
static int vec_max_grid() {
  static int cached[kMaxDevices] = {};
  const int dev = current_device();
  if (!cached[dev]) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, apply_vec_kernel<T, ADJ>, kThreads, 0) != cudaSuccess ||
        per_sm < 1)
      per_sm = 1;
    cached[dev] = per_sm * sm_count();
  }
  return cached[dev];
}

template <typename T, bool ADJ>
static int vec_wide_max_grid() {
  static int cached[kMaxDevices] = {};
  const int dev = current_device();
  if (!cached[dev]) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, apply_vec_wide_kernel<T, ADJ>, kThreads, 0) !=
            cudaSuccess ||
        per_sm < 1)
      per_sm = 1;
    cached[dev] = per_sm * sm_count();
  }
  return cached[dev];
}

template <typename T, int R, bool ADJ>
static int mv_max_grid() {
  static int cached[kMaxDevices] = {};
  const int dev = current_device();
  if (!cached[dev]) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, apply_mv_kernel<T, R, ADJ>, kThreads, 0) !=
            cudaSuccess ||
        per_sm < 1)
      per_sm = 1;
    cached[dev] = per_sm * sm_count();
  }
  return cached[dev];
}

// Working sets up to this size are prefetched into L2 by the vector apply.
constexpr long long kVecPrefetchMax = 32ll << 20;

// ------------------------------------------------------ scalar-row vectors
// Forward vectors on blocks of at most 8 x 8 with S consecutive threads per
// scalar output row: thread s of row i takes the blocks s, s + S, ... of
// i's block row -- its own row of each block (contiguous values) against
// the block column's X -- the S partial sums meet by shuffles and the first
// thread runs the epilogue on output i, so the epilogue's loads and stores
// are coalesced.  srow[i] holds i's slot range and its row inside the block,
// so a thread is one dependent load from its block list.  Against a warp per
// block row this issues far fewer instructions per row on small blocks (no
// per-block shuffles, no shared-memory reduction of partial rows).
constexpr int kSrowThreads = 256;
constexpr int kSrowCtas = 5;  // per SM (at most 51 registers)
template <typename T>
constexpr int kSrowCh = std::is_same<T, cplx>::value ? 4 : 8;

// ADJ: the adjoint over the column view -- a thread of output (scalar
// column) j takes the blocks of j's block column, reads the block's column
// (stride: its columns) conjugated against X over the block's rows;
// a.srow, a.slot_meta and a.blk_off then hold the scalar-column records and
// the column view's entry records and value offsets.
template <typename T, int S, bool ADJ = false>
__global__ void __launch_bounds__(kSrowThreads, kSrowCtas) apply_vec_srow_kernel(ApplyArgs a,
                                                                                 const T* __restrict__ vals,
                                                                                 int part_base, int total) {
  constexpr int CH = kSrowCh<T>;
  const T* __restrict__ x = static_cast<const T*>(a.X);
  const int lane = threadIdx.x & 31;
  const int64_t nt = a.n_scal * S;
  const int64_t stride = (int64_t)gridDim.x * kSrowThreads;
  double d0 = 0.0, d1 = 0.0;
  // warp-uniform trip count (the shuffles below need every lane)
  for (int64_t base = (int64_t)blockIdx.x * kSrowThreads + (threadIdx.x - lane); base < nt; base += stride) {
    const int64_t t = base + lane;
    const bool on = t < nt;
    const int64_t i = t / S;
    const int sl = (int)(t & (S - 1));
    T acc = zero_s<T>();
    if (on) {
      const int2 rec = __ldg(a.srow + i);
      const int o = rec.y & 0xff;
      const int e1 = rec.x + (rec.y >> 8);
      for (int e = rec.x + sl; e < e1; e += S) {
        const int2 mt = __ldg(a.slot_meta + e);
        const long long vo = __ldg(a.blk_off + e);
        const int nb = mt.y & 0xff;  // block columns
        const int jc = ADJ ? mt.y >> 8 : nb;  // inner length: the block's rows (ADJ) or columns
        const T* __restrict__ ap = vals + vo + (ADJ ? (long long)o : (long long)o * jc);
        const int st = ADJ ? nb : 1;
        const T* __restrict__ xp = x + (unsigned)mt.x;
        for (int q0 = 0; q0 < jc; q0 += CH) {
          T av[CH], xv[CH];
#pragma unroll
          for (int q = 0; q < CH; ++q) {
            av[q] = q0 + q < jc ? ap[(q0 + q) * st] : zero_s<T>();
            if (ADJ) av[q] = conj_s(av[q]);
            xv[q] = q0 + q < jc ? xp[q0 + q] : zero_s<T>();
          }
#pragma unroll
          for (int q = 0; q < CH; ++q) acc = fma_s(av[q], xv[q], acc);
        }
      }
    }
#pragma unroll
    for (int off = S / 2; off > 0; off >>= 1) acc = add_s(acc, shfl_xor_s(acc, off));
    if (on && sl == 0) {
      const T y = epi_value(a, acc, i);
      static_cast<T*>(a.Y)[i] = y;
      epi_finish(a, y, i, d0, d1);
    }
  }
  if (a.want_dots) grid_reduce2(d0, d1, a.partials, a.counter, a.dots_out, part_base, total);
}

__global__ void build_srow_kernel(int n, const int* __restrict__ ptr, const int* __restrict__ bsz,
                                  const int64_t* __restrict__ scal_off, int2* __restrict__ srow) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const int e0 = ptr[r], cnt = ptr[r + 1] - e0, b = bsz[r];
    const int64_t so = scal_off[r];
    for (int o = 0; o < b; ++o) srow[so + o] = make_int2(e0, (cnt << 8) | o);
  }
}

__global__ void build_scol_kernel(int n, const int* __restrict__ cptr, const int* __restrict__ cslot,
                                  const int* __restrict__ crow, const int* __restrict__ bsz,
                                  const int64_t* __restrict__ scal_off, const int64_t* __restrict__ blk_off,
                                  int2* __restrict__ scol, int2* __restrict__ cmeta, int64_t* __restrict__ cboff) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const int e0 = cptr[j], e1 = cptr[j + 1], c = bsz[j];
    for (int e = e0; e < e1; ++e) {
      const int i = crow[e];
      cmeta[e] = make_int2((int)scal_off[i], (bsz[i] << 8) | c);
      cboff[e] = blk_off[cslot[e]];
    }
    const int64_t so = scal_off[j];
    for (int o = 0; o < c; ++o) scol[so + o] = make_int2(e0, ((e1 - e0) << 8) | o);
  }
}

// Threads per scalar row of the scalar-row vector apply: option
// "apply.vec_lanes" (0 = by size, the default: the fewest of 1, 2, 4, 8 that
// give every SM 1024 threads; 1, 2, 4 or 8 fixed).
static std::atomic<int> g_opt_vec_lanes{0};
// Forward vector kernel: option "apply.vec_kernel" (0 = the autotuner's
// choice, the default; 1 = a warp per block row; 2 = scalar rows).
static std::atomic<int> g_opt_vec_kernel{0};

static int srow_lanes(const vbg_matrix* m) {
  const int opt = g_opt_vec_lanes.load(std::memory_order_relaxed);
  if (opt > 0) return opt;
  const int64_t want = (int64_t)sm_count() * 1024;
  int S = 1;
  while (S < 8 && m->N * S < want) S *= 2;
  return S;
}

// Whether the scalar-row kernel can run this matrix's forward vector applies
// (blocks of at most 8 x 8, the slot records in use, its thread count in
// range).
static bool srow_possible(const vbg_matrix* m) {
  return g_opt_vec_kernel.load(std::memory_order_relaxed) != 1 && m->max_bs <= 8 && m->n > 0 &&
         m->N <= (int64_t)INT32_MAX / 8;
}

// The scalar-row records when the scalar-row apply can run this forward
// vector apply (else nullptr): blocks of at most 8 x 8, the slot records in
// use, fewer than 2^23 slots in every block row; built on first use, never
// while the stream is being captured or when the caller allows no
// allocation.
static int vec_srow(const vbg_matrix* cm, cudaStream_t s, bool allow_alloc, const int2** out) {
  *out = nullptr;
  auto* m = const_cast<vbg_matrix*>(cm);
  if (!srow_possible(m)) return 0;
  if (!m->srow_valid) {
    if (!allow_alloc) return 0;
    cudaStreamCaptureStatus st;
    if (cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) return 0;
    if (m->nnzb >= (1ll << 23)) {
      if (!m->host_struct) return 0;
      for (int r = 0; r < m->n; ++r)
        if (m->h_row_ptr[r + 1] - m->h_row_ptr[r] >= (1 << 23)) return 0;
    }
    int rc = m->srow.ensure(std::max<int64_t>(m->N, 1) * sizeof(int2), s);
    if (rc) return rc;
    const int grid = std::max(1, std::min((m->n + 255) / 256, sm_count() * 8));
    build_srow_kernel<<<grid, 256, 0, s>>>(m->n, m->row_ptr.as<int>(), m->bsz.as<int>(), m->scal_off.as<int64_t>(),
                                           m->srow.as<int2>());
    VBG_CUDA(cudaGetLastError());
    m->srow_valid = true;
  }
  *out = m->srow.as<int2>();
  return 0;
}

// The adjoint's scalar-column records (see vec_srow), after the column view.
static int vec_scol(const vbg_matrix* cm, cudaStream_t s, bool allow_alloc, const int2** out) {
  *out = nullptr;
  auto* m = const_cast<vbg_matrix*>(cm);
  if (!srow_possible(m) || m->nnzb >= (1ll << 23) || m->N >= (int64_t)INT32_MAX) return 0;
  if (!m->scol_valid) {
    if (!allow_alloc) return 0;
    cudaStreamCaptureStatus st;
    if (cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) return 0;
    int rc;
    if ((rc = ensure_csc(m, s))) return rc;
    if ((rc = m->scol.ensure(std::max<int64_t>(m->N, 1) * sizeof(int2), s))) return rc;
    if ((rc = m->csc_meta.ensure(std::max<int64_t>(m->nnzb, 1) * sizeof(int2), s))) return rc;
    if ((rc = m->csc_boff.ensure(std::max<int64_t>(m->nnzb, 1) * sizeof(int64_t), s))) return rc;
    const int grid = std::max(1, std::min((m->n + 255) / 256, sm_count() * 8));
    build_scol_kernel<<<grid, 256, 0, s>>>(m->n, m->csc_ptr.as<int>(), m->csc_slot.as<int>(), m->csc_row.as<int>(),
                                           m->bsz.as<int>(), m->scal_off.as<int64_t>(), m->blk_off.as<int64_t>(),
                                           m->scol.as<int2>(), m->csc_meta.as<int2>(), m->csc_boff.as<int64_t>());
    VBG_CUDA(cudaGetLastError());
    m->scol_valid = true;
  }
  *out = m->scol.as<int2>();
  return 0;
}

template <typename T, int S, bool ADJ>
static int srow_max_grid() {
  static int cached[kMaxDevices] = {};
  const int dev = current_device();
  if (!cached[dev]) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, apply_vec_srow_kernel<T, S, ADJ>, kSrowThreads, 0) !=
            cudaSuccess ||
        per_sm < 1)
      per_sm = 1;
    cached[dev] = per_sm * sm_count();
  }
  return cached[dev];
}

template <typename T, int S, bool ADJ>
static int launch_vec_srow_s(const ApplyArgs& a, const T* vals, cudaStream_t s) {
  const int64_t want = (a.n_scal * S + kSrowThreads - 1) / kSrowThreads;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(want, srow_max_grid<T, S, ADJ>()));
  if (int rc = check_dot_ctas(a, grid)) return rc;
  apply_vec_srow_kernel<T, S, ADJ><<<grid, kSrowThreads, 0, s>>>(a, vals, 0, grid);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

template <typename T, bool ADJ>
static int launch_vec_srow(const vbg_matrix* m, const ApplyArgs& a0, const T* vals, cudaStream_t s) {
  ApplyArgs a = a0;
  if (ADJ) {
    a.slot_meta = m->csc_meta.as<int2>();
    a.blk_off = m->csc_boff.as<int64_t>();
  }
  switch (srow_lanes(m)) {
    case 1: return launch_vec_srow_s<T, 1, ADJ>(a, vals, s);
    case 2: return launch_vec_srow_s<T, 2, ADJ>(a, vals, s);
    case 4: return launch_vec_srow_s<T, 4, ADJ>(a, vals, s);
    default: return launch_vec_srow_s<T, 8, ADJ>(a, vals, s);
  }
}

template <typename T, bool ADJ>
static int launch_vec_t(const vbg_matrix* m, const ApplyArgs& a0, const T* vals, cudaStream_t s) {
  if (a0.srow) return launch_vec_srow<T, ADJ>(m, a0, vals, s);
  // warps per row as the multivector rows take them (row_split); FP32 forward
  // only where rows are split (vec_row_wide)
  const int split = m->min_bs > 8 ? row_split(m, m->n) : 1;
  if (m->min_bs > 8 && (ADJ || !std::is_same<T, float>::value || split > 1)) {
    const int per_cta = kWarps / split;
    const int wgrid = std::max(1, std::min((m->n + per_cta - 1) / per_cta, vec_wide_max_grid<T, ADJ>()));
    if (int rc = check_dot_ctas(a0, wgrid)) return rc;
    apply_vec_wide_kernel<T, ADJ><<<wgrid, kThreads, 0, s>>>(a0, vals, m->max_bs, split, 0, wgrid);
    VBG_CUDA(cudaGetLastError());
    return 0;
  }
  if constexpr (ADJ) {
    if (m->max_bs <= 8 && m->N < (int64_t)INT32_MAX) return launch_vec_adj<T>(m, a0, vals, s);
  }
  const bool meta_only = !ADJ && a0.slot_meta && m->max_bs <= 8;
  const int wpc = meta_only ? kMetaWarps : kWarps;
  int grid = (a0.n_rows + wpc - 1) / wpc;
  grid = std::max(1, std::min(grid, meta_only ? vec_meta_max_grid<T>() : vec_max_grid<T, ADJ>()));
  if (int rc = check_dot_ctas(a0, grid)) return rc;
  ApplyArgs a = a0;
  if (!ADJ && a.slot_meta) {
    const void* ptrs[4] = {vals, a.slot_meta, a.blk_off, a.X};
    const long long bytes[4] = {m->nnz * (long long)sizeof(T), m->nnzb * 8ll, m->nnzb * 8ll,
                                m->N * (long long)sizeof(T)};
    long long total = 0;
    for (int r = 0; r < 4; ++r) total += bytes[r];
    a.npf = 0;
    if (total <= kVecPrefetchMax)
      for (int r = 0; r < 4; ++r)
        if (bytes[r] >= 16 && reinterpret_cast<uintptr_t>(ptrs[r]) % 16 == 0) {
          a.pf_ptr[a.npf] = ptrs[r];
          a.pf_bytes[a.npf++] = bytes[r];
        }
  }
  if (meta_only)
    apply_vec_meta_kernel<T><<<grid, kMetaWarps * 32, 0, s>>>(a, vals, 0, grid);
  else
    apply_vec_kernel<T, ADJ><<<grid, kThreads, 0, s>>>(a, vals, 0, grid);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

template <typename T, int R, bool ADJ>
static int launch_mv_class(const ApplyArgs& a, const T* vals, int w0, int w1, int lpr, int G, int grid, int base,
                           int total, cudaStream_t s) {
  apply_mv_kernel<T, R, ADJ><<<grid, kThreads, 0, s>>>(a, vals, w0, w1, lpr, G, base, total);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

template <typename T, bool ADJ>
static int mv_class_grid(int r, int rows) {
  int cap;
  switch (r) {
    case 1: cap = mv_max_grid<T, 1, ADJ>(); break;
    case 2: cap = mv_max_grid<T, 2, ADJ>(); break;
    case 3: cap = mv_max_grid<T, 3, ADJ>(); break;
    case 4: cap = mv_max_grid<T, 4, ADJ>(); break;
    case 5: cap = mv_max_grid<T, 5, ADJ>(); break;
    case 6: cap = mv_max_grid<T, 6, ADJ>(); break;
    case 7: cap = mv_max_grid<T, 7, ADJ>(); break;
    case 8: cap = mv_max_grid<T, 8, ADJ>(); break;
    default: cap = mv_max_grid<T, 0, ADJ>(); break;
  }
  return std::max(1, std::min((rows + kWarps - 1) / kWarps, cap));
}

template <typename T, bool ADJ>
static int launch_mv_t(const vbg_matrix* m, const ApplyArgs& a, const T* vals, cudaStream_t s) {
  const int nvec = a.ld / VT<T>::E;
  int lpr = nvec >= 32 ? 32 : nvec;
  int G = 32 / lpr;
  if (G > 1 && (lpr & (lpr - 1))) G = 1;  // butterflies need power-of-two groups
  // class segments of the class-ordered row list; rows > 8 share one launch
  std::vector<std::tuple<int, int, int>> segs;  // (R template, w0, w1)
  for (const auto& cs : m->class_segs) {
    const int rt = cs.r <= 8 ? cs.r : 0;
    if (!segs.empty() && rt == 0 && std::get<0>(segs.back()) == 0)
      std::get<2>(segs.back()) = cs.w1;
    else
      segs.emplace_back(rt, cs.w0, cs.w1);
  }
  std::vector<int> grids;
  int total = 0;
  for (auto& sg : segs) {
    grids.push_back(mv_class_grid<T, ADJ>(std::get<0>(sg), std::get<2>(sg) - std::get<1>(sg)));
    total += grids.back();
  }
  if (int rc = check_dot_ctas(a, total)) return rc;
  int base = 0;
  for (size_t i = 0; i < segs.size(); ++i) {
    const int w0 = std::get<1>(segs[i]), w1 = std::get<2>(segs[i]);
    int rc = 0;
    switch (std::get<0>(segs[i])) {
      case 1: rc = launch_mv_class<T, 1, ADJ>(a, vals, w0, w1, lpr, G, grids[i], base, total, s); break;
      case 2: rc = launch_mv_class<T, 2, ADJ>(a, vals, w0, w1, lpr, G, grids[i], base, total, s); break;
      case 3: rc = launch_mv_class<T, 3, ADJ>(a, vals, w0, w1, lpr, G, grids[i], base, total, s); break;
      case 4: rc = launch_mv_class<T, 4, ADJ>(a, vals, w0, w1, lpr, G, grids[i], base, total, s); break;
      case 5: rc = launch_mv_class<T, 5, ADJ>(a, vals, w0, w1, lpr, G, grids[i], base, total, s); break;
      case 6: rc = launch_mv_class<T, 6, ADJ>(a, vals, w0, w1, lpr, G, grids[i], base, total, s); break;
      case 7: rc = launch_mv_class<T, 7, ADJ>(a, vals, w0, w1, lpr, G, grids[i], base, total, s); break;
      case 8: rc = launch_mv_class<T, 8, ADJ>(a, vals, w0, w1, lpr, G, grids[i], base, total, s); break;
      default: rc = launch_mv_class<T, 0, ADJ>(a, vals, w0, w1, lpr, G, grids[i], base, total, s); break;
    }
    if (rc) return rc;
    base += grids[i];
  }
  return 0;
}

// Whether apply_pipe_kernel handles this (forward) multivector apply: blocks
// at most 8 x 8, rows a whole number of warp widths, buffers aligned to the
// per-lane piece.
// Lane groups of apply_pipe_kernel for leading dimension ld: 1 when a row
// of X is at least a warp of pieces wide, 2 or 4 for narrower rows, 0 when
// ld is no whole number of group widths.
template <typename T>
static int pipe_groups(int ld) {
  constexpr int EV = PipeEV<T>::v;
  if (ld % (32 * EV) == 0) return 1;
  if (ld % (16 * EV) == 0) return 2;
  if (ld % (8 * EV) == 0) return 4;
  return 0;
}

template <typename T>
static bool pipe_eligible(const vbg_matrix* m, bool adj, const ApplyArgs& a) {
  constexpr int EV = PipeEV<T>::v;
  constexpr uintptr_t LB = EV * sizeof(T);
  if (adj || a.ld <= 1 || m->max_bs < 1 || m->max_bs > kPipeMaxBs || pipe_groups<T>(a.ld) == 0) return false;
  if (m->N >= (int64_t)INT32_MAX || !a.slot_meta) return false;
  if (reinterpret_cast<uintptr_t>(a.X) % 16) return false;  // bulk copies of X rows
  const void* ptrs[5] = {a.X, a.Xprev, a.Y, a.dotw, a.acc};
  for (const void* p : ptrs)
    if (p && reinterpret_cast<uintptr_t>(p) % LB) return false;
  return true;
}

// X rows per span (and per stage of the ring): at least the largest block.
static int pipe_span_cap(const vbg_matrix* m) { return std::max(m->max_bs, std::min(kPipeSpanCap, kPipeMaxBs)); }

// Grid and dynamic shared memory of apply_pipe_kernel<T, EV, G> for this apply.
template <typename T, int G>
static int pipe_grid_g(const vbg_matrix* m, const ApplyArgs& a, int* grid, size_t* smem) {
  constexpr int EV = PipeEV<T>::v;
  static bool attr_set[kMaxDevices] = {};
  static int per_sm_dev[kMaxDevices][kPipeMaxBs + 1] = {};
  const int dev = current_device();
  int* per_sm = per_sm_dev[dev];
  const int cm = pipe_span_cap(m);
  *smem = kPipeWarps * pipe_warp_bytes<T, G>(cm);
  if (!attr_set[dev]) {
    VBG_CUDA(cudaFuncSetAttribute(apply_pipe_kernel<T, EV, G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(kPipeWarps * pipe_warp_bytes<T, G>(kPipeMaxBs))));
    attr_set[dev] = true;
  }
  if (!per_sm[cm]) {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, apply_pipe_kernel<T, EV, G>, kPipeWarps * 32, *smem) !=
            cudaSuccess ||
        b < 1)
      b = 1;
    per_sm[cm] = b;
  }
  const int nitems = ((a.n_rows + kPipeRows - 1) / kPipeRows) * (a.ld / (PipeShape<G>::L * EV));
  *grid = std::max(1, std::min((nitems + kPipeWarps - 1) / kPipeWarps, per_sm[cm] * sm_count()));
  return 0;
}

template <typename T>
static int pipe_grid(const vbg_matrix* m, const ApplyArgs& a, int* grid, size_t* smem) {
  switch (pipe_groups<T>(a.ld)) {
    case 1: return pipe_grid_g<T, 1>(m, a, grid, smem);
    case 2: return pipe_grid_g<T, 2>(m, a, grid, smem);
    default: return pipe_grid_g<T, 4>(m, a, grid, smem);
  }
}

// Whether this apply runs on apply_pipe_kernel: eligible, and the kernel
// layout of the values exists or may be built here (never while the stream
// is being captured, nor when the caller allows no allocation).
template <typename T>
static bool pipe_use(const vbg_matrix* m, bool adj, const ApplyArgs& a, cudaStream_t s, bool allow_alloc) {
  if (!pipe_eligible<T>(m, adj, a)) return false;
  constexpr bool f32 = std::is_same<T, float>::value;
  if ((f32 ? m->valsK32_valid : m->valsK_valid) && m->span_cap == pipe_span_cap(m)) return true;
  if (!allow_alloc) return false;
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) return false;
  return ensure_kernel_layout(m, f32, s) == 0 && ensure_spans(m, pipe_span_cap(m), s) == 0;
}

template <typename T, int G>
static int launch_pipe_g(const vbg_matrix* m, const ApplyArgs& a0, cudaStream_t s) {
  constexpr int EV = PipeEV<T>::v;
  constexpr bool f32 = std::is_same<T, float>::value;
  int grid = 0;
  size_t smem = 0;
  int rc = pipe_grid_g<T, G>(m, a0, &grid, &smem);
  if (rc) return rc;
  if ((rc = check_dot_ctas(a0, grid))) return rc;
  ApplyArgs a = a0;
  a.koff = (f32 ? m->koff32 : m->koff).as<int64_t>();
  a.spans = m->spans.as<int4>();
  a.span_koff32 = m->span_koff32.as<int64_t>();
  a.row_sptr = m->row_sptr.as<int>();
  const T* vals = (f32 ? m->valsK32 : m->valsK).as<T>();
  apply_pipe_kernel<T, EV, G><<<grid, kPipeWarps * 32, smem, s>>>(a, vals, m->span_cap,
                                                                 a.ld / (PipeShape<G>::L * EV), 0, grid);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

template <typename T>
static int launch_pipe_t(const vbg_matrix* m, const ApplyArgs& a, cudaStream_t s) {
  switch (pipe_groups<T>(a.ld)) {
    case 1: return launch_pipe_g<T, 1>(m, a, s);
    case 2: return launch_pipe_g<T, 2>(m, a, s);
    default: return launch_pipe_g<T, 4>(m, a, s);
  }
}

// Largest tile height (block rows) of the tiled applies at this leading
// dimension and value size: the autotuner's choice, kTileRowsMax before it.
static int tile_cap(const vbg_matrix* m, int ld, int es) {
  auto it = m->tile_rows_cap.find(std::make_pair(ld, es));
  return it == m->tile_rows_cap.end() ? kTileRowsMax : it->second;
}

// Whether the tiled kernel takes its tiles from the plan's work queue (the
// autotuner's choice) or in a fixed stride (default).
static bool tile_queue_on(const vbg_matrix* m, int ld, int es) {
  auto it = m->tile_queue.find(std::make_pair(ld, es));
  return it != m->tile_queue.end() && it->second != 0;
}

// Pieces of 128 bytes of a multivector row with leading dimension ld that
// apply_dtile_kernel<T, NP> takes (1 or 2), else 0.  At four pieces scalar
// multiply-adds with two columns a lane are faster (200 x 200 lattice, FP64, 64
// columns: 410 us a step against 313).  Not for the tensor pipe, which the
// padded steps of blocks of 3 and 5 kept 37 % busy; what else held that form
// back (129 M warp instructions at 16 warps an SM) was not pursued.
template <typename T>
static int dtile_pieces(int ld) {
  const int64_t bytes = (int64_t)ld * (int)sizeof(T);
  return std::is_same<T, float>::value || (bytes != 128 && bytes != 256) ? 0 : (int)(bytes / 128);
}

// Whether this apply runs on a tiled kernel: FP64 and complex on
// apply_dtile_kernel<T, NP> when a row of X is 1 or 2 pieces of 128 bytes,
// else on apply_tile_kernel<T, EV, G> when it is 32 / G lanes of EV scalars
// (FP64 and FP32 at 64 columns, complex at 32; FP32 at 32 and 16 columns
// with EV = 4 and G = 4 and 8 lane groups); the pipelined apply's value
// layout applies, the staged rows (X, Xprev, the dot partner) start on
// 16-byte boundaries, and the matrix has a tile plan for it (built here
// unless capturing or allocation is not allowed) of at least `floor` block rows.
template <typename T, int EV = PipeEV<T>::v, int G = 1>
static bool tile_use(const vbg_matrix* m, bool adj, const ApplyArgs& a, cudaStream_t s, bool allow_alloc,
                     TilePlan** plan, int floor = 0) {
  *plan = nullptr;
  if (dtile_pieces<T>(a.ld) == 0 && a.ld != 32 / G * EV) return false;
  if (!pipe_use<T>(m, adj, a, s, allow_alloc)) return false;
  const void* copied[3] = {a.X, a.Xprev, a.dotw};
  for (const void* p : copied)
    if (p && reinterpret_cast<uintptr_t>(p) % 16) return false;
  const int rb = a.ld * (int)sizeof(T);
  const int cap = tile_cap(m, a.ld, (int)sizeof(T));
  auto it = m->tile_plans.find(std::make_tuple(rb, (int)sizeof(T), cap));
  if (it != m->tile_plans.end()) {
    if (it->second->rows > std::max(floor - 1, 0)) *plan = it->second.get();
    return *plan != nullptr;
  }
  if (!allow_alloc) return false;
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) return false;
  return tile_plan(m, rb, (int)sizeof(T), s, plan, cap, floor) == 0 && *plan != nullptr;
}

// Grid of apply_tile_kernel<T, EV, G> for a plan: the CTAs resident at once,
// at most one per tile.
template <typename T, int EV, int G = 1>
static int tile_grid(TilePlan* plan, int* grid) {
  static bool attr_set[kMaxDevices] = {};
  const int dev = current_device();
  if (!attr_set[dev]) {
    VBG_CUDA(cudaFuncSetAttribute(apply_tile_kernel<T, EV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kTileSmemBudget));
    attr_set[dev] = true;
  }
  if (!plan->grid) {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, apply_tile_kernel<T, EV>, kTileWarps * 32, plan->smem) !=
            cudaSuccess ||
        b < 1)
      b = 1;
    plan->grid = std::max(1, std::min(plan->ntiles, b * sm_count()));
  }
  *grid = plan->grid;
  return 0;
}

template <typename T, int EV = PipeEV<T>::v>
static int launch_tile(const vbg_matrix* m, const ApplyArgs& a0, TilePlan* plan, cudaStream_t s) {
  constexpr bool f32 = std::is_same<T, float>::value;
  int grid = 0;
  int rc = tile_grid<T, EV>(plan, &grid);
  if (rc) return rc;
  if ((rc = check_dot_ctas(a0, grid))) return rc;
  ApplyArgs a = a0;
  a.koff = (f32 ? m->koff32 : m->koff).as<int64_t>();
  a.spans = m->spans.as<int4>();
  a.span_koff32 = m->span_koff32.as<int64_t>();
  a.row_sptr = m->row_sptr.as<int>();
  const T* vals = (f32 ? m->valsK32 : m->valsK).as<T>();
  apply_tile_kernel<T, EV><<<grid, kTileWarps * 32, plan->smem, s>>>(
      a, vals, plan->tiles.as<int4>(), plan->ranges.as<int4>(), plan->qidx.as<unsigned short>(),
      plan->rowinfo.as<int4>(), plan->ntiles, (unsigned)tile_vals_bytes(plan->vcap, (int)sizeof(T)),
      (unsigned)plan->qcap, tile_queue_on(m, a.ld, (int)sizeof(T)) ? plan->queue.as<int>() : nullptr, 0, grid);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

template <int G, int S>
static int launch_narrow_s(const vbg_matrix* m, const ApplyArgs& a, TilePlan* plan, cudaStream_t s) {
  static bool attr_set[kMaxDevices] = {};
  const int dev = current_device();
  if (!attr_set[dev]) {
    VBG_CUDA(cudaFuncSetAttribute(apply_narrow_kernel<G, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kTileSmemBudget32));
    attr_set[dev] = true;
  }
  if (!plan->grid) {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, apply_narrow_kernel<G, S>, kTileWarps * 32, plan->smem) !=
            cudaSuccess ||
        b < 1)
      b = 1;
    plan->grid = std::max(1, std::min(plan->ntiles, b * sm_count()));
  }
  if (int rc = check_dot_ctas(a, plan->grid)) return rc;
  apply_narrow_kernel<G, S><<<plan->grid, kTileWarps * 32, plan->smem, s>>>(
      a, m->valsK32.as<float>(), plan->tiles.as<int4>(), plan->ranges.as<int4>(), plan->qidx.as<unsigned short>(),
      plan->rowinfo.as<int4>(), plan->ntiles, (unsigned)tile_vals_bytes(plan->vcap, 4), (unsigned)plan->qcap,
      (unsigned)narrow_stage_bytes(plan->vcap, plan->qcap, plan->xcap, a.ld * 4), 0, plan->grid);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

template <int G>
static int launch_narrow(const vbg_matrix* m, const ApplyArgs& a, TilePlan* plan, cudaStream_t s) {
  return plan->stages == 2 ? launch_narrow_s<G, 2>(m, a, plan, s) : launch_narrow_s<G, 1>(m, a, plan, s);
}

template <typename T, int NP>
static int launch_dtile_np(const vbg_matrix* m, const ApplyArgs& a, TilePlan* plan, cudaStream_t s) {
  static bool attr_set[kMaxDevices] = {};
  const int dev = current_device();
  if (!attr_set[dev]) {
    VBG_CUDA(cudaFuncSetAttribute(apply_dtile_kernel<T, NP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kTileSmemBudget));
    attr_set[dev] = true;
  }
  if (!plan->grid) {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, apply_dtile_kernel<T, NP>, kTileWarps * 32, plan->smem) !=
            cudaSuccess ||
        b < 1)
      b = 1;
    plan->grid = std::max(1, std::min(plan->ntiles, b * sm_count()));
  }
  if (int rc = check_dot_ctas(a, plan->grid)) return rc;
  apply_dtile_kernel<T, NP><<<plan->grid, kTileWarps * 32, plan->smem, s>>>(
      a, m->valsK.as<T>(), plan->tiles.as<int4>(), plan->xrows.as<int>(), plan->qidx.as<unsigned short>(),
      plan->rowinfo.as<int4>(), plan->ntiles, (unsigned)tile_vals_bytes(plan->vcap, (int)sizeof(T)),
      (unsigned)plan->qcap, 0, plan->grid);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

template <typename T>
static int launch_dtile(const vbg_matrix* m, const ApplyArgs& a, TilePlan* plan, cudaStream_t s) {
  return dtile_pieces<T>(a.ld) == 1 ? launch_dtile_np<T, 1>(m, a, plan, s) : launch_dtile_np<T, 2>(m, a, plan, s);
}

// Whether this apply runs on apply_chain_kernel<T, EV, G>: the tiled
// apply's conditions, and the matrix has a chain plan (built here unless
// capturing or allocation is not allowed).
template <typename T, int EV = PipeEV<T>::v, int G = 1>
static bool chain_use(const vbg_matrix* m, const ApplyArgs& a, cudaStream_t s, bool allow_alloc, ChainPlan** plan) {
  *plan = nullptr;
  if (g_opt_chain.load(std::memory_order_relaxed) == 0) return false;
  if (a.ld != 32 / G * EV || !pipe_use<T>(m, false, a, s, allow_alloc)) return false;
  const void* aligned[3] = {a.X, a.Xprev, a.dotw};
  for (const void* p : aligned)
    if (p && reinterpret_cast<uintptr_t>(p) % 16) return false;
  const int rb = 32 / G * EV * (int)sizeof(T);
  auto it = m->chain_plans.find(std::make_pair(rb, (int)sizeof(T)));
  if (it != m->chain_plans.end()) {
    if (it->second->rows > 0) *plan = it->second.get();
    return *plan != nullptr;
  }
  if (!allow_alloc) return false;
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) return false;
  return chain_plan(m, rb, (int)sizeof(T), s, plan) == 0 && *plan != nullptr;
}

template <typename T, int EV = PipeEV<T>::v, int G = 1>
static int launch_chain(const vbg_matrix* m, const ApplyArgs& a0, ChainPlan* plan, cudaStream_t s) {
  constexpr bool f32 = std::is_same<T, float>::value;
  static bool attr_set[kMaxDevices] = {};
  const int dev = current_device();
  if (!attr_set[dev]) {
    VBG_CUDA(cudaFuncSetAttribute(apply_chain_kernel<T, EV, G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kChainSmemBudget));
    attr_set[dev] = true;
  }
  const int grid = plan->nctas;
  int rc = check_dot_ctas(a0, grid);
  if (rc) return rc;
  ApplyArgs a = a0;
  a.koff = (f32 ? m->koff32 : m->koff).as<int64_t>();
  a.spans = m->spans.as<int4>();
  a.span_koff32 = m->span_koff32.as<int64_t>();
  a.row_sptr = m->row_sptr.as<int>();
  const T* vals = (f32 ? m->valsK32 : m->valsK).as<T>();
  apply_chain_kernel<T, EV, G><<<grid, (plan->rows + 1) * 32, plan->smem, s>>>(
      a, vals, plan->tiles.as<int4>(), plan->loads.as<int4>(), plan->cta_ptr.as<int>(), plan->qidx.as<unsigned short>(),
      plan->rowinfo.as<int4>(), plan->rows, (unsigned)tile_vals_bytes(plan->vcap, (int)sizeof(T)),
      (unsigned)plan->qcap, 0, grid);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

// Builds the tile plan an apply with leading dimension ld would use (before
// a graph capture, which may not build it).  Real matrices only for f32.
static int tile_prepare(const vbg_matrix* m, bool f32, int ld, cudaStream_t s) {
  TilePlan* tp = nullptr;
  ChainPlan* cp = nullptr;
  int rb = 0, es = 0;
  if (f32) {
    if (ld != 16 && ld != 32 && ld != 64) return 0;
    rb = ld * 4;
    es = 4;
  } else {
    es = (int)elem_size(m->dtype);
    if (ld * es != 128 && ld * es != 256 && ld * es != 512) return 0;
    rb = ld * es;
  }
  if (chain_enabled(es)) {
    const int rc = chain_plan(m, rb, es, s, &cp);
    if (rc || cp) return rc;
  }
  return tile_plan(m, rb, es, s, &tp);
}

// Validates arguments and fills the structure part of ApplyArgs.
static int prepare(const vbg_matrix* m, bool adj, int k, int ld, ApplyArgs& a, cudaStream_t s) {
  VBG_CHECK(m, VBG_E_ARG, "null matrix");
  VBG_CHECK(k >= 1 && ld >= k, VBG_E_ARG, "invalid k / ld");
  std::memset(&a, 0, sizeof(a));
  a.n_rows = m->n;
  a.bsz = m->bsz.as<int>();
  a.scal_off = m->scal_off.as<int64_t>();
  a.blk_off = m->blk_off.as<int64_t>();
  a.ld = ld;
  a.alpha = 1.0;
  if (!adj) {
    a.order = m->row_perm.as<int>();
    a.ptr = m->row_ptr.as<int>();
    a.ent_slot = nullptr;
    a.ent_src = m->col_ind.as<int>();
    // the records hold 32-bit X offsets and 8-bit block sizes
    a.slot_meta = (m->N < (int64_t)INT32_MAX && m->max_bs <= 255) ? m->slot_meta.as<int2>() : nullptr;
  } else {
    int rc = ensure_csc(m, s);
    if (rc) return rc;
    a.order = m->row_perm.as<int>();
    a.ptr = m->csc_ptr.as<int>();
    a.ent_slot = m->csc_slot.as<int>();
    a.ent_src = m->csc_row.as<int>();
  }
  return 0;
}

// Whether rows of FP64 or complex values run on apply_mv_kernel instead of the
// tensor-core rows of vbg_mma.cu (the adjoint, and forward what no staged
// apply takes).  A tensor-core step holds 32 values however few a block fills,
// while a warp here spends its lanes on columns and its lane groups on several
// blocks, but the block sizes' launches follow one another.  So: blocks of at
// most 7 values on average, with at least 1200 block rows a size (3600 where
// real columns leave lanes idle: 5000 rows of 1-2, 96 columns 57 / 65, 20000 of
// 1-2 161 / 127), unless the columns leave over a quarter of the lanes idle (nvec 16-byte vectors a row;
// lane groups need a power of two below 32) and the blocks are not single
// values (20000 rows, real 24 columns: sizes 1-2 68 / 66, 1 66 / 50).  And complex adjoints of larger small blocks,
// whose steps are four real ones, on many rows: whole warps of columns, or so
// few that the groups take several blocks (4 columns), or 24.  And rows of at
// most 32 bytes on blocks of up to 17 values, which fill a quarter of a piece
// (30000 rows of 3 and 5, real 2 columns 66 / 58, adjoint 68 / 52, 20000 random
// rows of 3-5 52 / 46 and 58 / 47; but 5000 of 2-4, adjoint at 4, 23 / 31).
// us an apply, tensor-core rows / these (20000 random block rows of 13 blocks,
// adjoint): sizes 1-2 real 8 columns 58 / 29, 64 columns 140 / 89, complex 16
// columns 105 / 55; sizes 2-3 74 real 32 columns / 61; sizes 2-4 (mean 9) real
// 16 columns 60 / 84, complex 64 columns 472 / 443; 60000 banded rows of 1-3,
// complex 128 columns 2890 / 985.  5000 rows of 1-2: real 8 columns 23 / 17,
// 32 columns 23 / 25; 1500 rows of 1-2, real 32 columns 15 / 26.  120000 rows
// of 3 and 5, complex adjoint, 4 / 16 / 64 columns 480 / 624 / 2513 against
// 428 / 800 / 1840.
template <typename T>
static bool lane_rows(const vbg_matrix* m, const ApplyArgs& a, bool adj) {
  constexpr bool cx = std::is_same<T, cplx>::value;
  // (a caller's own dot scratch is sized for the single launch)
  if (std::is_same<T, float>::value || a.max_ctas > 0 || m->nnzb == 0) return false;
  const int nvec = a.ld / VT<T>::E;
  const bool lanes = nvec < 24 ? (nvec & (nvec - 1)) == 0 : 4 * nvec >= 3 * ((nvec + 31) / 32 * 32);
  const double mean = (double)m->nnz / (double)m->nnzb;
  const bool full = nvec < 32 ? (nvec & (nvec - 1)) == 0 : nvec % 32 == 0;
  const int64_t rows = (cx || full ? 1200 : 3600) * (int64_t)m->class_segs.size();
  if (mean <= (lanes ? 7.0 : 1.5) && m->n >= rows) return true;
  if (nvec <= 2 && mean <= 17.0 && m->n >= 8000) return true;
  return cx && adj && mean <= 15.0 && m->n >= 8000 && (nvec <= 4 || nvec == 24 || nvec % 32 == 0);
}

// Forward multivector apply on kernel `which` (VBG_KERNEL_CHAIN, _TILE, _PIPE,
// _ROWS or _LANE_ROWS; -1: the default order -- chained tiles when the
// apply.chain option allows them, tiles, the pipelined kernel, rows).  Returns
// kNotApplicable when `which` cannot run this apply.
constexpr int kNotApplicable = 1;

template <typename T>
static int launch_fwd_mv(const vbg_matrix* m, const ApplyArgs& a, const T* v, cudaStream_t s, bool allow_alloc,
                         int which) {
  const bool any = which < 0;
  TilePlan* tp = nullptr;
  ChainPlan* cp = nullptr;
  if (any ? chain_enabled((int)sizeof(T)) : which == VBG_KERNEL_CHAIN) {
    if (chain_use<T>(m, a, s, allow_alloc, &cp)) return launch_chain<T>(m, a, cp, s);
    if constexpr (std::is_same<T, float>::value) {
      if (chain_use<float, 1>(m, a, s, allow_alloc, &cp)) return launch_chain<float, 1>(m, a, cp, s);
    }
    if constexpr (!std::is_same<T, cplx>::value) {
      if (chain_use<T, 1, 2>(m, a, s, allow_alloc, &cp)) return launch_chain<T, 1, 2>(m, a, cp, s);
    }
    if (!any) return kNotApplicable;
  }
  if (any || which == VBG_KERNEL_TILE) {
    if constexpr (std::is_same<T, float>::value) {
      if (tile_use<float>(m, false, a, s, allow_alloc, &tp)) return launch_tile<float>(m, a, tp, s);
      if (tile_use<float, 4, 4>(m, false, a, s, allow_alloc, &tp)) return launch_narrow<4>(m, a, tp, s);
      if (tile_use<float, 4, 8>(m, false, a, s, allow_alloc, &tp)) return launch_narrow<8>(m, a, tp, s);
    } else {
      if (tile_use<T>(m, false, a, s, allow_alloc, &tp))
        return dtile_pieces<T>(a.ld) ? launch_dtile<T>(m, a, tp, s) : launch_tile<T>(m, a, tp, s);
    }
    if (!any) return kNotApplicable;
  }
  if (any || which == VBG_KERNEL_PIPE) {
    if (pipe_use<T>(m, false, a, s, allow_alloc)) return launch_pipe_t<T>(m, a, s);
    if (!any) return kNotApplicable;
  }
  if constexpr (std::is_same<T, float>::value) return launch_mv_t<float, false>(m, a, v, s);
  if (which == VBG_KERNEL_LANE_ROWS || (any && lane_rows<T>(m, a, false))) return launch_mv_t<T, false>(m, a, v, s);
  return launch_mma(m, false, a, s);
}

// The kernel of a forward multivector apply whose matrix has no tiles (FP64 and
// complex: none of at least 8 block rows).  FP32: the pipelined kernel where it
// applies.  FP64 and
// complex: rows (lane_rows or on the tensor cores), except where the pipelined
// kernel, whose cost goes with the values, is faster.  On rows of a multiple of
// 512 bytes it fills whole warps: blocks of at most 20 values on average, once
// there are rows enough to fill the SMs with its warps of 512 bytes (3000;
// complex, whose products are four times the work, 2500).  On other complex rows: blocks of at most 10
// values, whose products would be four tensor-core steps each.
// us an apply, pipelined / tensor-core rows, random rows of 13 blocks, real 64
// columns: 20000 rows of sizes 2-4 (mean 9) 99 / 130, 3-5 (16) 109 / 151, 4-8
// (36) 412 / 169, 8 (64) 175 / 195 (but a Chebyshev step with its dots 233 / 211); 5000 rows 2-4 36 / 38, 3-5 40 / 40, 8
// 62 / 54; 1500 rows 2-4 32 / 19; 500 rows 2-4 32 / 11, where tiles of 4 rows
// took 13.  Real 128 columns, 20000 rows: 203 / 287, 229 / 311, 560 / 351, 8
// 369 / 345; complex 16 columns 1-2 (2) 77 / 106, 2-4 99 / 107, 3-5 120 / 116,
// 64 columns 1500 rows 2-4 1.16 of the rows', 5000 0.81.  Real 32 columns 90 / 69,
// 115 / 75; rows of no multiple of 512 bytes beyond (48, 80, 96, 112, 144 real
// columns) never were faster pipelined: 20000 rows of 3-5 222 / 136 at 48, 314 /
// 219 at 96, a lattice of 30000 rows 285 / 189 and 388 / 298.
template <typename T>
static int untiled_choice(const vbg_matrix* m, const ApplyArgs& a, cudaStream_t s) {
  constexpr bool f32 = std::is_same<T, float>::value, cx = std::is_same<T, cplx>::value;
  const int64_t bytes = (int64_t)a.ld * (int)sizeof(T);
  const double mean = m->nnzb ? (double)m->nnz / (double)m->nnzb : 0.0;
  bool pipe = f32;
  if (!f32 && bytes % 512 == 0) {
    const bool enough = m->n * (bytes / 512) >= (cx ? 2500 : 3000);
    pipe = enough && mean <= 20.0;
  } else if (cx) {
    pipe = mean <= 10.0;
  }
  if (pipe && pipe_use<T>(m, false, a, s, true)) return VBG_KERNEL_PIPE;
  return lane_rows<T>(m, a, false) ? VBG_KERNEL_LANE_ROWS : VBG_KERNEL_ROWS;
}

// The autotuner: the first forward multivector apply with a given leading
// dimension and precision on a matrix (outside a stream capture, with
// allocation allowed) times each kernel that can run it -- the chained
// tiles, the tiles at three tile heights (at most 16, 12 and 8 block rows,
// each its own plan) with their tiles in a fixed stride or from a work
// queue, the pipelined kernel -- three launches each after one
// untimed launch, on the caller's buffers (the trials write Y and the dots,
// which the real launch then overwrites; they leave the accumulator alone)
// and keeps the fastest kernel for the matrix (vbg_matrix::tuned) and the
// fastest tile height and order for its tiled kernel
// (vbg_matrix::tile_rows_cap, tile_queue).  Option
// "apply.autotune" (default 1) switches it off; an explicit "apply.chain" of
// 0 or 1 takes the kernel choice out of its hands.
static std::atomic<int> g_opt_autotune{1};

template <typename T>
static int autotune_fwd(const vbg_matrix* m, const ApplyArgs& a0, const T* v, cudaStream_t s, int* choice) {
  ApplyArgs a = a0;
  a.acc = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  VBG_CUDA(cudaEventCreate(&e0));
  cudaError_t ce = cudaEventCreate(&e1);
  if (ce != cudaSuccess) {
    cudaEventDestroy(e0);
    return cuda_fail(ce, "cudaEventCreate");
  }
  float best = 0.0f, best_tile = 0.0f;
  int rc = 0, best_cap = 0, best_queue = 0;
  *choice = -1;
  auto* mm = const_cast<vbg_matrix*>(m);
  const auto cap_key = std::make_pair(a.ld, (int)sizeof(T));
  // Kernels that add a row's products in different orders are not timed
  // against each other, so that equal matrices give the same bits in Y whatever
  // the clock said.  (The dots may differ in their last bits: tile height and
  // order, which are timed, decide whose partial sums a CTA holds.)  FP64 and complex values at 512-byte rows: tiles, chained or
  // not (which add alike), where tiles of at least 8 block rows fit, else
  // untiled_choice.  FP32 at 64 columns and up: as timed (the chained, tiled
  // and pipelined forms add alike).
  constexpr bool f32 = std::is_same<T, float>::value;
  std::vector<int> cands = {VBG_KERNEL_CHAIN, VBG_KERNEL_TILE, VBG_KERNEL_PIPE};
  TilePlan* tp = nullptr;
  if constexpr (!f32) {
    const bool tiles = tile_use<T>(m, false, a, s, true, &tp, 8);
    if (tiles) cands = {VBG_KERNEL_CHAIN, VBG_KERNEL_TILE};
    else cands.clear();
  }
  for (int cand : cands) {
    // the tiled kernel once per tile height cap (its own plan each) and per
    // tile order (fixed stride, work queue)
    for (int trial = 0; trial < 6; ++trial) {
      const int cap = trial < 2 ? kTileRowsMax : trial < 4 ? 12 : 8;
      const int queue = trial & 1;
      if (cand != VBG_KERNEL_TILE && trial > 0) break;
      if (cand == VBG_KERNEL_TILE) {
        mm->tile_rows_cap[cap_key] = cap;
        mm->tile_queue[cap_key] = queue;
      }
      rc = launch_fwd_mv<T>(m, a, v, s, true, cand);
      if (rc == kNotApplicable) {
        rc = 0;
        break;
      }
      if (rc) break;
      cudaEventRecord(e0, s);
      for (int k = 0; k < 3 && !rc; ++k) rc = launch_fwd_mv<T>(m, a, v, s, true, cand);
      cudaEventRecord(e1, s);
      if (rc) break;
      if ((ce = cudaEventSynchronize(e1)) != cudaSuccess) {
        rc = cuda_fail(ce, "autotune");
        break;
      }
      float ms = 0.0f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (cand == VBG_KERNEL_TILE && (best_cap == 0 || ms < best_tile)) {
        best_tile = ms;
        best_cap = cap;
        best_queue = queue;
      }
      if (*choice < 0 || ms < best) {
        best = ms;
        *choice = cand;
      }
    }
    if (cand == VBG_KERNEL_TILE) {
      mm->tile_rows_cap[cap_key] = best_cap ? best_cap : kTileRowsMax;
      mm->tile_queue[cap_key] = best_cap ? best_queue : 0;
    }
    if (rc) break;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (!rc && *choice < 0) *choice = untiled_choice<T>(m, a, s);
  return rc;
}

// The kernel a forward multivector apply runs: the tuned choice when the
// autotuner may decide (tuning now if it has not), else -1 (default order).
template <typename T>
static int fwd_choice(const vbg_matrix* m, bool f32, const ApplyArgs& a, const T* v, cudaStream_t s,
                      bool allow_alloc, int* which) {
  *which = -1;
  if (!g_opt_autotune.load() || g_opt_chain.load() != 2) return 0;
  auto* mm = const_cast<vbg_matrix*>(m);
  const auto key = std::make_pair(a.ld, f32 ? 1 : 0);
  auto it = mm->tuned.find(key);
  if (it != mm->tuned.end()) {
    *which = it->second;
    return 0;
  }
  if (!allow_alloc) return 0;
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) return 0;
  int choice = -1;
  int rc = 0;
  const bool narrow = std::is_same<T, float>::value && (a.ld == 16 || a.ld == 32);
  if (dtile_pieces<T>(a.ld) != 0 || narrow) {
    // by rule, not by trials (three plans cost more than they gain: within
    // 5 % on lattices of 1.2k to 11k block rows): the tallest tiles that give
    // every SM two, of at most 8 block rows on smaller matrices
    const auto cap_key = std::make_pair(a.ld, (int)sizeof(T));
    int cap = kTileRowsMax;
    while (cap > 8 && m->n / cap < 2 * sm_count()) cap -= 4;
    mm->tile_rows_cap[cap_key] = cap;
    TilePlan* tp = nullptr;
    bool tiles;
    if constexpr (std::is_same<T, float>::value)
      tiles = tile_use<float, 4, 4>(m, false, a, s, true, &tp) || tile_use<float, 4, 8>(m, false, a, s, true, &tp);
    else
      tiles = tile_use<T>(m, false, a, s, true, &tp, 8);
    // FP32: tiles of any height, which the planner then stages one at a time
    // (us a step at 16 / 32 columns, tiles of 4 rows / pipelined: 5000 rows of
    // random 4-8 blocks 21 / 68 and 27 / 107, of 1-2 16 / 25 and 17 / 32;
    // 20000 of 3-5 58 / 75 and 67 / 95, of 8 89 / 103 and 130 / 145)
    choice = tiles ? VBG_KERNEL_TILE : untiled_choice<T>(m, a, s);
  } else if ((rc = autotune_fwd<T>(m, a, v, s, &choice))) {
    return rc;
  }
  mm->tuned[key] = choice;
  *which = choice;
  return 0;
}

// Dispatch on scalar type / vector-vs-multivector.  `f32` selects the FP32
// shadow values (real matrices only).
// `allow_alloc` false: the call may not allocate device memory (the pipelined
// kernel then runs only if its value layout already exists).
// The forward vector kernel: a warp per block row (VBG_KERNEL_VECTOR) or the
// scalar-row kernel (VBG_KERNEL_SCALAR_ROWS; *srow_out set).  Option
// "apply.vec_kernel" forces one; at 0 the autotuner times both on the first
// vector apply per matrix and precision (three launches each, the
// accumulator off) and keeps the faster (they add in different orders: where
// they are about as fast, the last bits of a vector depend on the clock).  Untuned (autotuner off, no
// allocation allowed, or the stream being captured) complex values take the
// scalar-row kernel, real ones a warp per block row.
template <typename T, bool ADJ = false>
static int vec_kernel(const vbg_matrix* m, bool f32, const ApplyArgs& a0, const T* vals, cudaStream_t s,
                      bool allow_alloc, const int2** srow_out) {
  *srow_out = nullptr;
  const int2* sr = nullptr;
  if (int rc = ADJ ? vec_scol(m, s, allow_alloc, &sr) : vec_srow(m, s, allow_alloc, &sr)) return rc;
  if (!sr) return 0;
  if (g_opt_vec_kernel.load() == 2) {
    *srow_out = sr;
    return 0;
  }
  auto* mm = const_cast<vbg_matrix*>(m);
  // the adjoint's choice under its own key
  const auto key = std::make_pair(1, (f32 ? 1 : 0) + (ADJ ? 2 : 0));
  auto it = mm->tuned.find(key);
  if (it != mm->tuned.end()) {
    if (it->second == VBG_KERNEL_SCALAR_ROWS) *srow_out = sr;
    return 0;
  }
  cudaStreamCaptureStatus st;
  if (!g_opt_autotune.load() || !allow_alloc || cudaStreamIsCapturing(s, &st) != cudaSuccess ||
      st != cudaStreamCaptureStatusNone) {
    if (std::is_same<T, cplx>::value) *srow_out = sr;
    return 0;
  }
  ApplyArgs c[2];
  c[0] = a0;
  c[0].acc = nullptr;
  c[0].srow = nullptr;
  c[1] = c[0];
  c[1].srow = sr;
  c[1].n_scal = m->N;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  VBG_CUDA(cudaEventCreate(&e0));
  cudaError_t ce = cudaEventCreate(&e1);
  if (ce != cudaSuccess) {
    cudaEventDestroy(e0);
    return cuda_fail(ce, "cudaEventCreate");
  }
  float ms[2] = {0.0f, 0.0f};
  int rc = 0;
  for (int k = 0; k < 2 && !rc; ++k) {
    if ((rc = launch_vec_t<T, ADJ>(m, c[k], vals, s))) break;
    cudaEventRecord(e0, s);
    for (int r = 0; r < 3 && !rc; ++r) rc = launch_vec_t<T, ADJ>(m, c[k], vals, s);
    cudaEventRecord(e1, s);
    if (rc) break;
    if ((ce = cudaEventSynchronize(e1)) != cudaSuccess) {
      rc = cuda_fail(ce, "autotune");
      break;
    }
    cudaEventElapsedTime(&ms[k], e0, e1);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc) return rc;
  mm->tuned[key] = ms[1] < ms[0] ? VBG_KERNEL_SCALAR_ROWS : VBG_KERNEL_VECTOR;
  if (ms[1] < ms[0]) *srow_out = sr;
  return 0;
}

static int launch_apply(const vbg_matrix* m, bool adj, bool f32, const ApplyArgs& a_in, cudaStream_t s,
                        bool allow_alloc = true) {
  if (m->n == 0) return 0;
  const bool mv = a_in.ld > 1;
  ApplyArgs a = a_in;
  if (!mv && !adj && a.slot_meta && !a.row_dots) {
    int rc;
    a.n_scal = m->N;
    if (f32) {
      if ((rc = ensure_vals32(m, s))) return rc;
      rc = vec_kernel<float>(m, true, a, m->vals32.as<float>(), s, allow_alloc, &a.srow);
    } else if (m->dtype == VBG_C128) {
      rc = vec_kernel<cplx>(m, false, a, m->vals.as<cplx>(), s, allow_alloc, &a.srow);
    } else {
      rc = vec_kernel<double>(m, false, a, m->vals.as<double>(), s, allow_alloc, &a.srow);
    }
    if (rc) return rc;
  } else if (!mv && adj && !a.row_dots && m->N < (int64_t)INT32_MAX) {
    int rc;
    a.n_scal = m->N;
    if (f32) {
      if ((rc = ensure_vals32(m, s))) return rc;
      rc = vec_kernel<float, true>(m, true, a, m->vals32.as<float>(), s, allow_alloc, &a.srow);
    } else if (m->dtype == VBG_C128) {
      rc = vec_kernel<cplx, true>(m, false, a, m->vals.as<cplx>(), s, allow_alloc, &a.srow);
    } else {
      rc = vec_kernel<double, true>(m, false, a, m->vals.as<double>(), s, allow_alloc, &a.srow);
    }
    if (rc) return rc;
  }
  if (mv) {
    const size_t es = f32 ? 4 : elem_size(m->dtype);
    VBG_CHECK(((size_t)a.ld * es) % 16 == 0, VBG_E_ARG,
              "multivector leading dimension must span a multiple of 16 bytes");
  }
  auto fwd = [&](auto tag, const auto* v) -> int {
    using T = decltype(tag);
    int which = -1;
    int rc = fwd_choice<T>(m, f32, a, v, s, allow_alloc, &which);
    if (rc) return rc;
    rc = launch_fwd_mv<T>(m, a, v, s, allow_alloc, which);
    return rc == kNotApplicable ? launch_fwd_mv<T>(m, a, v, s, allow_alloc, -1) : rc;
  };
  if (f32) {
    int rc = ensure_vals32(m, s);
    if (rc) return rc;
    const float* v = m->vals32.as<float>();
    if (adj) {
      VBG_CHECK(!mv, VBG_E_STATE, "FP32 multivectors have no adjoint apply");
      return launch_vec_t<float, true>(m, a, v, s);
    }
    return mv ? fwd(float{}, v) : launch_vec_t<float, false>(m, a, v, s);
  }
  if (m->dtype == VBG_C128) {
    const cplx* v = m->vals.as<cplx>();
    if (adj && mv) return lane_rows<cplx>(m, a, true) ? launch_mv_t<cplx, true>(m, a, v, s) : launch_mma(m, true, a, s);
    if (adj) return launch_vec_t<cplx, true>(m, a, v, s);
    return mv ? fwd(cplx{}, v) : launch_vec_t<cplx, false>(m, a, v, s);
  }
  const double* v = m->vals.as<double>();
  if (adj && mv) return lane_rows<double>(m, a, true) ? launch_mv_t<double, true>(m, a, v, s) : launch_mma(m, true, a, s);
  if (adj) return launch_vec_t<double, true>(m, a, v, s);
  return mv ? fwd(double{}, v) : launch_vec_t<double, false>(m, a, v, s);
}

// ------------------------------------------------------------ helpers

template <typename T>
__global__ void sumsq_kernel(const T* __restrict__ x, int64_t n, double* partials, unsigned* counter, double* out) {
  double d = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    d += re_dot(x[i], x[i]);
  grid_reduce2(d, 0.0, partials, counter, out, 0, gridDim.x);
}

__global__ void f64_to_f32_rows(const double* __restrict__ src, int64_t rows, int ld_src, float* __restrict__ dst,
                                int ld_dst) {
  const int64_t total = rows * ld_dst;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / ld_dst;
    const int c = (int)(i - r * ld_dst);
    dst[i] = c < ld_src ? (float)src[r * ld_src + c] : 0.0f;
  }
}

// dots[step] = (d0, d1) -> moments.  Batched: segment sg (one thread each)
// reads dots[step * stride + 2 * sg + {0, 1}] and writes mu[sg * M + n].
__global__ void kpm_finalize(const double* __restrict__ dots, int M, int two_moment, double* __restrict__ mu,
                             int stride, int nseg) {
  const int sg = blockIdx.x * blockDim.x + threadIdx.x;
  if (sg >= nseg) return;
  auto D = [&](int step, int w) { return dots[(size_t)step * stride + 2 * sg + w]; };
  double* out = mu + (size_t)sg * M;
  // step 0 = (sum |v0|^2, -), step 1 = the apply producing t_1, step n+1 = the one producing t_{n+1}
  const double mu0 = D(0, 0);
  out[0] = mu0;
  if (M < 2) return;
  const double mu1 = D(1, 0);
  out[1] = mu1;
  if (two_moment) {
    if (M > 2) out[2] = 2.0 * D(1, 1) - mu0;
    for (int n = 1;; ++n) {
      const int odd = 2 * n + 1, even = 2 * n + 2;
      if (odd >= M) break;
      out[odd] = 2.0 * D(n + 1, 0) - mu1;
      if (even < M) out[even] = 2.0 * D(n + 1, 1) - mu0;
    }
  } else {
    for (int n = 2; n < M; ++n) out[n] = D(n, 0);
  }
}

// Fixed-order sum of two values over the threads of a block (blockDim.x
// a multiple of 32, at most 1024); result in thread 0.
__device__ void block_sum2(double& a0, double& a1) {
  __shared__ double red[32][2];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    a0 += __shfl_xor_sync(0xffffffffu, a0, off);
    a1 += __shfl_xor_sync(0xffffffffu, a1, off);
  }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    red[w][0] = a0;
    red[w][1] = a1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double s0 = 0.0, s1 = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      s0 += red[k][0];
      s1 += red[k][1];
    }
    a0 = s0;
    a1 = s1;
  }
  __syncthreads();
}

// Sums per segment of a batched recurrence.  A segment's block rows are cut
// into chunks of kSegChunkRows ({segment, first row, end row, first chunk of
// the segment}), a CTA per chunk; the last CTA of a segment to finish adds
// the segment's partial sums in chunk order (so the result does not depend
// on which one that is) and resets its counter.  A CTA per segment instead
// leaves all but nseg SMs idle: on 10 lattices of 40-100 cells a side (164k
// block rows, 9.6 M vector elements) the row-dot sums took 24-56 us per step
// and the initial sum of squares 2.97 ms.
constexpr int kSegChunkRows = 512;

__device__ void seg_chunk_finish(double a0, double a1, const int4 ch, const int* __restrict__ seg_chunk,
                                 double* __restrict__ partials, unsigned* __restrict__ counters,
                                 double* __restrict__ out) {
  __shared__ bool last;
  block_sum2(a0, a1);
  const int c1 = seg_chunk[ch.x + 1];
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = a0;
    partials[2 * blockIdx.x + 1] = a1;
    __threadfence();
    last = atomicAdd(counters + ch.x, 1u) == (unsigned)(c1 - ch.w) - 1u;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double s0 = 0.0, s1 = 0.0;
  for (int c = ch.w + threadIdx.x; c < c1; c += blockDim.x) {
    s0 += __ldcg(partials + 2 * c);
    s1 += __ldcg(partials + 2 * c + 1);
  }
  block_sum2(s0, s1);
  if (threadIdx.x == 0) {
    out[2 * ch.x] = s0;
    out[2 * ch.x + 1] = s1;
    counters[ch.x] = 0u;
  }
}

// out[2 sg + {0,1}] = sums of the per-row dots over segment sg's block rows.
__global__ void seg_row_dots_kernel(const double* __restrict__ row_dots, const int4* __restrict__ chunks,
                                    const int* __restrict__ seg_chunk, double* __restrict__ partials,
                                    unsigned* __restrict__ counters, double* __restrict__ out) {
  const int4 ch = chunks[blockIdx.x];
  double a0 = 0.0, a1 = 0.0;
  for (int i = ch.y + threadIdx.x; i < ch.z; i += blockDim.x) {
    a0 += row_dots[2 * (int64_t)i];
    a1 += row_dots[2 * (int64_t)i + 1];
  }
  seg_chunk_finish(a0, a1, ch, seg_chunk, partials, counters, out);
}

// out[2 sg] = sum |x|^2 over segment sg's scalar rows (all ld lanes).
template <typename T>
__global__ void seg_sumsq_kernel(const T* __restrict__ x, const int64_t* __restrict__ scal_off, int ld,
                                 const int4* __restrict__ chunks, const int* __restrict__ seg_chunk,
                                 double* __restrict__ partials, unsigned* __restrict__ counters,
                                 double* __restrict__ out) {
  const int4 ch = chunks[blockIdx.x];
  double a0 = 0.0;
  const int64_t e1 = scal_off[ch.z] * ld;
  for (int64_t i = scal_off[ch.y] * ld + threadIdx.x; i < e1; i += blockDim.x) a0 += re_dot(x[i], x[i]);
  seg_chunk_finish(a0, 0.0, ch, seg_chunk, partials, counters, out);
}

static int ensure_grid_scratch(const vbg_matrix* m) { return ensure_scratch(m, max_total_ctas()); }

template <typename T>
static int launch_sumsq(const vbg_matrix* m, const T* x, int64_t n, double* out, cudaStream_t s) {
  int grid = (int)std::min<int64_t>((n + kThreads - 1) / kThreads, (int64_t)sm_count() * 8);
  grid = std::max(grid, 1);
  sumsq_kernel<T><<<grid, kThreads, 0, s>>>(x, n, m->partials.as<double>(), m->counter.as<unsigned>(), out);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

// Runs the autotuner for the forward applies of a Chebyshev recurrence on
// these buffers (before a graph capture, where it cannot run): one step
// Y = 2 A X - Xprev with its dots (per block row when row_dots is set).
template <typename T>
static int tune_recurrence(const vbg_matrix* m, bool f32, int R, int ld, const T* X, const T* Xprev, T* Y,
                           double* dots, double* row_dots, cudaStream_t s) {
  ApplyArgs a;
  int rc = prepare(m, false, R, ld, a, s);
  if (rc) return rc;
  if (R <= 1) {
    // the vector kernel's records and choice, before a graph capture
    if (!a.slot_meta || row_dots) return 0;
    a.X = X;
    a.Xprev = Xprev;
    a.Y = Y;
    a.alpha = 2.0;
    a.gamma = -1.0;
    a.n_scal = m->N;
    const int2* sr;
    const T* v = f32 ? reinterpret_cast<const T*>(m->vals32.as<float>()) : reinterpret_cast<const T*>(m->vals.p);
    return vec_kernel<T>(m, f32, a, v, s, true, &sr);
  }
  a.X = X;
  a.Xprev = Xprev;
  a.Y = Y;
  a.alpha = 2.0;
  a.gamma = -1.0;
  a.want_dots = 1;
  a.partials = m->partials.as<double>();
  a.counter = m->counter.as<unsigned>();
  a.dots_out = dots;
  a.row_dots = row_dots;
  const T* v = f32 ? reinterpret_cast<const T*>(m->vals32.as<float>()) : reinterpret_cast<const T*>(m->vals.p);
  int which = -1;
  return fwd_choice<T>(m, f32, a, v, s, true, &which);
}

// Enqueues the whole KPM recurrence on stream s.
template <typename T>
static int kpm_enqueue(const vbg_matrix* m, int R, int ld, const T* V0, int M, bool f32, int two_moment, T* B0,
                       T* B1, T* B2, double* dots, double* moments, cudaStream_t s) {
  int rc = launch_sumsq<T>(m, V0, m->N * (int64_t)ld, dots, s);
  if (rc) return rc;
  if (M >= 2) {
    ApplyArgs a;
    if ((rc = prepare(m, false, R, ld, a, s))) return rc;
    a.want_dots = 1;
    a.partials = m->partials.as<double>();
    a.counter = m->counter.as<unsigned>();
    // t_1 = A t_0
    a.X = V0;
    a.Y = B0;
    a.alpha = 1.0;
    a.dotw = V0;
    a.dots_out = dots + 2;
    if ((rc = launch_apply(m, false, f32, a, s))) return rc;
    T* bufs[3] = {B0, B1, B2};
    const T* prev = V0;
    const T* cur = B0;
    int nb = 1;
    const int steps = two_moment ? (M - 2) / 2 : M - 2;  // SpMMs after the first
    for (int n = 1; n <= steps; ++n) {
      T* next = bufs[nb];
      nb = (nb + 1) % 3;
      a.X = cur;
      a.Xprev = prev;
      a.Y = next;
      a.alpha = 2.0;
      a.gamma = -1.0;
      a.dotw = two_moment ? nullptr : V0;
      a.dots_out = dots + 2 * (n + 1);
      if ((rc = launch_apply(m, false, f32, a, s))) return rc;
      prev = cur;
      cur = next;
    }
  }
  kpm_finalize<<<1, 32, 0, s>>>(dots, M, two_moment, moments, 2, 1);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace vbg

using namespace vbg;

extern "C" {

int vbg_set_option(const char* name, long long value) {
  VBG_CHECK(name, VBG_E_ARG, "null option name");
  if (std::strcmp(name, "apply.chain") == 0) {
    VBG_CHECK(value >= 0 && value <= 2, VBG_E_ARG, "apply.chain takes 0, 1 or 2");
    g_opt_chain.store((int)value);
    return 0;
  }
  if (std::strcmp(name, "apply.autotune") == 0) {
    g_opt_autotune.store(value != 0 ? 1 : 0);
    return 0;
  }
  if (std::strcmp(name, "apply.vec_lanes") == 0) {
    VBG_CHECK(value == 0 || value == 1 || value == 2 || value == 4 || value == 8, VBG_E_ARG,
              "apply.vec_lanes takes 0, 1, 2, 4 or 8");
    g_opt_vec_lanes.store((int)value);
    return 0;
  }
  if (std::strcmp(name, "apply.vec_kernel") == 0) {
    VBG_CHECK(value >= 0 && value <= 2, VBG_E_ARG, "apply.vec_kernel takes 0, 1 or 2");
    g_opt_vec_kernel.store((int)value);
    return 0;
  }
  return fail(VBG_E_ARG, std::string("unknown option '") + name + "'");
}

int vbg_get_option(const char* name, long long* value) {
  VBG_CHECK(name && value, VBG_E_ARG, "null argument");
  if (std::strcmp(name, "apply.chain") == 0) {
    *value = g_opt_chain.load();
    return 0;
  }
  if (std::strcmp(name, "apply.autotune") == 0) {
    *value = g_opt_autotune.load();
    return 0;
  }
  if (std::strcmp(name, "apply.vec_lanes") == 0) {
    *value = g_opt_vec_lanes.load();
    return 0;
  }
  if (std::strcmp(name, "apply.vec_kernel") == 0) {
    *value = g_opt_vec_kernel.load();
    return 0;
  }
  return fail(VBG_E_ARG, std::string("unknown option '") + name + "'");
}

int vbg_device_status(unsigned* status, int clear) {
  VBG_CHECK(status, VBG_E_ARG, "null argument");
  VBG_CUDA(cudaMemcpyFromSymbol(status, g_pipe_status, sizeof(unsigned)));
  if (clear) {
    const unsigned zero = 0;
    VBG_CUDA(cudaMemcpyToSymbol(g_pipe_status, &zero, sizeof(unsigned)));
  }
  return 0;
}

int vbg_spmv(const vbg_matrix* m, const void* x, void* y, void* stream) {
  ApplyArgs a;
  cudaStream_t s = as_stream(stream);
  int rc = prepare(m, false, 1, 1, a, s);
  if (rc) return rc;
  VBG_CHECK(x && y, VBG_E_ARG, "null vector");
  a.X = x;
  a.Y = y;
  return launch_apply(m, false, false, a, s);
}

int vbg_spmv_adjoint(const vbg_matrix* m, const void* x, void* y, void* stream) {
  ApplyArgs a;
  cudaStream_t s = as_stream(stream);
  int rc = prepare(m, true, 1, 1, a, s);
  if (rc) return rc;
  VBG_CHECK(x && y, VBG_E_ARG, "null vector");
  a.X = x;
  a.Y = y;
  return launch_apply(m, true, false, a, s);
}

int vbg_spmm(const vbg_matrix* m, int k, int ld, const void* X, void* Y, void* stream) {
  ApplyArgs a;
  cudaStream_t s = as_stream(stream);
  int rc = prepare(m, false, k, ld, a, s);
  if (rc) return rc;
  VBG_CHECK(X && Y, VBG_E_ARG, "null multivector");
  a.X = X;
  a.Y = Y;
  return launch_apply(m, false, false, a, s);
}

int vbg_apply_tile_rows(const vbg_matrix* m, int ld, int precision, int* rows) {
  VBG_CHECK(m && rows, VBG_E_ARG, "null argument");
  VBG_CHECK(precision == VBG_PREC_F64 || (precision == VBG_PREC_F32 && m->dtype == VBG_F64), VBG_E_ARG,
            "precision must be VBG_PREC_F64, or VBG_PREC_F32 for a real matrix");
  const int es = precision == VBG_PREC_F32 ? 4 : (int)elem_size(m->dtype);
  *rows = 0;
  auto it = m->tile_plans.find(std::make_tuple(ld * es, es, tile_cap(m, ld, es)));
  if (it != m->tile_plans.end()) *rows = it->second->rows;
  return 0;
}

int vbg_apply_kernel(const vbg_matrix* m, int ld, int precision, int* kernel) {
  VBG_CHECK(m && kernel, VBG_E_ARG, "null argument");
  VBG_CHECK(precision == VBG_PREC_F64 || (precision == VBG_PREC_F32 && m->dtype == VBG_F64), VBG_E_ARG,
            "precision must be VBG_PREC_F64, or VBG_PREC_F32 for a real matrix");
  ApplyArgs a;
  int rc = prepare(m, false, 1, ld, a, nullptr);
  if (rc) return rc;
  if (ld <= 1) {
    *kernel = VBG_KERNEL_VECTOR;
    if (a.slot_meta && srow_possible(m)) {
      const int forced = g_opt_vec_kernel.load();
      auto it = m->tuned.find(std::make_pair(1, precision == VBG_PREC_F32 ? 1 : 0));
      if (forced == 2 || (forced == 0 && (it != m->tuned.end() ? it->second != VBG_KERNEL_VECTOR
                                                              : (m->dtype == VBG_C128 && precision == VBG_PREC_F64))))
        *kernel = VBG_KERNEL_SCALAR_ROWS;
    }
    return 0;
  }
  // the autotuner's choice once it has made one
  if (g_opt_autotune.load() && g_opt_chain.load() == 2) {
    auto it = m->tuned.find(std::make_pair(ld, precision == VBG_PREC_F32 ? 1 : 0));
    if (it != m->tuned.end()) {
      *kernel = it->second;
      return 0;
    }
  }
  // buffers aligned as the library's own allocations are
  a.X = a.Y = reinterpret_cast<void*>(static_cast<uintptr_t>(256));
  TilePlan* tp = nullptr;
  ChainPlan* cp = nullptr;
  bool chain, tile, pipe;
  const bool chain_ok = chain_enabled(precision == VBG_PREC_F32 ? 4 : (int)elem_size(m->dtype));
  if (precision == VBG_PREC_F32) {
    chain = chain_ok && (chain_use<float>(m, a, nullptr, true, &cp) || chain_use<float, 1>(m, a, nullptr, true, &cp) ||
                         chain_use<float, 1, 2>(m, a, nullptr, true, &cp));
    tile = chain || tile_use<float>(m, false, a, nullptr, true, &tp) ||
           tile_use<float, 4, 4>(m, false, a, nullptr, true, &tp) || tile_use<float, 4, 8>(m, false, a, nullptr, true, &tp);
    pipe = tile || pipe_use<float>(m, false, a, nullptr, true);
  } else if (m->dtype == VBG_C128) {
    chain = chain_ok && chain_use<cplx>(m, a, nullptr, true, &cp);
    tile = chain || tile_use<cplx>(m, false, a, nullptr, true, &tp);
    pipe = tile || pipe_use<cplx>(m, false, a, nullptr, true);
  } else {
    chain = chain_ok && (chain_use<double>(m, a, nullptr, true, &cp) || chain_use<double, 1, 2>(m, a, nullptr, true, &cp));
    tile = chain || tile_use<double>(m, false, a, nullptr, true, &tp);
    pipe = tile || pipe_use<double>(m, false, a, nullptr, true);
  }
  const bool lane = m->dtype == VBG_C128 ? lane_rows<cplx>(m, a, false)
                                         : precision == VBG_PREC_F64 && lane_rows<double>(m, a, false);
  *kernel = chain ? VBG_KERNEL_CHAIN
            : tile ? VBG_KERNEL_TILE
            : pipe ? VBG_KERNEL_PIPE
            : lane ? VBG_KERNEL_LANE_ROWS
                   : VBG_KERNEL_ROWS;
  return 0;
}

int vbg_adjoint_kernel(const vbg_matrix* m, int ld, int* kernel) {
  VBG_CHECK(m && kernel, VBG_E_ARG, "null argument");
  VBG_CHECK(ld > 1, VBG_E_ARG, "the adjoint of multivectors only (ld > 1)");
  ApplyArgs a;
  std::memset(&a, 0, sizeof(a));
  a.ld = ld;
  const bool lane = m->dtype == VBG_C128 ? lane_rows<cplx>(m, a, true) : lane_rows<double>(m, a, true);
  *kernel = lane ? VBG_KERNEL_LANE_ROWS : VBG_KERNEL_ROWS;
  return 0;
}

int vbg_spmm_adjoint(const vbg_matrix* m, int k, int ld, const void* X, void* Y, void* stream) {
  ApplyArgs a;
  cudaStream_t s = as_stream(stream);
  int rc = prepare(m, true, k, ld, a, s);
  if (rc) return rc;
  VBG_CHECK(X && Y, VBG_E_ARG, "null multivector");
  a.X = X;
  a.Y = Y;
  return launch_apply(m, true, false, a, s);
}

// The fused step of vbg_cheb_step / vbg_cheb_step_adjoint.
static int fused_step(const vbg_matrix* m, bool adj, int k, int ld, double alpha, double beta, double gamma,
                      const void* X, const void* Xprev, void* Y, const void* dot_with, double* dots, void* acc,
                      double cre, double cim, void* stream) {
  ApplyArgs a;
  cudaStream_t s = as_stream(stream);
  int rc = prepare(m, adj, k, ld, a, s);
  if (rc) return rc;
  VBG_CHECK(X && Y, VBG_E_ARG, "null multivector");
  VBG_CHECK(gamma == 0.0 || Xprev, VBG_E_ARG, "Xprev is required when gamma != 0");
  a.alpha = alpha;
  a.beta = beta;
  a.gamma = gamma;
  a.X = X;
  a.Xprev = Xprev;
  a.Y = Y;
  a.dotw = dot_with;
  a.acc = acc;
  a.cre = cre;
  a.cim = cim;
  if (dots) {
    if ((rc = ensure_grid_scratch(m))) return rc;
    a.want_dots = 1;
    a.partials = m->partials.as<double>();
    a.counter = m->counter.as<unsigned>();
    a.dots_out = dots;
  }
  return launch_apply(m, adj, false, a, s);
}

int vbg_cheb_step(const vbg_matrix* m, int k, int ld, double alpha, double beta, double gamma, const void* X,
                  const void* Xprev, void* Y, const void* dot_with, double* dots, void* acc, double cre, double cim,
                  void* stream) {
  return fused_step(m, false, k, ld, alpha, beta, gamma, X, Xprev, Y, dot_with, dots, acc, cre, cim, stream);
}

int vbg_cheb_step_adjoint(const vbg_matrix* m, int k, int ld, double alpha, double beta, double gamma, const void* X,
                          const void* Xprev, void* Y, const void* dot_with, double* dots, void* acc, double cre,
                          double cim, void* stream) {
  return fused_step(m, true, k, ld, alpha, beta, gamma, X, Xprev, Y, dot_with, dots, acc, cre, cim, stream);
}

int vbg_cheb_series(const vbg_matrix* m, int k, int ld, const void* V, int M, const double* coeffs, double scale,
                    double center, void* psi, int K, void* ckpt, void* stream) {
  VBG_CHECK(m && V && psi && coeffs, VBG_E_ARG, "null argument");
  VBG_CHECK(M >= 1 && k >= 1 && ld >= k && scale != 0.0, VBG_E_ARG, "invalid M / k / ld / scale");
  VBG_CHECK(K <= 0 || ckpt || M <= K, VBG_E_ARG, "checkpoint buffer required when K > 0");
  const int dtype = m->dtype;
  const size_t es = elem_size(dtype);
  const int64_t rows = m->N;
  const size_t bytes = (size_t)rows * (size_t)ld * es;
  cudaStream_t s = as_stream(stream);
  int rc;
  // psi = c_0 t_0
  VBG_CUDA(cudaMemsetAsync(psi, 0, bytes, s));
  if ((rc = vbg_mv_axpby(dtype, rows, k, ld, coeffs[0], coeffs[1], V, 0.0, 0.0, psi, stream))) return rc;
  if (M == 1) return 0;
  if (ld == 1 && !g_opt_vec_kernel.load()) {
    // the whole series in one launch when the matrix fits the SMs' shared memory
    std::vector<double> cf((size_t)(M - 1) * kResCoef);
    for (int n = 1; n < M; ++n) {
      const double w = n == 1 ? 1.0 : 2.0;
      double* c = &cf[(size_t)(n - 1) * kResCoef];
      c[0] = w / scale;
      c[1] = -w * center / scale;
      c[2] = n == 1 ? 0.0 : -1.0;
      c[3] = coeffs[2 * n];
      c[4] = coeffs[2 * n + 1];
    }
    ResidentArgs a{};
    a.x0 = V;
    a.steps = M - 1;
    a.psi = psi;
    a.K = K;
    a.M = M;
    a.ckpt = ckpt;
    DevBuf scratch(s);
    bool ran = false;
    if ((rc = resident_run(m, false, a, cf.data(), scratch, s, &ran))) return rc;
    if (ran) {
      // K = 1: the first pair's t_0 is V
      if (K == 1)
        VBG_CUDA(cudaMemcpyAsync(static_cast<char*>(ckpt) + bytes, V, bytes, cudaMemcpyDeviceToDevice, s));
      return 0;
    }
  }
  DevBuf buf[3] = {DevBuf(s), DevBuf(s), DevBuf(s)};
  for (auto& b : buf) {
    if ((rc = b.ensure(std::max<size_t>(bytes, 16)))) return rc;
    VBG_CUDA(cudaMemsetAsync(b.p, 0, bytes, s));  // pad lanes stay zero
  }
  const int n_ck = K > 0 ? (M - 1) / K : 0;
  if (n_ck > 0) VBG_CUDA(cudaMemsetAsync(ckpt, 0, (size_t)2 * n_ck * bytes, s));
  const void* t_prev = nullptr;
  const void* t = V;
  // t_n is written straight into its checkpoint slot when n = K, 2K, ...
  // (vector 2j) or n + 1 is (vector 2j + 1), else into a working vector
  // that holds neither t_{n-1} nor t_{n-2}
  auto slot = [&](int j, int w) { return static_cast<char*>(ckpt) + (size_t)(2 * j + w) * bytes; };
  for (int n = 1; n < M; ++n) {
    void* y = nullptr;
    if (K > 0 && n % K == 0)
      y = slot(n / K - 1, 0);
    else if (K > 0 && (n + 1) % K == 0 && n + 1 < M)
      y = slot((n + 1) / K - 1, 1);
    else
      for (auto& b : buf)
        if (b.p != t && b.p != t_prev) {
          y = b.p;
          break;
        }
    const bool first = n == 1;
    const double alpha = (first ? 1.0 : 2.0) / scale;
    const double beta = -(first ? 1.0 : 2.0) * center / scale;
    const double gamma = first ? 0.0 : -1.0;
    if ((rc = vbg_cheb_step(m, k, ld, alpha, beta, gamma, t, first ? nullptr : t_prev, y, nullptr, nullptr, psi,
                            coeffs[2 * n], coeffs[2 * n + 1], stream)))
      return rc;
    // K = 1: t_{n-1} sits in the previous pair's slot (or is V)
    if (K > 0 && n % K == 0 && t != slot(n / K - 1, 1))
      VBG_CUDA(cudaMemcpyAsync(slot(n / K - 1, 1), t, bytes, cudaMemcpyDeviceToDevice, s));
    t_prev = t;
    t = y;
  }
  return 0;
}

int vbg_cheb_columns(const vbg_matrix* m, int adjoint, const void* x0, const void* x1, int steps,
                     const double* coeffs, const void* source, void* cols, int64_t ldc, int ncol, int col0, int dcol,
                     void* last, void* before, void* stream) {
  VBG_CHECK(m && x0 && coeffs, VBG_E_ARG, "null argument");
  VBG_CHECK(steps >= 0 && (!cols || (ncol >= 0 && ldc >= ncol)), VBG_E_ARG, "invalid steps / ncol / ldc");
  cudaStream_t s = as_stream(stream);
  if (m->N == 0) return 0;
  const size_t es = elem_size(m->dtype), bytes = (size_t)m->N * es;
  int rc;
  auto copy = [&](void* to, const void* from) -> int {
    if (to && to != from) VBG_CUDA(cudaMemcpyAsync(to, from, bytes, cudaMemcpyDeviceToDevice, s));
    return 0;
  };
  auto column = [&](int c, const void* v) -> int {
    if (cols && c >= 0 && c < ncol)
      VBG_CUDA(cudaMemcpy2DAsync(static_cast<char*>(cols) + (size_t)c * es, (size_t)ldc * es, v, es, es, m->N,
                                 cudaMemcpyDeviceToDevice, s));
    return 0;
  };
  ResidentArgs a{};
  a.x0 = x0;
  a.x1 = x1;
  a.steps = steps;
  a.source = source;
  a.cols = cols;
  a.ldc = ldc;
  a.col0 = col0;
  a.dcol = dcol;
  a.ncol = ncol;
  DevBuf scratch(s);
  bool ran = false;
  // (a forced vector kernel runs its own steps)
  if (!g_opt_vec_kernel.load() && (rc = resident_run(m, adjoint != 0, a, coeffs, scratch, s, &ran))) return rc;
  if (ran) {
    if ((rc = copy(last, a.xch[(steps - 1) & 1]))) return rc;
    return copy(before, steps > 1 ? a.xch[steps & 1] : x0);
  }
  // a fused step at a time, on three working vectors
  if ((rc = column(col0, x0))) return rc;
  DevBuf buf(s);
  const size_t room = (bytes + 255) / 256 * 256;
  if ((rc = buf.ensure(3 * room))) return rc;
  const void *x = x0, *p = x1;
  for (int k = 0; k < steps; ++k) {
    const double* c = coeffs + (size_t)kResCoef * k;
    char* y = buf.as<char>();
    while (y == x || y == p) y += room;
    const double gamma = p ? c[2] : 0.0;
    if ((rc = fused_step(m, adjoint != 0, 1, 1, c[0], c[1], gamma, x, p, y, nullptr, nullptr, nullptr, 0.0, 0.0,
                         stream)))
      return rc;
    if (source && (rc = vbg_mv_axpby(m->dtype, m->N, 1, 1, c[3], c[4], source, 1.0, 0.0, y, stream))) return rc;
    if ((rc = column(col0 + (k + 1) * dcol, y))) return rc;
    p = x;
    x = y;
  }
  if ((rc = copy(last, x))) return rc;
  return p ? copy(before, p) : 0;
}

int vbg_recurrence_resident(const vbg_matrix* m, int adjoint, int* resident) {
  VBG_CHECK(m && resident, VBG_E_ARG, "null argument");
  const auto& plan = m->resident[adjoint ? 1 : 0];
  *resident = plan && plan->ran ? 1 : 0;
  return 0;
}

int vbg_kpm_moments(const vbg_matrix* m, int R, int ld, const void* V0, int M, int precision, int two_moment,
                    int use_graph, double* moments, void* stream) {
  VBG_CHECK(m && V0 && moments, VBG_E_ARG, "null argument");
  VBG_CHECK(m->dtype == VBG_F64, VBG_E_ARG, "KPM moments are defined for real symmetric matrices");
  VBG_CHECK(R >= 1 && ld >= R && M >= 1, VBG_E_ARG, "invalid R / ld / M");
  VBG_CHECK(precision == VBG_PREC_F64 || precision == VBG_PREC_F32, VBG_E_ARG, "unknown precision");
  VBG_CHECK(R == 1 ? true : (ld * 8) % 16 == 0, VBG_E_ARG, "ld must span a multiple of 16 bytes");
  cudaStream_t s = as_stream(stream);
  auto* mm = const_cast<vbg_matrix*>(m);
  int rc = ensure_grid_scratch(m);
  if (rc) return rc;
  const bool f32 = precision == VBG_PREC_F32;
  // FP32 multivectors use the reference's padding rule for 4-byte scalars.
  const int ldw = f32 ? (R == 1 ? 1 : ((R * 4 + 63) / 64) * 16) : ld;
  const size_t es = f32 ? 4 : 8;
  const size_t nbuf = f32 ? 4 : 3;
  const size_t buf_bytes = ((size_t)m->N * ldw * es + 255) / 256 * 256;
  const void* ws_before = mm->kpm_ws.p;
  const void* dots_before = mm->kpm_dots.p;
  if ((rc = mm->kpm_ws.ensure(std::max<size_t>(nbuf * buf_bytes, 256)))) return rc;
  const int nsteps = M + 2;
  if ((rc = mm->kpm_dots.ensure((size_t)nsteps * 2 * sizeof(double)))) return rc;
  // captured graphs hold raw workspace pointers
  if (mm->kpm_ws.p != ws_before || mm->kpm_dots.p != dots_before) mm->graphs.clear();
  char* base = mm->kpm_ws.as<char>();
  double* dots = mm->kpm_dots.as<double>();
  if (f32) {
    const int64_t tot = m->N * (int64_t)ldw;
    f64_to_f32_rows<<<std::max<int64_t>(1, std::min<int64_t>((tot + 255) / 256, sm_count() * 16)), 256, 0, s>>>(
        static_cast<const double*>(V0), m->N, ld, reinterpret_cast<float*>(base + 3 * buf_bytes), ldw);
    VBG_CUDA(cudaGetLastError());
    if ((rc = ensure_vals32(m, s))) return rc;
  }
  // the pipelined kernel's value layout must exist before a graph capture
  if (R > 1 && m->max_bs <= kPipeMaxBs && (f32 ? pipe_groups<float>(ldw) : pipe_groups<double>(ldw)) != 0) {
    if ((rc = ensure_kernel_layout(m, f32, s))) return rc;
    if ((rc = ensure_spans(m, pipe_span_cap(m), s))) return rc;
    // (with the autotuner on, tune_recurrence makes the plan it wants)
    if (!(g_opt_autotune.load() && g_opt_chain.load() == 2) && (rc = tile_prepare(m, f32, ldw, s))) return rc;
  }
  // the kernel choice, before a graph capture freezes it
  if (f32)
    rc = tune_recurrence<float>(m, true, R, ldw, reinterpret_cast<const float*>(base + 3 * buf_bytes),
                                reinterpret_cast<const float*>(base + buf_bytes), reinterpret_cast<float*>(base),
                                dots + 2, nullptr, s);
  else
    rc = tune_recurrence<double>(m, false, R, ldw, static_cast<const double*>(V0),
                                 reinterpret_cast<const double*>(base + buf_bytes), reinterpret_cast<double*>(base),
                                 dots + 2, nullptr, s);
  if (rc) return rc;
  auto enqueue = [&](cudaStream_t st) -> int {
    if (f32)
      return kpm_enqueue<float>(m, R, ldw, reinterpret_cast<const float*>(base + 3 * buf_bytes), M, true, two_moment,
                                reinterpret_cast<float*>(base), reinterpret_cast<float*>(base + buf_bytes),
                                reinterpret_cast<float*>(base + 2 * buf_bytes), dots, moments, st);
    return kpm_enqueue<double>(m, R, ldw, static_cast<const double*>(V0), M, false, two_moment,
                               reinterpret_cast<double*>(base), reinterpret_cast<double*>(base + buf_bytes),
                               reinterpret_cast<double*>(base + 2 * buf_bytes), dots, moments, st);
  };
  if (!use_graph) return enqueue(s);

  auto key = std::make_tuple(R, ld, V0, M, precision, two_moment, moments);
  auto it = mm->graphs.find(key);
  if (it == mm->graphs.end()) {
    if (!mm->graph_stream) VBG_CUDA(cudaStreamCreateWithFlags(&mm->graph_stream, cudaStreamNonBlocking));
    auto ge = std::make_unique<GraphEntry>();
    VBG_CUDA(cudaStreamBeginCapture(mm->graph_stream, cudaStreamCaptureModeThreadLocal));
    rc = enqueue(mm->graph_stream);
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(mm->graph_stream, &g);
    if (rc) {
      if (g) cudaGraphDestroy(g);
      return rc;
    }
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture");
    ge->graph = g;
    VBG_CUDA(cudaGraphInstantiate(&ge->exec, g, 0));
    it = mm->graphs.emplace(key, std::move(ge)).first;
  }
  VBG_CUDA(cudaGraphLaunch(it->second->exec, s));
  return 0;
}

int vbg_kpm_moments_host(const vbg_matrix* m, int R, const double* V0, int M, int precision, int two_moment,
                         double* moments, void* stream) {
  VBG_CHECK(m && V0 && moments, VBG_E_ARG, "null argument");
  VBG_CHECK(R >= 1 && M >= 1, VBG_E_ARG, "invalid R / M");
  cudaStream_t s = as_stream(stream);
  const int ld = R == 1 ? 1 : ((R * 8 + 63) / 64) * 8;
  DevBuf dv, dm;
  int rc;
  if ((rc = dv.ensure((size_t)m->N * ld * 8))) return rc;
  if ((rc = dm.ensure((size_t)M * 8))) return rc;
  if (ld != R) VBG_CUDA(cudaMemsetAsync(dv.p, 0, (size_t)m->N * ld * 8, s));
  VBG_CUDA(cudaMemcpy2DAsync(dv.p, (size_t)ld * 8, V0, (size_t)R * 8, (size_t)R * 8, m->N, cudaMemcpyHostToDevice, s));
  if ((rc = vbg_kpm_moments(m, R, ld, dv.p, M, precision, two_moment, 0, dm.as<double>(), s))) return rc;
  VBG_CUDA(cudaMemcpyAsync(moments, dm.p, (size_t)M * 8, cudaMemcpyDeviceToHost, s));
  VBG_CUDA(cudaStreamSynchronize(s));
  return 0;
}

}  // extern "C"

namespace vbg {

// Enqueues the batched recurrence: one block-diagonal matrix whose diagonal
// blocks (segments) are independent Hamiltonians; every apply writes per-row
// dots that a segmented reduction turns into per-segment dots.
template <typename T>
static int kpm_enqueue_batched(const vbg_matrix* m, int nseg, int R, int ld, const T* V0, int M, bool f32,
                               int two_moment, T* B0, T* B1, T* B2, double* row_dots, double* dots, double* moments,
                               cudaStream_t s) {
  const int stride = 2 * nseg;
  const int nch = m->kpm_nchunks;
  const int4* chunks = m->kpm_chunks.as<int4>();
  const int* seg_chunk = m->kpm_segchunk.as<int>();
  double* part = m->kpm_segpart.as<double>();
  unsigned* cnt = m->kpm_segcnt.as<unsigned>();
  auto row_sums = [&](double* out) -> int {
    seg_row_dots_kernel<<<nch, 256, 0, s>>>(row_dots, chunks, seg_chunk, part, cnt, out);
    VBG_CUDA(cudaGetLastError());
    return 0;
  };
  // segments without rows have no chunk: their sums are zero
  VBG_CUDA(cudaMemsetAsync(dots, 0, (size_t)(M + 2) * stride * sizeof(double), s));
  if (nch) {
    seg_sumsq_kernel<T><<<nch, 256, 0, s>>>(V0, m->scal_off.as<int64_t>(), ld, chunks, seg_chunk, part, cnt, dots);
    VBG_CUDA(cudaGetLastError());
  }
  if (M >= 2) {
    ApplyArgs a;
    int rc;
    if ((rc = prepare(m, false, R, ld, a, s))) return rc;
    a.want_dots = 1;
    a.row_dots = row_dots;
    a.X = V0;
    a.Y = B0;
    a.alpha = 1.0;
    a.dotw = V0;
    if ((rc = launch_apply(m, false, f32, a, s))) return rc;
    if (nch && (rc = row_sums(dots + stride))) return rc;
    T* bufs[3] = {B0, B1, B2};
    const T* prev = V0;
    const T* cur = B0;
    int nb = 1;
    const int steps = two_moment ? (M - 2) / 2 : M - 2;
    for (int n = 1; n <= steps; ++n) {
      T* next = bufs[nb];
      nb = (nb + 1) % 3;
      a.X = cur;
      a.Xprev = prev;
      a.Y = next;
      a.alpha = 2.0;
      a.gamma = -1.0;
      a.dotw = two_moment ? nullptr : V0;
      if ((rc = launch_apply(m, false, f32, a, s))) return rc;
      if (nch && (rc = row_sums(dots + (size_t)stride * (n + 1)))) return rc;
      prev = cur;
      cur = next;
    }
  }
  kpm_finalize<<<(nseg + 127) / 128, 128, 0, s>>>(dots, M, two_moment, moments, stride, nseg);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace vbg

extern "C" {

int vbg_kpm_moments_batched(const vbg_matrix* m, int nseg, const int* seg_rows, int R, int ld, const void* V0, int M,
                            int precision, int two_moment, int use_graph, double* moments, void* stream) {
  VBG_CHECK(m && seg_rows && V0 && moments, VBG_E_ARG, "null argument");
  VBG_CHECK(m->dtype == VBG_F64, VBG_E_ARG, "KPM moments are defined for real symmetric matrices");
  VBG_CHECK(nseg >= 1 && R >= 2 && ld >= R && M >= 1, VBG_E_ARG,
            "invalid nseg / R / ld / M (batched moments need a multivector, R >= 2)");
  VBG_CHECK((ld * 8) % 16 == 0, VBG_E_ARG, "ld must span a multiple of 16 bytes");
  VBG_CHECK(precision == VBG_PREC_F64 || precision == VBG_PREC_F32, VBG_E_ARG, "unknown precision");
  VBG_CHECK(seg_rows[0] == 0 && seg_rows[nseg] == m->n, VBG_E_ARG, "segments must cover the block rows");
  for (int i = 0; i < nseg; ++i) VBG_CHECK(seg_rows[i + 1] >= seg_rows[i], VBG_E_ARG, "segments not monotone");
  cudaStream_t s = as_stream(stream);
  auto* mm = const_cast<vbg_matrix*>(m);
  int rc;
  // segment tables (device), rebuilt when the layout changes
  std::vector<int> segv(seg_rows, seg_rows + nseg + 1);
  if (segv != mm->kpm_seg_host) {
    std::vector<int4> chunks;
    std::vector<int> seg_chunk(nseg + 1, 0);
    for (int i = 0; i < nseg; ++i) {
      seg_chunk[i] = (int)chunks.size();
      for (int r = seg_rows[i]; r < seg_rows[i + 1]; r += kSegChunkRows)
        chunks.push_back(make_int4(i, r, std::min(r + kSegChunkRows, seg_rows[i + 1]), seg_chunk[i]));
    }
    seg_chunk[nseg] = (int)chunks.size();
    const size_t nch = std::max<size_t>(chunks.size(), 1);
    mm->kpm_seg_host.clear();
    mm->graphs.clear();
    if ((rc = mm->kpm_chunks.ensure(nch * sizeof(int4)))) return rc;
    if ((rc = mm->kpm_segchunk.ensure((nseg + 1) * sizeof(int)))) return rc;
    if ((rc = mm->kpm_segpart.ensure(nch * 2 * sizeof(double)))) return rc;
    if ((rc = mm->kpm_segcnt.ensure(nseg * sizeof(unsigned)))) return rc;
    VBG_CUDA(cudaMemcpyAsync(mm->kpm_chunks.p, chunks.data(), chunks.size() * sizeof(int4), cudaMemcpyHostToDevice, s));
    VBG_CUDA(cudaMemcpyAsync(mm->kpm_segchunk.p, seg_chunk.data(), (nseg + 1) * sizeof(int), cudaMemcpyHostToDevice, s));
    VBG_CUDA(cudaMemsetAsync(mm->kpm_segcnt.p, 0, nseg * sizeof(unsigned), s));
    VBG_CUDA(cudaStreamSynchronize(s));
    mm->kpm_nchunks = (int)chunks.size();
    mm->kpm_seg_host = segv;
  }
  const bool f32 = precision == VBG_PREC_F32;
  // FP32 multivectors use the reference's padding rule for 4-byte scalars
  // (16 columns stay 16: the tiled applies take them with two lane groups)
  const int ldw = f32 ? ((R * 4 + 63) / 64) * 16 : ld;
  const size_t es = f32 ? 4 : 8;
  const size_t nbuf = f32 ? 4 : 3;
  const size_t buf_bytes = ((size_t)m->N * ldw * es + 255) / 256 * 256;
  const void* ws_before = mm->kpm_ws.p;
  const void* dots_before = mm->kpm_dots.p;
  const void* rd_before = mm->kpm_rowdots.p;
  if ((rc = mm->kpm_ws.ensure(std::max<size_t>(nbuf * buf_bytes, 256)))) return rc;
  if ((rc = mm->kpm_dots.ensure((size_t)(M + 2) * 2 * nseg * sizeof(double)))) return rc;
  if ((rc = mm->kpm_rowdots.ensure((size_t)std::max(m->n, 1) * 2 * sizeof(double)))) return rc;
  if (mm->kpm_ws.p != ws_before || mm->kpm_dots.p != dots_before || mm->kpm_rowdots.p != rd_before)
    mm->graphs.clear();
  char* base = mm->kpm_ws.as<char>();
  double* dots = mm->kpm_dots.as<double>();
  double* row_dots = mm->kpm_rowdots.as<double>();
  if (f32) {
    const int64_t tot = m->N * (int64_t)ldw;
    f64_to_f32_rows<<<std::max<int64_t>(1, std::min<int64_t>((tot + 255) / 256, sm_count() * 16)), 256, 0, s>>>(
        static_cast<const double*>(V0), m->N, ld, reinterpret_cast<float*>(base + 3 * buf_bytes), ldw);
    VBG_CUDA(cudaGetLastError());
    if ((rc = ensure_vals32(m, s))) return rc;
  }
  if (m->max_bs <= kPipeMaxBs && (f32 ? pipe_groups<float>(ldw) : pipe_groups<double>(ldw)) != 0) {
    if ((rc = ensure_kernel_layout(m, f32, s))) return rc;
    if ((rc = ensure_spans(m, pipe_span_cap(m), s))) return rc;
    // (with the autotuner on, tune_recurrence makes the plan it wants)
    if (!(g_opt_autotune.load() && g_opt_chain.load() == 2) && (rc = tile_prepare(m, f32, ldw, s))) return rc;
  }
  if ((rc = ensure_grid_scratch(m))) return rc;
  if (f32)
    rc = tune_recurrence<float>(m, true, R, ldw, reinterpret_cast<const float*>(base + 3 * buf_bytes),
                                reinterpret_cast<const float*>(base + buf_bytes), reinterpret_cast<float*>(base),
                                dots, row_dots, s);
  else
    rc = tune_recurrence<double>(m, false, R, ldw, static_cast<const double*>(V0),
                                 reinterpret_cast<const double*>(base + buf_bytes), reinterpret_cast<double*>(base),
                                 dots, row_dots, s);
  if (rc) return rc;
  auto enqueue = [&](cudaStream_t st) -> int {
    if (f32)
      return kpm_enqueue_batched<float>(m, nseg, R, ldw, reinterpret_cast<const float*>(base + 3 * buf_bytes),
                                        M, true, two_moment, reinterpret_cast<float*>(base),
                                        reinterpret_cast<float*>(base + buf_bytes),
                                        reinterpret_cast<float*>(base + 2 * buf_bytes), row_dots, dots, moments, st);
    return kpm_enqueue_batched<double>(m, nseg, R, ldw, static_cast<const double*>(V0), M, false, two_moment,
                                       reinterpret_cast<double*>(base), reinterpret_cast<double*>(base + buf_bytes),
                                       reinterpret_cast<double*>(base + 2 * buf_bytes), row_dots, dots, moments, st);
  };
  if (!use_graph) return enqueue(s);
  auto key = std::make_tuple(R, ld, V0, M, precision, two_moment + 2, moments);
  auto it = mm->graphs.find(key);
  if (it == mm->graphs.end()) {
    if (!mm->graph_stream) VBG_CUDA(cudaStreamCreateWithFlags(&mm->graph_stream, cudaStreamNonBlocking));
    auto ge = std::make_unique<GraphEntry>();
    VBG_CUDA(cudaStreamBeginCapture(mm->graph_stream, cudaStreamCaptureModeThreadLocal));
    rc = enqueue(mm->graph_stream);
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(mm->graph_stream, &g);
    if (rc) {
      if (g) cudaGraphDestroy(g);
      return rc;
    }
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture");
    ge->graph = g;
    VBG_CUDA(cudaGraphInstantiate(&ge->exec, g, 0));
    it = mm->graphs.emplace(key, std::move(ge)).first;
  }
  VBG_CUDA(cudaGraphLaunch(it->second->exec, s));
  return 0;
}

int vbg_spmv_host(const vbg_matrix* m, const void* x, void* y, void* stream) {
  VBG_CHECK(m && x && y, VBG_E_ARG, "null argument");
  cudaStream_t s = as_stream(stream);
  const size_t bytes = (size_t)m->N * elem_size(m->dtype);
  DevBuf dx, dy;
  int rc;
  if ((rc = dx.ensure(bytes))) return rc;
  if ((rc = dy.ensure(bytes))) return rc;
  VBG_CUDA(cudaMemcpyAsync(dx.p, x, bytes, cudaMemcpyHostToDevice, s));
  if ((rc = vbg_spmv(m, dx.p, dy.p, s))) return rc;
  VBG_CUDA(cudaMemcpyAsync(y, dy.p, bytes, cudaMemcpyDeviceToHost, s));
  VBG_CUDA(cudaStreamSynchronize(s));
  return 0;
}

int vbg_spmm_host(const vbg_matrix* m, int k, const void* X, void* Y, void* stream) {
  VBG_CHECK(m && X && Y && k >= 1, VBG_E_ARG, "invalid argument");
  cudaStream_t s = as_stream(stream);
  const size_t es = elem_size(m->dtype);
  const int ld = k == 1 ? 1 : (int)(((k * es + 63) / 64) * 64 / es);
  const size_t bytes = (size_t)m->N * ld * es;
  DevBuf dx, dy;
  int rc;
  if ((rc = dx.ensure(bytes))) return rc;
  if ((rc = dy.ensure(bytes))) return rc;
  if (ld != k) VBG_CUDA(cudaMemsetAsync(dx.p, 0, bytes, s));
  VBG_CUDA(cudaMemcpy2DAsync(dx.p, ld * es, X, k * es, k * es, m->N, cudaMemcpyHostToDevice, s));
  if ((rc = vbg_spmm(m, k, ld, dx.p, dy.p, s))) return rc;
  VBG_CUDA(cudaMemcpy2DAsync(Y, k * es, dy.p, ld * es, k * es, m->N, cudaMemcpyDeviceToHost, s));
  VBG_CUDA(cudaStreamSynchronize(s));
  return 0;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free variant of the fused Chebyshev step.
//
// vbg_cheb_step keeps its per-CTA dot-product partials in scratch that the
// library allocates (cudaMalloc) on first use.  Some callers cannot allow
// any device allocation inside the library call: code that owns the whole
// device memory budget through its own pool or arena, or that runs where an
// allocation would synchronise the device at a point it must not.  For them
// vbg_cheb_step_noalloc takes that scratch from the file-scope array below
// instead.  The array is part of the library image: every GPU that loads the
// library holds it (64 KiB + 256 bytes) until the process exits.
namespace vbg {

// Per-CTA partial sums (two doubles each) for at most this many CTAs, then the
// grid-reduction counter.
constexpr int kNoAllocMaxCtas = 4096;
static __device__ __align__(256) double g_noalloc_scratch[2 * kNoAllocMaxCtas + 32];

// Device address of g_noalloc_scratch per device, looked up once per device.
static int noalloc_scratch(double** out) {
  static std::mutex mu;
  static std::map<int, double*> addr;
  int dev = 0;
  VBG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  auto it = addr.find(dev);
  if (it == addr.end()) {
    void* p = nullptr;
    VBG_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    it = addr.emplace(dev, static_cast<double*>(p)).first;
  }
  *out = it->second;
  return 0;
}

}  // namespace vbg

extern "C" int vbg_cheb_step_noalloc(const vbg_matrix* m, int k, int ld, double alpha, double beta, double gamma,
                                     const void* X, const void* Xprev, void* Y, const void* dot_with, double* dots,
                                     void* acc, double cre, double cim, void* stream) {
  ApplyArgs a;
  cudaStream_t s = as_stream(stream);
  int rc = prepare(m, false, k, ld, a, s);
  if (rc) return rc;
  VBG_CHECK(X && Y, VBG_E_ARG, "null multivector");
  VBG_CHECK(dots, VBG_E_ARG, "vbg_cheb_step_noalloc: dots is required (use vbg_cheb_step without dots)");
  VBG_CHECK(gamma == 0.0 || Xprev, VBG_E_ARG, "Xprev is required when gamma != 0");
  a.alpha = alpha;
  a.beta = beta;
  a.gamma = gamma;
  a.X = X;
  a.Xprev = Xprev;
  a.Y = Y;
  a.dotw = dot_with;
  a.acc = acc;
  a.cre = cre;
  a.cim = cim;
  double* scratch = nullptr;
  if ((rc = noalloc_scratch(&scratch))) return rc;
  unsigned* counter = reinterpret_cast<unsigned*>(scratch + 2 * kNoAllocMaxCtas);
  // the counter must start at zero; the previous call's value is not trusted
  VBG_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned), s));
  a.want_dots = 1;
  a.partials = scratch;
  a.counter = counter;
  a.dots_out = dots;
  // the launcher checks the CTAs it actually starts against this room and
  // rejects the call (VBG_E_ARG) before any launch that would not fit
  a.max_ctas = kNoAllocMaxCtas;
  const int rc2 = launch_apply(m, false, false, a, s, false);
  if (rc2) set_error(std::string("vbg_cheb_step_noalloc: ") + vbg_last_error());
  return rc2;
}
