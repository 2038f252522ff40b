// Row-wise multivector apply on the FP64 tensor cores: Y = A X and Y = A^H X
// with the fused epilogue, real and complex, any block sizes and any leading
// dimension.  It runs what the staged applies (vbg_pipe.cuh, vbg_tile.cuh,
// vbg_dtile.cuh, vbg_chain.cuh) do not take -- the adjoint, blocks over 8,
// leading dimensions that are no lane-group width -- and matrices without
// tiles unless their blocks are small (untiled_choice).
//
// A warp multiplies one task: 8 MT scalar rows of one block row against NP
// column pieces of 128 bytes (16 real or 8 complex columns), by m8n8k4
// products whose A operand is the block's values and whose B operand is the
// block column's X rows, both straight from global memory in fragment order
// (lane l: row l / 4 of A and column pair l / 4 of the piece, inner index
// l % 4).  With columns 2 g and 2 g + 1 of a piece in two accumulator tiles
// (for complex values: real and imaginary parts), a lane loads its X operands
// of a piece as one 16-byte vector and ends up with 32 contiguous bytes of an
// output row.  The next eight inner indices are loaded while these are
// multiplied.  A complex product is four real ones.
//
// What bounds it: the latency of the dependent loads (row range, entry
// records, then values and X) and the L2 traffic of X, not the tensor pipe.
// So every class of block sizes shares one launch (separate launches ran one
// after the other), all 32 lanes work whatever the leading dimension, and a
// block row's entries are split over up to eight warps of the CTA when there
// are too few tasks to fill the SMs (row_split).  Against the scalar
// row-per-warp kernels, one launch per size class, that it replaces
// (5000 block rows of 4-8, 24 columns: forward 270 us and adjoint 373 us of
// five launches each; 4096 rows of 9-16, 16 columns: 175 us, now 54).  The
// whole of the first example's forward, adjoint and value gradient went from
// 590 to 180 us.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "vbg_args.cuh"

namespace vbg {

constexpr int kMmaWarps = 8;

// The A operand of a lane: a real value, or a complex one.
template <typename T> struct MmaA { double re; };
template <> struct MmaA<cplx> { double re, im; };

template <typename T, bool ADJ>
__device__ __forceinline__ MmaA<T> mma_load_a(const T* __restrict__ p) {
  if constexpr (std::is_same<T, cplx>::value) {
    const double2 v = __ldg(reinterpret_cast<const double2*>(p));
    return {v.x, ADJ ? -v.y : v.y};
  } else {
    return {__ldg(p)};
  }
}

// The operands of eight inner indices (two m8n8k4 steps).
template <typename T, int MT, int NP>
struct MmaFrag {
  MmaA<T> a[2][MT];
  double2 b[2][NP];
  bool two;  // the second step has inner indices
};

// acc in memory order of the lane's 32 bytes: {tile 0 c0, tile 1 c0, tile 0
// c1, tile 1 c1}.
template <typename T, int MT, int NP>
__device__ __forceinline__ void mma_step(double (&acc)[MT][NP][4], const MmaFrag<T, MT, NP>& f, int mlive) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (h == 1 && !f.two) break;
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      if (MT > 1 && m >= mlive) break;
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        double(&c)[4] = acc[m][p];
        if constexpr (std::is_same<T, cplx>::value) {
          dmma_884(c[0], c[2], f.a[h][m].re, f.b[h][p].x);
          dmma_884(c[1], c[3], f.a[h][m].re, f.b[h][p].y);
          dmma_884(c[0], c[2], -f.a[h][m].im, f.b[h][p].y);
          dmma_884(c[1], c[3], f.a[h][m].im, f.b[h][p].x);
        } else {
          dmma_884(c[0], c[2], f.a[h][m].re, f.b[h][p].x);
          dmma_884(c[1], c[3], f.a[h][m].re, f.b[h][p].y);
        }
      }
    }
  }
}

// 16 bytes of one output row: E = 2 real or 1 complex elements at element
// offset `el` (vectors) of the multivectors.
template <typename T>
__device__ __forceinline__ void mma_epilogue(const ApplyArgs& a, const double* acc, int64_t el, double& d0,
                                             double& d1) {
  constexpr int E = std::is_same<T, cplx>::value ? 1 : 2;
  struct alignas(16) V {
    T v[E];
  };
  V s, y;
  memcpy(&s, acc, 16);
  auto at = [&](const void* base) { return reinterpret_cast<const V*>(static_cast<const double*>(base) + el); };
  V xs, xp, xd, ac;
  if (a.beta != 0.0 || (a.want_dots && !a.dotw)) xs = *at(a.X);
  if (a.gamma != 0.0) xp = *at(a.Xprev);
  if (a.want_dots) xd = a.dotw ? *at(a.dotw) : xs;
  if (a.acc) ac = *at(a.acc);
#pragma unroll
  for (int u = 0; u < E; ++u) {
    T yy = scal_r(a.alpha, s.v[u]);
    if (a.beta != 0.0) yy = axpy_r(a.beta, xs.v[u], yy);
    if (a.gamma != 0.0) yy = axpy_r(a.gamma, xp.v[u], yy);
    y.v[u] = yy;
    if (a.want_dots) {
      d0 += re_dot(xd.v[u], yy);
      d1 += re_dot(yy, yy);
    }
    if (a.acc) ac.v[u] = cmad(a.cre, a.cim, yy, ac.v[u]);
  }
  if (a.acc) *reinterpret_cast<V*>(static_cast<double*>(a.acc) + el) = ac;
  *reinterpret_cast<V*>(static_cast<double*>(a.Y) + el) = y;
}

// rgroups x cgroups tasks per block row (groups of 8 MT rows, of NP pieces);
// with per-row dots one warp group runs all of a row's tasks in turn.  `split`
// warps share a task: warp `sub` takes its entries sub, sub + split, ... and
// the first one adds the partial tiles in warp order.
template <typename T, int MT, int NP, bool ADJ>
__global__ void __launch_bounds__(kMmaWarps * 32, 2)
    apply_mma_kernel(ApplyArgs a, const T* __restrict__ vals, int rgroups, int cgroups, int split, int part_base,
                     int total) {
  constexpr int W = std::is_same<T, cplx>::value ? 2 : 1;  // doubles per element
  // even and odd fragments are summed apart where the registers allow it
  constexpr bool DUAL = MT * NP == 1;
  extern __shared__ double mma_red[];  // split > 1: kMmaWarps tiles of MT * NP * 4 * 32 doubles
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int64_t ldd = (int64_t)a.ld * W;
  const double* __restrict__ X = static_cast<const double*>(a.X);
  const int per_cta = kMmaWarps / split, sub = warp % split;
  const int parts = rgroups * cgroups, tasks_row = a.row_dots ? 1 : parts;
  const int64_t ntasks = (int64_t)a.n_rows * tasks_row;
  double d0 = 0.0, d1 = 0.0;
  // CTA-uniform trip counts: the split's sums meet at CTA barriers
  for (int64_t tb = (int64_t)blockIdx.x * per_cta; tb < ntasks; tb += (int64_t)gridDim.x * per_cta) {
    const int64_t task = tb + warp / split;
    const bool on = task < ntasks;
    const int row = on ? (int)(task / tasks_row) : 0;
    const int u0 = a.row_dots ? 0 : (int)(task - (int64_t)row * tasks_row);
    const int u1 = a.row_dots ? parts : u0 + 1;
    const int r = on ? a.bsz[row] : 0;
    const int e0 = a.ptr[row], e1 = a.ptr[row + 1];
    double rd0 = 0.0, rd1 = 0.0;
    for (int u = u0; u < u1; ++u) {
      const int rg = u / cgroups, cg = u - rg * cgroups;
      const int o0 = rg * 8 * MT;
      const int64_t c0 = (int64_t)cg * NP * 16;
      const int mlive = (r - o0 + 7) / 8;
      double acc[MT][NP][4];
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
          for (int t = 0; t < 4; ++t) acc[m][p][t] = 0.0;
      double odd[DUAL ? MT : 1][DUAL ? NP : 1][4] = {};
      if (o0 < r) {
        for (int base = e0 + sub; base < e1; base += 32 * split) {
          const int cnt = min(32, (e1 - base + split - 1) / split);
          // lane j's entry: first X element, first value, inner size
          long long xo = 0, vo = 0;
          int in = 0;
          if (lane < cnt) {
            const int e = base + lane * split;
            if (!ADJ && a.slot_meta) {
              const int2 mt = __ldg(a.slot_meta + e);
              xo = mt.x * ldd;
              in = mt.y & 0xff;
              vo = __ldg(a.blk_off + e);
            } else {
              const int src = __ldg(a.ent_src + e);
              xo = a.scal_off[src] * ldd;
              in = a.bsz[src];
              vo = a.blk_off[ADJ ? __ldg(a.ent_slot + e) : e];
            }
          }
          int j = 0, q0 = 0;
          int jin = __shfl_sync(0xffffffffu, in, 0);
          auto load = [&](MmaFrag<T, MT, NP>& f) {
            const double* xb = X + __shfl_sync(0xffffffffu, xo, j) + c0 + 2 * g;
            const T* vb = vals + __shfl_sync(0xffffffffu, vo, j);
            f.two = q0 + 4 < jin;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int q = q0 + 4 * h + t4;
              const bool kv = q < jin;
#pragma unroll
              for (int m = 0; m < MT; ++m) {
                const int o = o0 + 8 * m + g;
                f.a[h][m] = kv && o < r ? mma_load_a<T, ADJ>(vb + (ADJ ? (int64_t)q * r + o : (int64_t)o * jin + q))
                                        : MmaA<T>{};
              }
#pragma unroll
              for (int p = 0; p < NP; ++p)
                f.b[h][p] = kv && c0 + 16 * p + 2 * g < ldd
                                ? __ldg(reinterpret_cast<const double2*>(xb + q * ldd + 16 * p))
                                : make_double2(0.0, 0.0);
            }
          };
          auto next = [&]() {  // to the next eight inner indices; false past the last entry
            q0 += 8;
            if (q0 < jin) return true;
            q0 = 0;
            if (++j >= cnt) return false;
            jin = __shfl_sync(0xffffffffu, in, j);
            return true;
          };
          MmaFrag<T, MT, NP> f0, f1;
          load(f0);
          while (true) {
            bool more = next();
            if (more) load(f1);
            mma_step<T, MT, NP>(acc, f0, mlive);
            if (!more) break;
            more = next();
            if (more) load(f0);
            if constexpr (DUAL) mma_step<T, MT, NP>(odd, f1, mlive);
            else mma_step<T, MT, NP>(acc, f1, mlive);
            if (!more) break;
          }
        }
      }
      if constexpr (DUAL) {
#pragma unroll
        for (int t = 0; t < 4; ++t) acc[0][0][t] += odd[0][0][t];
      }
      if (split > 1) {
        double* mine = mma_red + (size_t)warp * (MT * NP * 4 * 32) + lane;
        if (sub > 0) {
#pragma unroll
          for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int p = 0; p < NP; ++p)
#pragma unroll
              for (int t = 0; t < 4; ++t) mine[((m * NP + p) * 4 + t) * 32] = acc[m][p][t];
        }
        __syncthreads();
        if (sub == 0)
          for (int w = 1; w < split; ++w) {
            const double* o = mine + (size_t)w * (MT * NP * 4 * 32);
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
              for (int p = 0; p < NP; ++p)
#pragma unroll
                for (int t = 0; t < 4; ++t) acc[m][p][t] += o[((m * NP + p) * 4 + t) * 32];
          }
        __syncthreads();
      }
      if (sub == 0 && o0 < r) {
        const int64_t y0 = a.scal_off[row];
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const int o = o0 + 8 * m + g;
          if (o >= r) continue;
#pragma unroll
          for (int p = 0; p < NP; ++p)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
              const int64_t c = c0 + 16 * p + 4 * t4 + 2 * hh;
              if (c < ldd) mma_epilogue<T>(a, &acc[m][p][2 * hh], (y0 + o) * ldd + c, rd0, rd1);
            }
        }
      }
    }
    if (a.want_dots) {
      if (!a.row_dots) {
        d0 += rd0;
        d1 += rd1;
      } else if (on && sub == 0) {
        write_row_dots(a.row_dots, row, rd0, rd1);
      }
    }
  }
  if (a.want_dots && !a.row_dots) grid_reduce2(d0, d1, a.partials, a.counter, a.dots_out, part_base, total);
}

template <typename T, int MT, int NP, bool ADJ>
static int launch_mma_k(const vbg_matrix* m, const ApplyArgs& a, const T* vals, cudaStream_t s) {
  constexpr int W = std::is_same<T, cplx>::value ? 2 : 1;
  constexpr size_t kRed = (size_t)kMmaWarps * MT * NP * 4 * 32 * sizeof(double);
  static int per_sm[kMaxDevices][2] = {};  // resident CTAs without / with the split's scratch
  const int rgroups = (m->max_bs + 8 * MT - 1) / (8 * MT);
  const int cgroups = (int)(((int64_t)a.ld * W + 16 * NP - 1) / (16 * NP));
  const int64_t ntasks = (int64_t)a.n_rows * (a.row_dots ? 1 : (int64_t)rgroups * cgroups);
  const int split = row_split(m, ntasks);
  const int dev = current_device();
  int& occ = per_sm[dev][split > 1];
  if (!occ) {
    VBG_CUDA(cudaFuncSetAttribute(apply_mma_kernel<T, MT, NP, ADJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kRed));
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, apply_mma_kernel<T, MT, NP, ADJ>, kMmaWarps * 32,
                                                      split > 1 ? kRed : 0) != cudaSuccess ||
        b < 1)
      b = 1;
    occ = b;
  }
  const int per_cta = kMmaWarps / split;
  const int grid =
      (int)std::max<int64_t>(1, std::min<int64_t>((ntasks + per_cta - 1) / per_cta, (int64_t)occ * sm_count()));
  if (int rc = check_dot_ctas(a, grid)) return rc;
  apply_mma_kernel<T, MT, NP, ADJ>
      <<<grid, kMmaWarps * 32, split > 1 ? kRed : 0, s>>>(a, vals, rgroups, cgroups, split, 0, grid);
  VBG_CUDA(cudaGetLastError());
  return 0;
}

// Blocks over 8 take two row tiles per warp (their X operands are loaded once
// for 16 rows); multivectors over one 128-byte piece take two pieces.
template <typename T, bool ADJ>
static int launch_mma_t(const vbg_matrix* m, const ApplyArgs& a, const T* vals, cudaStream_t s) {
  const bool wide = m->max_bs > 8, two = (int64_t)a.ld * sizeof(T) > 128;
  if (wide) return two ? launch_mma_k<T, 2, 2, ADJ>(m, a, vals, s) : launch_mma_k<T, 2, 1, ADJ>(m, a, vals, s);
  return two ? launch_mma_k<T, 1, 2, ADJ>(m, a, vals, s) : launch_mma_k<T, 1, 1, ADJ>(m, a, vals, s);
}

int launch_mma(const vbg_matrix* m, bool adj, const ApplyArgs& a, cudaStream_t s) {
  if (m->dtype == VBG_C128) {
    const cplx* v = m->vals.as<cplx>();
    return adj ? launch_mma_t<cplx, true>(m, a, v, s) : launch_mma_t<cplx, false>(m, a, v, s);
  }
  const double* v = m->vals.as<double>();
  return adj ? launch_mma_t<double, true>(m, a, v, s) : launch_mma_t<double, false>(m, a, v, s);
}

}  // namespace vbg
