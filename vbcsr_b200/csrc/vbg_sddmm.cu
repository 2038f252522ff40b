// Pattern-restricted outer products (SDDMM) for the gradients of the sparse
// apply: out_ij += alpha * G_i X_j^H over the stored blocks (i, j) of A, with
// G_i the r rows of G at block row i and X_j the c rows of X at block column
// j (k columns each).  For Y = A X and a real loss with dL/dY* = G this is
// dL/dA* restricted to A's pattern, the term a hand-written backward of the
// apply (and of the Chebyshev recurrence built on it) needs; the reference
// has no gradients, so there is no reference routine to mirror.
//
// Layout: `out` has A's value layout (slot order, r x c row-major blocks);
// G and X are row-major multivectors with leading dimension ld (ld = 1: plain
// vectors).  A warp takes the stored blocks of one block row (every split-th
// of them when the rows are too few to fill the SMs) and forms each as 8 x 8
// tiles on the FP64 tensor cores (m8n8k4): lane l holds row l / 4 of G_i and
// row l / 4 of X_j, both read in fragment order straight from global memory
// -- for real values two neighbouring columns per lane as one 16-byte vector
// (the sum runs over the columns in any order, so the two go to two steps),
// for complex ones one element.  A complex tile step is four real ones.  The
// G rows stay in L1.  What bounds it is the latency of those loads: staging
// the rows in shared memory and reducing each value's products in one lane
// spent ten times the instructions (126k complex blocks, 16 columns: 123 us,
// now 67; 65k real blocks, 24 columns: 88 us, now 37).  A block row's slots are written by
// one warp each, so the read-modify-write of `out` needs no atomics.
#include <algorithm>
#include <type_traits>

#include "vbg_args.cuh"

namespace vbg {

constexpr int kSddmmWarps = 8;

__device__ __forceinline__ double mul_s(double a, double b) { return a * b; }
__device__ __forceinline__ cplx mul_s(cplx a, cplx b) { return {fma(a.re, b.re, -a.im * b.im), fma(a.re, b.im, a.im * b.re)}; }
template <typename T> __device__ __forceinline__ T scalar_from(double re, double im);
template <> __device__ __forceinline__ double scalar_from<double>(double re, double) { return re; }
template <> __device__ __forceinline__ cplx scalar_from<cplx>(double re, double im) { return {re, im}; }

// V2: rows of G and X start on 16-byte boundaries (two real columns or a
// complex element per load).
template <typename T, bool V2>
__global__ void __launch_bounds__(kSddmmWarps * 32, 4)
    sddmm_kernel(int n_rows, const int* __restrict__ row_ptr, const int* __restrict__ col_ind,
                 const int* __restrict__ bsz, const int64_t* __restrict__ scal_off,
                 const int64_t* __restrict__ blk_off, int k, int ld, const T* __restrict__ G,
                 const T* __restrict__ X, double are, double aim, int split, T* __restrict__ out) {
  constexpr bool CX = std::is_same<T, cplx>::value;
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const T alpha = scalar_from<T>(are, aim);
  const int64_t nw = (int64_t)n_rows * split;
  for (int64_t w = (int64_t)blockIdx.x * kSddmmWarps + (threadIdx.x >> 5); w < nw;
       w += (int64_t)gridDim.x * kSddmmWarps) {
    const int i = (int)(w / split), sub = (int)(w - (int64_t)i * split);
    const int r = bsz[i];
    const T* Gi = G + scal_off[i] * (int64_t)ld;
    const int e0 = row_ptr[i] + sub, e1 = row_ptr[i + 1];
    for (int base = e0; base < e1; base += 32 * split) {
      const int cnt = min(32, (e1 - base + split - 1) / split);
      long long xo = 0, oo = 0;
      int cj = 0;
      if (lane < cnt) {
        const int e = base + lane * split;
        const int j = __ldg(col_ind + e);
        xo = scal_off[j] * (long long)ld;
        cj = bsz[j];
        oo = blk_off[e];
      }
      for (int jj = 0; jj < cnt; ++jj) {
        const T* Xj = X + __shfl_sync(0xffffffffu, xo, jj);
        T* ob = out + __shfl_sync(0xffffffffu, oo, jj);
        const int c = __shfl_sync(0xffffffffu, cj, jj);
        for (int m0 = 0; m0 < r; m0 += 8)
          for (int n0 = 0; n0 < c; n0 += 8) {
            // rows past the block repeat its last one: their results are not
            // stored
            const T* gp = Gi + (int64_t)min(m0 + g, r - 1) * ld;
            const T* xp = Xj + (int64_t)min(n0 + g, c - 1) * ld;
            T acc[2] = {zero_s<T>(), zero_s<T>()};
            if constexpr (CX) {
#pragma unroll 4
              for (int t = t4; t < k + t4; t += 4) {  // warp-uniform trip count
                double2 a = make_double2(0.0, 0.0), b = a;
                if (t < k) {
                  if constexpr (V2) {
                    a = __ldg(reinterpret_cast<const double2*>(gp + t));
                    b = __ldg(reinterpret_cast<const double2*>(xp + t));
                  } else {
                    const T av = gp[t], bv = xp[t];
                    a = make_double2(av.re, av.im);
                    b = make_double2(bv.re, bv.im);
                  }
                }
                // G conj(X)
                dmma_884(acc[0].re, acc[1].re, a.x, b.x);
                dmma_884(acc[0].im, acc[1].im, a.y, b.x);
                dmma_884(acc[0].re, acc[1].re, a.y, b.y);
                dmma_884(acc[0].im, acc[1].im, -a.x, b.y);
              }
            } else {
#pragma unroll 4
              for (int t0 = 0; t0 < k; t0 += 8) {
                const int t = t0 + 2 * t4;
                double2 a = make_double2(0.0, 0.0), b = a;
                if (V2 && t + 1 < k) {
                  a = __ldg(reinterpret_cast<const double2*>(gp + t));
                  b = __ldg(reinterpret_cast<const double2*>(xp + t));
                } else {
                  if (t < k) {
                    a.x = __ldg(gp + t);
                    b.x = __ldg(xp + t);
                  }
                  if (t + 1 < k) {
                    a.y = __ldg(gp + t + 1);
                    b.y = __ldg(xp + t + 1);
                  }
                }
                dmma_884(acc[0], acc[1], a.x, b.x);
                dmma_884(acc[0], acc[1], a.y, b.y);
              }
            }
            const int o = m0 + g, q = n0 + 2 * t4;
            if (o < r) {
              T* p = ob + (int64_t)o * c + q;
              if (q < c) p[0] = p[0] + mul_s(alpha, acc[0]);
              if (q + 1 < c) p[1] = p[1] + mul_s(alpha, acc[1]);
            }
          }
      }
    }
  }
}

// The same for blocks of at most 8 x 8 and at most 32 real or 16 complex
// columns: a row's G operands stay in registers, and the X operands and old
// output values of several blocks are loaded before their products -- the
// general form waits for each block's rows, then for its output.
// F: 16-byte operands per lane.  At one operand (8 real, 4 complex columns) four
// CTAs share an SM instead of two.
constexpr int kSddmmFrags = 4;

template <typename T, bool V2, int F>
__global__ void __launch_bounds__(kSddmmWarps * 32, F == 1 ? 4 : 2)
    sddmm_small_kernel(int n_rows, const int* __restrict__ row_ptr, const int* __restrict__ col_ind,
                       const int* __restrict__ bsz, const int64_t* __restrict__ scal_off,
                       const int64_t* __restrict__ blk_off, int k, int ld, const T* __restrict__ G,
                       const T* __restrict__ X, double are, double aim, int split, T* __restrict__ out) {
  constexpr bool CX = std::is_same<T, cplx>::value;
  constexpr int KF = CX ? 4 : 8;                   // columns per operand
  constexpr int B = CX ? 2 : 3;                     // blocks in flight
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const T alpha = scalar_from<T>(are, aim);
  const int64_t nw = (int64_t)n_rows * split;
  // the lane's columns of row p
  auto frags = [&](const T* p, double2(&f)[F]) {
#pragma unroll
    for (int u = 0; u < F; ++u) {
      f[u] = make_double2(0.0, 0.0);
      if (u * KF >= k) continue;
      if constexpr (CX) {
        const int t = u * KF + t4;
        if (t < k) {
          if constexpr (V2) {
            f[u] = __ldg(reinterpret_cast<const double2*>(p + t));
          } else {
            const T v = p[t];
            f[u] = make_double2(v.re, v.im);
          }
        }
      } else {
        const int t = u * KF + 2 * t4;
        if (V2 && t + 1 < k) {
          f[u] = __ldg(reinterpret_cast<const double2*>(p + t));
        } else {
          if (t < k) f[u].x = __ldg(p + t);
          if (t + 1 < k) f[u].y = __ldg(p + t + 1);
        }
      }
    }
  };
  for (int64_t w = (int64_t)blockIdx.x * kSddmmWarps + (threadIdx.x >> 5); w < nw;
       w += (int64_t)gridDim.x * kSddmmWarps) {
    const int i = (int)(w / split), sub = (int)(w - (int64_t)i * split);
    const int r = bsz[i];
    const int e0 = row_ptr[i] + sub, e1 = row_ptr[i + 1];
    double2 a[F];
    // rows past the block repeat its last one: their results are not stored
    frags(G + (scal_off[i] + min(g, r - 1)) * (int64_t)ld, a);
    for (int base = e0; base < e1; base += 32 * split) {
      const int cnt = min(32, (e1 - base + split - 1) / split);
      long long xo = 0, oo = 0;
      int cj = 1;
      if (lane < cnt) {
        const int e = base + lane * split;
        const int j = __ldg(col_ind + e);
        xo = scal_off[j];
        cj = bsz[j];
        oo = blk_off[e];
      }
      for (int j0 = 0; j0 < cnt; j0 += B) {
        double2 b[B][F];
        T v[B][2];
        T* p[B];
        int c[B];
        // the X operands and old values of B blocks, then their products
#pragma unroll
        for (int u = 0; u < B; ++u) {
          c[u] = 0;
          if (j0 + u >= cnt) continue;
          c[u] = __shfl_sync(0xffffffffu, cj, j0 + u);
          frags(X + (__shfl_sync(0xffffffffu, xo, j0 + u) + min(g, c[u] - 1)) * (int64_t)ld, b[u]);
          p[u] = out + __shfl_sync(0xffffffffu, oo, j0 + u) + g * c[u] + 2 * t4;
          v[u][0] = g < r && 2 * t4 < c[u] ? p[u][0] : zero_s<T>();
          v[u][1] = g < r && 2 * t4 + 1 < c[u] ? p[u][1] : zero_s<T>();
        }
#pragma unroll
        for (int u = 0; u < B; ++u) {
          if (j0 + u >= cnt) continue;
          T acc[2] = {zero_s<T>(), zero_s<T>()};
#pragma unroll
          for (int f = 0; f < F; ++f) {
            if (f * KF >= k) break;
            if constexpr (CX) {  // G conj(X)
              dmma_884(acc[0].re, acc[1].re, a[f].x, b[u][f].x);
              dmma_884(acc[0].im, acc[1].im, a[f].y, b[u][f].x);
              dmma_884(acc[0].re, acc[1].re, a[f].y, b[u][f].y);
              dmma_884(acc[0].im, acc[1].im, -a[f].x, b[u][f].y);
            } else {
              dmma_884(acc[0], acc[1], a[f].x, b[u][f].x);
              dmma_884(acc[0], acc[1], a[f].y, b[u][f].y);
            }
          }
          if (g < r) {
            if (2 * t4 < c[u]) p[u][0] = v[u][0] + mul_s(alpha, acc[0]);
            if (2 * t4 + 1 < c[u]) p[u][1] = v[u][1] + mul_s(alpha, acc[1]);
          }
        }
      }
    }
  }
}

template <typename T, bool V2>
static int launch_sddmm(const vbg_matrix* m, int k, int ld, const void* G, const void* X, double are, double aim,
                        void* out, cudaStream_t s) {
  const int kf = std::is_same<T, cplx>::value ? 4 : 8;
  const bool small = m->max_bs <= 8 && k <= kSddmmFrags * kf, one = small && k <= kf;
  int split = 1;
  if (small) {
    // a row's blocks go to several warps while all are resident at once; two
    // when the rows make one to four rounds of them, so that the last round
    // ends together (us, split 1 / 2 / 4, blocks of 2-4, 32 columns: 500 rows 14
    // / 9 / 8, 1000 of 4-8 15 / 11 / 13, 2000 15 / 17 / 19, 5000 35 / 33 / 37,
    // 12000 64 / 64 / 78)
    const int64_t wave = (int64_t)sm_count() * 16;
    if (m->n <= wave) {
      while (split < 4 && 2 * (int64_t)m->n * split <= wave && m->nnzb >= 4 * (int64_t)split * m->n) split *= 2;
    } else if (m->n < 4 * wave && m->nnzb >= 4 * (int64_t)m->n) {
      split = 2;
    }
  } else {
    // several tasks per resident warp, so that the last ones end together
    while (split < 4 && (int64_t)m->n * split < (int64_t)sm_count() * 128 && m->nnzb >= 4 * (int64_t)split * m->n)
      split *= 2;
  }
  const int64_t want = ((int64_t)m->n * split + kSddmmWarps - 1) / kSddmmWarps;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)sm_count() * 8));
  auto* kernel = one ? sddmm_small_kernel<T, V2, 1> : small ? sddmm_small_kernel<T, V2, kSddmmFrags> : sddmm_kernel<T, V2>;
  kernel<<<grid, kSddmmWarps * 32, 0, s>>>(
      m->n, m->row_ptr.as<int>(), m->col_ind.as<int>(), m->bsz.as<int>(), m->scal_off.as<int64_t>(),
      m->blk_off.as<int64_t>(), k, ld, static_cast<const T*>(G), static_cast<const T*>(X), are, aim, split,
      static_cast<T*>(out));
  VBG_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace vbg

using namespace vbg;

extern "C" int vbg_sddmm(const vbg_matrix* m, int k, int ld, const void* G, const void* X, double alpha_re,
                         double alpha_im, void* out, void* stream) {
  VBG_CHECK(m, VBG_E_ARG, "null matrix");
  VBG_CHECK(k >= 1 && ld >= k, VBG_E_ARG, "invalid k / ld");
  VBG_CHECK((G && X && out) || m->nnz == 0, VBG_E_ARG, "null argument");
  if (m->n == 0 || m->nnz == 0) return 0;
  cudaStream_t s = as_stream(stream);
  const bool aligned = reinterpret_cast<uintptr_t>(G) % 16 == 0 && reinterpret_cast<uintptr_t>(X) % 16 == 0;
  if (m->dtype == VBG_C128)
    return aligned ? launch_sddmm<cplx, true>(m, k, ld, G, X, alpha_re, alpha_im, out, s)
                   : launch_sddmm<cplx, false>(m, k, ld, G, X, alpha_re, alpha_im, out, s);
  const bool v2 = ld % 2 == 0 && aligned;
  return v2 ? launch_sddmm<double, true>(m, k, ld, G, X, alpha_re, alpha_im, out, s)
            : launch_sddmm<double, false>(m, k, ld, G, X, alpha_re, alpha_im, out, s);
}
