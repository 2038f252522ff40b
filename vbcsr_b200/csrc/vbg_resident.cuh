// Chebyshev recurrences of plain vectors with the matrix resident in shared
// memory.  Included by vbg_apply.cu inside namespace vbg, after vbg_pipe.cuh
// (it uses the status word and the clock).
//
// A recurrence y_{s} = alpha_s A y_{s-1} + beta_s y_{s-1} + gamma_s y_{s-2}
// (+ c_s g) of a few hundred steps on a matrix whose values fit the SMs'
// shared memory (148 x 227 KB) reads the same 30 MB from L2 at every step when
// each step is a launch of its own, and pays a launch and its tail per step:
// 14.5 us a step on a 60 x 60 lattice with complex values (28.7 MB).  Here
// one cooperative launch runs all steps: a CTA per SM copies the values of
// its block rows into shared memory once (as r x K panels, K the scalar
// columns of the row's blocks side by side), and per step gathers the X
// elements its rows read (each once, about 860 on that lattice), multiplies
// out of shared memory and meets the other CTAs at a barrier.  What bounds a
// step is that barrier (4.4k cycles), the gather's L2 latency (2.3k) and the
// rows' chains of loads, multiply-adds and shuffles (about 10k); 256 steps on
// that lattice take 2.2 ms, 3.7 ms as launches.
//
// S = 8 lanes share a scalar row of a block row of at most 4 rows, S = 4 of
// one of at most 8: every lane of the row's group takes every S-th column.
//
// The plan (resident_plan) is made on the host once per structure and
// direction: contiguous block rows per CTA with about equal values, the
// elements of X each CTA reads, and their places for every column of its
// rows.  A matrix whose share does not fit, or with blocks over 8, has none.
//
// Waits at the barrier are bounded (kResPolls): a CTA that gives up sets
// bit 0 of g_pipe_status and the abort bit of the arrival word, at which the
// others leave too.

// Threads of a CTA: 1024 would leave 64 registers each, and what they spill
// goes to L2, since the panels leave hardly any L1 (10.7 and, with the chains
// of ResAcc, 16.6 us a step against 8.7).
constexpr int kResThreads = 512;
constexpr size_t kResSmemMax = 226 * 1024;
constexpr int kResMinSteps = 4;   // fewer steps do not repay the copy of the values
constexpr int kResRowsPerCta = 8; // fewest block rows a CTA is used for
// A plan costs the host about 60 us and 3.5 ns a block, a resident step saves 3 to
// 6 us: it is made when a matrix has run this many steps of recurrences and one
// more for every so many blocks (made at once, the first series of 5 terms on a
// 60 x 60 lattice took 1.1 ms instead of 0.27).
constexpr int kResPlanSteps = 12;
constexpr int kResPlanBlocks = 1500;

// Per step {alpha, beta, gamma, re c, im c}.
constexpr int kResCoef = 5;

struct ResidentArgs {
  // plan: per CTA {first block row, end, first X list entry, X list entries},
  // {values, places, first place, 0}; per block row {first value in the CTA's
  // panel, K, first place, block size}, {place of its own first X element,
  // first scalar row, 0, 0}
  const int4* cta;
  const int4* rows;
  const int* xlist;
  const unsigned short* place;
  // entries of a row (row_ptr / csc_ptr), their slot (nullptr: the entry) and
  // source block
  const int* ptr;
  const int* ent_slot;
  const int* ent_src;
  const int* bsz;
  const int64_t* blk_off;
  // recurrence
  const void* x0;      // y_{-1}
  const void* x1;      // y_{-2} (nullptr: zero)
  void* xch[2];        // y_s goes to xch[s & 1]
  const double* coef;  // steps x kResCoef
  int steps;
  const void* source;  // g (nullptr: none)
  void* psi;           // psi += c_s y_s (nullptr: none; not with a source)
  // columns of a row-major matrix: y_s to column col0 + (s + 1) dcol and x0 to
  // col0, where that lies in [0, ncol)
  void* cols;
  int64_t ldc;
  int col0, dcol, ncol;
  // checkpoints of a series (vbg_cheb_series): t_n = y_{n - 1}
  void* ckpt;
  int K, M;
  int64_t N;
  unsigned* sync;      // arrivals, zeroed
};

// A sum of products in independent chains.
template <typename T> struct ResAcc {
  double s = 0.0;
  __device__ __forceinline__ void add(double a, double x) { s = fma(a, x, s); }
  __device__ __forceinline__ double sum() const { return s; }
};
template <> struct ResAcc<cplx> {
  double rr = 0.0, ii = 0.0, ri = 0.0, ir = 0.0;
  __device__ __forceinline__ void add(cplx a, cplx x) {
    rr = fma(a.re, x.re, rr);
    ii = fma(a.im, x.im, ii);
    ri = fma(a.re, x.im, ri);
    ir = fma(a.im, x.re, ir);
  }
  __device__ __forceinline__ cplx sum() const { return {rr - ii, ri + ir}; }
};

__device__ __forceinline__ double res_ld(const double* p) { return __ldcg(p); }
__device__ __forceinline__ cplx res_ld(const cplx* p) {
  // vectors of complex elements need not start on a 16-byte boundary
  const double* d = reinterpret_cast<const double*>(p);
  return {__ldcg(d), __ldcg(d + 1)};
}

// All CTAs of the launch; false when the wait ran out or another CTA gave up
// (kResAbort set in the arrival word: one load polls both).  The wait is
// bounded by polls, about a microsecond each at most: reading a clock in the
// loop would cost as much as the rest of the barrier.
constexpr unsigned kResAbort = 0x80000000u;
constexpr int kResPolls = 1 << 21;
__device__ __forceinline__ bool res_barrier(unsigned* sync, unsigned target) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(sync, 1u);
    int ok = 0;
    for (int k = 0; k < kResPolls; ++k) {
      unsigned seen;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(seen) : "l"(sync) : "memory");
      if (seen & kResAbort) break;
      if (seen >= target) {
        ok = 1;
        break;
      }
    }
    if (!ok) {
      atomicOr(sync, kResAbort);
      atomicOr(&g_pipe_status, 1u);
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

template <typename T, bool ADJ>
__global__ void __launch_bounds__(kResThreads, 1) resident_kernel(ResidentArgs a, const T* __restrict__ vals) {
  extern __shared__ __align__(16) unsigned char res_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = kResThreads / 32;
  const int4 c0 = a.cta[2 * blockIdx.x], c1 = a.cta[2 * blockIdx.x + 1];
  const int row0 = c0.x, nrows = c0.y - c0.x, nx = c0.w;
  T* A = reinterpret_cast<T*>(res_raw);
  T* xs = A + c1.x;
  int4* rec = reinterpret_cast<int4*>(res_raw + (((size_t)c1.x + nx) * sizeof(T) + 15) / 16 * 16);
  unsigned short* place = reinterpret_cast<unsigned short*>(rec + 2 * (size_t)nrows);
  for (int t = threadIdx.x; t < 2 * nrows; t += kResThreads) rec[t] = a.rows[2 * (size_t)row0 + t];
  for (int t = threadIdx.x; t < c1.y; t += kResThreads) place[t] = a.place[c1.z + t];
  __syncthreads();
  // the rows' values, block by block, into the panels
  for (int li = warp; li < nrows; li += warps) {
    const int4 rr = rec[2 * li];
    const int r = rr.w, e0 = a.ptr[row0 + li], e1 = a.ptr[row0 + li + 1];
    int kbase = 0;
    for (int base = e0; base < e1; base += 32) {
      const int cnt = min(32, e1 - base);
      int c = 0;
      long long vo = 0;
      if (lane < cnt) {
        const int e = base + lane;
        c = a.bsz[a.ent_src[e]];
        vo = a.blk_off[ADJ ? a.ent_slot[e] : e];
      }
      int ko = c;  // inclusive scan of the entries' columns
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, ko, off);
        if (lane >= off) ko += v;
      }
      const int tot = __shfl_sync(0xffffffffu, ko, 31);
      ko += kbase - c;
      kbase += tot;
#pragma unroll 2
      for (int j = 0; j < cnt; ++j) {
        const int jc = __shfl_sync(0xffffffffu, c, j), jk = __shfl_sync(0xffffffffu, ko, j);
        const T* v = vals + __shfl_sync(0xffffffffu, vo, j);
        T* p = A + rr.x + jk;
        for (int i = lane; i < r * jc; i += 32) {
          // block element i: forward (o, q) of r x jc; adjoint (q, o) of jc x r
          const int hi = i / (ADJ ? r : jc), lo = i - hi * (ADJ ? r : jc);
          const int o = ADJ ? lo : hi, q = ADJ ? hi : lo;
          p[o * rr.y + q] = ADJ ? conj_s(v[i]) : v[i];
        }
      }
    }
  }
  const T* x = static_cast<const T*>(a.x0);
  const T* prev = static_cast<const T*>(a.x1);
  for (int s = 0; s < a.steps; ++s) {
    T* y = static_cast<T*>(a.xch[s & 1]);
    for (int t = threadIdx.x; t < nx; t += kResThreads) xs[t] = res_ld(x + __ldg(a.xlist + c0.z + t));
    const double* cf = a.coef + (size_t)kResCoef * s;
    const double alpha = __ldg(cf), beta = __ldg(cf + 1), gamma = __ldg(cf + 2), cre = __ldg(cf + 3),
                 cim = __ldg(cf + 4);
    const int n = s + 1, col = a.col0 + n * a.dcol;
    // the epilogue's operands (y_{s-2}, and the source or psi) of the warp's
    // first row, and in the loop of its next: their latency is behind the
    // gather or the row before
    const T* extra = static_cast<const T*>(a.source ? a.source : a.psi);
    T xp = zero_s<T>(), ex = xp;
    auto fetch = [&](int li, T& wp, T& we) {
      if (li >= nrows) return;
      const int r = rec[2 * li].w, S = r <= 4 ? 8 : 4, o = lane / S;
      if (o >= r || (lane & (S - 1))) return;
      const int64_t gi = (int64_t)rec[2 * li + 1].y + o;
      if (gamma != 0.0 && prev) wp = res_ld(prev + gi);
      if (extra) we = res_ld(extra + gi);
    };
    if (s > 0) fetch(warp, xp, ex);
    __syncthreads();  // the panels (first step) and this step's X
    if (s == 0) fetch(warp, xp, ex);
    for (int li = warp; li < nrows; li += warps) {
      const int4 rr = rec[2 * li], ro = rec[2 * li + 1];
      const int r = rr.w, K = rr.y;
      const int S = r <= 4 ? 8 : 4, o = lane / S, sl = lane & (S - 1);
      const bool on = o < r, lead = on && sl == 0;
      const int64_t gi = (int64_t)ro.y + o;
      T nxp = zero_s<T>(), nex = nxp;
      fetch(li + warps, nxp, nex);
      T acc = zero_s<T>();
      if (on) {
        // chains of their own for every second column and, complex, for the
        // two products of a part
        const T* ap = A + rr.x + o * K;
        const unsigned short* pl = place + rr.z;
        ResAcc<T> c0, c1;
        int k = sl;
#pragma unroll 2
        for (; k + S < K; k += 2 * S) {
          const T xa = xs[pl[k]], xb = xs[pl[k + S]];
          c0.add(ap[k], xa);
          c1.add(ap[k + S], xb);
        }
        if (k < K) c0.add(ap[k], xs[pl[k]]);
        acc = add_s(c0.sum(), c1.sum());
      }
      acc = add_s(acc, shfl_xor_s(acc, 1));
      acc = add_s(acc, shfl_xor_s(acc, 2));
      if (S == 8) acc = add_s(acc, shfl_xor_s(acc, 4));
      if (lead) {
        const T xo = xs[ro.x + o];
        T v = scal_r(alpha, acc);
        if (beta != 0.0) v = axpy_r(beta, xo, v);
        if (gamma != 0.0) v = axpy_r(gamma, xp, v);
        if (a.source) v = cmad(cre, cim, ex, v);
        y[gi] = v;
        if (a.psi) static_cast<T*>(a.psi)[gi] = cmad(cre, cim, v, ex);
        if (a.cols) {
          T* cp = static_cast<T*>(a.cols) + gi * a.ldc;
          if (s == 0 && a.col0 >= 0 && a.col0 < a.ncol) cp[a.col0] = xo;
          if (col >= 0 && col < a.ncol) cp[col] = v;
        }
        if (a.K > 0) {
          T* ck = static_cast<T*>(a.ckpt);
          if (n % a.K == 0) ck[(2 * (int64_t)(n / a.K) - 2) * a.N + gi] = v;
          if ((n + 1) % a.K == 0 && n + 1 < a.M) ck[(2 * (int64_t)((n + 1) / a.K) - 1) * a.N + gi] = v;
        }
      }
      xp = nxp;
      ex = nex;
    }
    if (s + 1 == a.steps) break;
    if (!res_barrier(a.sync, (unsigned)(s + 1) * gridDim.x)) return;
    prev = x;
    x = y;
  }
}

// Shared memory of one CTA.
static size_t res_smem(int64_t nvals, int64_t nx, int64_t nplace, int64_t nrows, size_t es) {
  return ((size_t)(nvals + nx) * es + 15) / 16 * 16 + (size_t)nrows * 32 + (size_t)nplace * 2;
}

// The plan of matrix m for its own rows (adj = false) or its columns, or
// nullptr when there is none; built on first use.
static int resident_plan(const vbg_matrix* cm, bool adj, cudaStream_t s, ResidentPlan** out) {
  auto* m = const_cast<vbg_matrix*>(cm);
  *out = nullptr;
  auto& slot = m->resident[adj ? 1 : 0];
  if (slot) {
    if (slot->grid > 0) *out = slot.get();
    return 0;
  }
  auto plan = std::make_unique<ResidentPlan>();
  const int n = m->n;
  const size_t es = elem_size(m->dtype);
  const int sms = sm_count();
  if (n == 0 || m->max_bs > 8 || m->N >= (int64_t)INT32_MAX || m->nnz * es > kResSmemMax * sms) {
    slot = std::move(plan);
    return 0;
  }
  int rc = ensure_host_structure(m, s);
  if (rc) return rc;
  const std::vector<int>& bsz = m->h_bsz;
  // entries of every output row: row_ptr / col_ind, or the column view (rows
  // ascending, as ensure_csc's)
  std::vector<int> cptr, crow;
  const std::vector<int>*ptr = &m->h_row_ptr, *src = &m->h_col_ind;
  if (adj) {
    cptr.assign(n + 1, 0);
    crow.resize(m->nnzb);
    for (int64_t e = 0; e < m->nnzb; ++e) ++cptr[m->h_col_ind[e] + 1];
    for (int j = 0; j < n; ++j) cptr[j + 1] += cptr[j];
    std::vector<int> at(cptr.begin(), cptr.end() - 1);
    for (int i = 0; i < n; ++i)
      for (int e = m->h_row_ptr[i]; e < m->h_row_ptr[i + 1]; ++e) crow[at[m->h_col_ind[e]]++] = i;
    ptr = &cptr;
    src = &crow;
  }
  const int ctas = std::max(1, std::min(sms, n / kResRowsPerCta));
  std::vector<int4> h_cta(2 * (size_t)ctas), h_rows(2 * (size_t)n);
  std::vector<int> h_x, where(n, -1), stamp(n, -1);
  int64_t places = 0;  // scalar columns over all rows
  for (const int j : *src) places += bsz[j];
  std::vector<unsigned short> h_place(places);
  h_x.reserve((size_t)m->N * 4);
  int64_t done = 0;
  size_t smem = 0;
  bool fits = places < (int64_t)INT32_MAX;
  int row = 0, p_at = 0;
  for (int b = 0; b < ctas && fits; ++b) {
    const int first = row;
    const int x_first = (int)h_x.size(), p_first = p_at;
    int64_t nv = 0;
    auto use = [&](int j) {  // place of block j's X elements in this CTA's list
      if (stamp[j] != b) {
        stamp[j] = b;
        where[j] = (int)h_x.size() - x_first;
        const int x0 = (int)m->h_scal_off[j];
        for (int q = 0; q < bsz[j]; ++q) h_x.push_back(x0 + q);
      }
      return where[j];
    };
    // rows until this CTA's share of the values is reached (the last takes
    // the rest), leaving a row for each CTA to come
    while (row < n && (b + 1 == ctas || ((done * ctas < (int64_t)(b + 1) * m->nnz || row == first) &&
                                         n - row > ctas - 1 - b))) {
      const int own = use(row), p_row = p_at - p_first;
      unsigned short* pp = h_place.data() + p_at;
      for (int e = (*ptr)[row]; e < (*ptr)[row + 1]; ++e) {
        const int j = (*src)[e], w0 = use(j), w1 = w0 + bsz[j];
        for (int w = w0; w < w1; ++w) *pp++ = (unsigned short)w;
      }
      const int64_t K = pp - (h_place.data() + p_at);
      p_at += (int)K;
      h_rows[2 * (size_t)row] = make_int4((int)nv, (int)K, p_row, bsz[row]);
      h_rows[2 * (size_t)row + 1] = make_int4(own, (int)m->h_scal_off[row], 0, 0);
      nv += K * bsz[row];
      done += K * bsz[row];
      ++row;
      if (nv * (int64_t)es > (int64_t)kResSmemMax) break;
    }
    const int nx = (int)h_x.size() - x_first, np = p_at - p_first;
    h_cta[2 * (size_t)b] = make_int4(first, row, x_first, nx);
    h_cta[2 * (size_t)b + 1] = make_int4((int)nv, np, p_first, 0);
    const size_t bytes = res_smem(nv, nx, np, row - first, es);
    smem = std::max(smem, bytes);
    fits = bytes <= kResSmemMax && nx <= 65535;
  }
  if (fits && row == n) {
    // one buffer, one copy
    const size_t sizes[4] = {h_cta.size() * sizeof(int4), h_rows.size() * sizeof(int4), h_x.size() * sizeof(int),
                             h_place.size() * sizeof(unsigned short)};
    const void* parts[4] = {h_cta.data(), h_rows.data(), h_x.data(), h_place.data()};
    size_t total = 0;
    for (int k = 0; k < 4; ++k) {
      plan->off[k] = total;
      total += (sizes[k] + 15) / 16 * 16;
    }
    std::vector<char> stage(total);
    for (int k = 0; k < 4; ++k)
      if (sizes[k]) std::memcpy(stage.data() + plan->off[k], parts[k], sizes[k]);
    if ((rc = plan->data.ensure(total, s))) return rc;
    VBG_CUDA(cudaMemcpyAsync(plan->data.p, stage.data(), total, cudaMemcpyHostToDevice, s));
    VBG_CUDA(cudaStreamSynchronize(s));  // the host vectors are locals
    plan->smem = smem;
    plan->grid = ctas;
    *out = plan.get();
  }
  slot = std::move(plan);
  return 0;
}

template <typename T, bool ADJ>
static int launch_resident_t(ResidentArgs& a, ResidentPlan* plan, const T* vals, cudaStream_t s, bool* ran) {
  static int state[kMaxDevices] = {};  // 1: usable, 2: not
  const int dev = current_device();
  if (!state[dev]) {
    int coop = 0, b = 0;
    VBG_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    VBG_CUDA(cudaFuncSetAttribute(resident_kernel<T, ADJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kResSmemMax));
    VBG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, resident_kernel<T, ADJ>, kResThreads, kResSmemMax));
    state[dev] = coop && b >= 1 ? 1 : 2;
  }
  *ran = state[dev] == 1;
  if (!*ran) return 0;
  void* params[2] = {&a, &vals};
  VBG_CUDA(cudaLaunchCooperativeKernel((const void*)resident_kernel<T, ADJ>, dim3(plan->grid), dim3(kResThreads),
                                       params, plan->smem, s));
  plan->ran = true;
  return 0;
}

// Runs the recurrence in `a` (recurrence and output fields set; coef on the
// host) on the resident kernel; *ran = false when it cannot run here: no plan,
// too few steps, or the stream is being captured (the plan and the scratch
// may not be made then).
static int resident_run(const vbg_matrix* m, bool adj, ResidentArgs& a, const double* coef, DevBuf& scratch,
                        cudaStream_t s, bool* ran) {
  *ran = false;
  if (a.steps < kResMinSteps || m->N == 0 || m->max_bs > 8) return 0;
  cudaStreamCaptureStatus st;
  if (cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) return 0;
  // the plan once the matrix's recurrences, this one among them, repay it
  auto* mm = const_cast<vbg_matrix*>(m);
  mm->recur_steps += a.steps;
  if (!m->resident[adj ? 1 : 0] && mm->recur_steps < kResPlanSteps + m->nnzb / kResPlanBlocks) return 0;
  ResidentPlan* plan = nullptr;
  int rc = resident_plan(m, adj, s, &plan);
  if (rc || !plan) return rc;
  if (adj && (rc = ensure_csc(m, s))) return rc;
  const size_t es = elem_size(m->dtype);
  const size_t vec = ((size_t)m->N * es + 255) / 256 * 256, cb = (size_t)a.steps * kResCoef * sizeof(double);
  if ((rc = scratch.ensure(256 + (cb + 255) / 256 * 256 + 2 * vec))) return rc;
  char* base = scratch.as<char>();
  a.sync = reinterpret_cast<unsigned*>(base);
  a.coef = reinterpret_cast<const double*>(base + 256);
  a.xch[0] = base + 256 + (cb + 255) / 256 * 256;
  a.xch[1] = static_cast<char*>(a.xch[0]) + vec;
  VBG_CUDA(cudaMemsetAsync(base, 0, 256, s));
  VBG_CUDA(cudaMemcpyAsync(base + 256, coef, cb, cudaMemcpyHostToDevice, s));
  const char* pd = plan->data.as<char>();
  a.cta = reinterpret_cast<const int4*>(pd + plan->off[0]);
  a.rows = reinterpret_cast<const int4*>(pd + plan->off[1]);
  a.xlist = reinterpret_cast<const int*>(pd + plan->off[2]);
  a.place = reinterpret_cast<const unsigned short*>(pd + plan->off[3]);
  a.ptr = (adj ? m->csc_ptr : m->row_ptr).as<int>();
  a.ent_slot = adj ? m->csc_slot.as<int>() : nullptr;
  a.ent_src = (adj ? m->csc_row : m->col_ind).as<int>();
  a.bsz = m->bsz.as<int>();
  a.blk_off = m->blk_off.as<int64_t>();
  a.N = m->N;
  if (m->dtype == VBG_C128)
    return adj ? launch_resident_t<cplx, true>(a, plan, m->vals.as<cplx>(), s, ran)
               : launch_resident_t<cplx, false>(a, plan, m->vals.as<cplx>(), s, ran);
  return adj ? launch_resident_t<double, true>(a, plan, m->vals.as<double>(), s, ran)
             : launch_resident_t<double, false>(a, plan, m->vals.as<double>(), s, ran);
}
