// Row-tiled forward multivector apply on the FP64 tensor cores (real and
// complex values).  Included by vbg_apply.cu inside namespace vbg, after
// vbg_tile.cuh, whose tiles, q-lists, balanced runs and kernel-layout values
// it shares (tile_plan); FP32 keeps that file's kernels.
//
// A multivector row is NP pieces of 128 bytes (16 real or 8 complex columns
// each), NP = 1 or 2; wider rows keep the scalar kernel.  A warp multiplies a
// block row of r <= 8 scalar rows as m8n8k4 steps: four X rows of its q-list at
// a time are the B operand (lane l: X row l % 4, 16-byte chunk l / 4 of every
// piece), the four columns of values the A operand (lane l: scalar row l / 4,
// column l % 4).
//
// What bounds a narrow apply is instructions and latency: in the scalar form
// a lane holds one column, and every X row costs the lane's piece, the
// column's values as broadcasts and their addresses for r multiply-adds.
// Here four X rows are one 8-byte load of values, NP 16-byte loads of X and
// 2 NP steps.  20 x 20 lattice, 16 columns: 8.4 us a step, now 6.4; 32
// columns had no tiled form (200 x 200 lattice: 230 us).
// The X rows are staged by 16-byte asynchronous copies with the chunks of a
// piece permuted by the row's place (dtile_chunk): the four rows of a step
// sit at the same bank offset otherwise (rows are multiples of 128 bytes),
// and every B load would take four passes.
//
// The values and the q-list come by bulk copy as in the FP32 kernel; waits are
// bounded the same way.

// Physical 16-byte chunk, within its 128-byte piece, of logical chunk c of the
// staged row at `slot`.
__device__ __forceinline__ int dtile_chunk(int c, int slot) { return c ^ ((slot & 3) << 1); }

__device__ __forceinline__ void cp_async16(unsigned dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Lane's A operand of inner index k: value `g` of the kernel-layout column.
template <typename T>
__device__ __forceinline__ void dtile_mma(double (&c)[4], const T& a, const double2& b) {
  if constexpr (std::is_same<T, cplx>::value) {
    dmma_884(c[0], c[2], a.re, b.x);
    dmma_884(c[1], c[3], a.re, b.y);
    dmma_884(c[0], c[2], -a.im, b.y);
    dmma_884(c[1], c[3], a.im, b.x);
  } else {
    dmma_884(c[0], c[2], a, b.x);
    dmma_884(c[1], c[3], a, b.y);
  }
}

// Y = alpha acc + beta X + gamma Xprev, dots and accumulator for one 16-byte
// chunk (two real or one complex element) at element offset `el` of the
// multivectors in doubles; xc: the row's own chunk of X in shared memory.
template <typename T>
__device__ __forceinline__ void dtile_epilogue(const ApplyArgs& a, const double* acc, const double* xc, int64_t el,
                                               double& d0, double& d1) {
  constexpr int E = std::is_same<T, cplx>::value ? 1 : 2;
  struct alignas(16) V {
    T v[E];
  };
  V s, y;
  memcpy(&s, acc, 16);
  auto at = [&](const void* base) { return reinterpret_cast<const V*>(static_cast<const double*>(base) + el); };
  V xs, xp, xd, ac;
  if (a.beta != 0.0 || (a.want_dots && !a.dotw)) xs = *reinterpret_cast<const V*>(xc);
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

template <typename T, int NP>
__global__ void __launch_bounds__(kTileWarps * 32, 2)
    apply_dtile_kernel(ApplyArgs a, const T* __restrict__ vals, const int4* __restrict__ tiles,
                       const int* __restrict__ xrows, const unsigned short* __restrict__ qidx,
                       const int4* __restrict__ rowinfo, int ntiles, unsigned vbytes16, unsigned qbytes16,
                       int part_base, int total) {
  constexpr int RB = 128 * NP;            // bytes of a multivector row
  constexpr int RPI = 4 / NP;             // rows per copy instruction of a warp
  constexpr int VP = 16 / (int)sizeof(T); // kernel-layout columns are padded to VP values
  extern __shared__ __align__(16) unsigned char dtile_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const unsigned bar = smem_addr(dtile_smem);
  const T* vs_base = reinterpret_cast<const T*>(dtile_smem + 16);
  const unsigned short* qs_base = reinterpret_cast<const unsigned short*>(dtile_smem + 16 + vbytes16);
  const unsigned char* xs_base = dtile_smem + 16 + vbytes16 + qbytes16;
  const unsigned xs_s = smem_addr(xs_base), vs_s = smem_addr(vs_base), qs_s = smem_addr(qs_base);
  const bool use_p = a.gamma != 0.0, use_d = a.want_dots && a.dotw;
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_init_fence();
  }
  __syncthreads();
  const unsigned char* X = static_cast<const unsigned char*>(a.X);
  double d0 = 0.0, d1 = 0.0;
  unsigned phase = 0;
  bool failed = false;
  int4 ra, rb, rc, rq;  // the next tile's record
  if (blockIdx.x < ntiles) {
    ra = tiles[4 * blockIdx.x];
    rb = tiles[4 * blockIdx.x + 1];
    rc = tiles[4 * blockIdx.x + 2];
    rq = tiles[4 * blockIdx.x + 3];
  }
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int nt = tile + (int)gridDim.x;
    const int4 ta = ra, tb = rb, tc = rc, tq = rq;
    if (nt < ntiles) {
      ra = tiles[4 * nt];
      rb = tiles[4 * nt + 1];
      rc = tiles[4 * nt + 2];
      rq = tiles[4 * nt + 3];
    }
    const long long k0 = (static_cast<long long>(tb.y) << 32) | static_cast<unsigned>(tb.x);
    // this tile's X rows: a warp 32 of them at a time
    const int nslots = tb.w / RB;
    for (int base = 32 * warp; base < nslots; base += 32 * kTileWarps) {
      const int mine = base + lane < nslots ? __ldg(xrows + tc.w + base + lane) : 0;
      const int cnt = min(32, nslots - base);
      const int sub = lane / (8 * NP), c = lane % (8 * NP);  // row of the instruction, chunk of the row
#pragma unroll 4
      for (int j = 0; j < cnt; j += RPI) {
        const int src = __shfl_sync(0xffffffffu, mine, j + sub);
        const int slot = base + j + sub;
        if (j + sub < cnt)
          cp_async16(xs_s + (unsigned)slot * RB + (unsigned)(c >> 3) * 128 + (unsigned)dtile_chunk(c & 7, slot) * 16,
                     X + (long long)src * RB + c * 16);
      }
    }
    if (threadIdx.x == 0) {
      const unsigned vbytes = (unsigned)tb.z, obytes = (unsigned)tc.y * RB;
      // the previous tile's shared-memory reads come before these copies
      fence_proxy_async();
      mbar_arm(bar, vbytes + (unsigned)tq.y);
      bulk_g2s(qs_s, qidx + tq.x, (unsigned)tq.y, bar);
      if (vbytes) bulk_g2s(vs_s, vals + k0, vbytes, bar);
      // the epilogue's streamed operands: have L2 fetch the tile's rows
      if (use_p) bulk_prefetch_l2(static_cast<const unsigned char*>(a.Xprev) + (long long)tc.z * RB, obytes);
      if (use_d) bulk_prefetch_l2(static_cast<const unsigned char*>(a.dotw) + (long long)tc.z * RB, obytes);
    }
    // this warp's run of block rows [row0, row1)
    auto run_end = [&](int k) {  // end of run k within the tile: byte k of (tq.z, tq.w)
      return (int)((((unsigned)(k < 4 ? tq.z : tq.w)) >> (8 * (k & 3))) & 0xffu);
    };
    const int row0 = ta.x + (warp == 0 ? 0 : run_end(warp - 1));
    const int row1 = ta.x + run_end(warp);
    int4 ri = make_int4(0, 0, 0, 0);  // {q-list entry, q-list length, first value, block size}
    long long y0 = 0;
    if (row0 < row1) {
      ri = rowinfo[row0];
      y0 = a.scal_off[row0];
    }
    cp_async_wait_all();
    const bool ok = warp == 0 ? pipe_wait(bar, phase) : true;
    if (!__syncthreads_and(ok)) {
      failed = true;
      break;
    }
    (void)mbar_try_wait(bar, phase);
    phase ^= 1u;
    for (int row = row0; row < row1; ++row) {
      if (row != row0) {
        ri = rowinfo[row];
        y0 = a.scal_off[row];
      }
      const int r = ri.w, nq = ri.y;
      const int rp = (r + VP - 1) / VP * VP;
      double acc[NP][4];
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int t = 0; t < 4; ++t) acc[p][t] = 0.0;
      const unsigned short* ql = qs_base + ri.x + t4;
      // rows past the block read a neighbouring value: their results are not
      // stored (past the last value the q-list's bytes are read)
      const T* va = vs_base + ri.z + t4 * rp + g;
      auto chunk = [&](int slot) {
        return xs_base + (unsigned)slot * RB + (unsigned)dtile_chunk(g, slot) * 16;
      };
      int q = 0;
      // even and odd steps summed apart: half the chain, and the rounding error
      // of the two lane groups that this replaced
      double odd[NP][4] = {};
      auto step = [&](double (&c)[NP][4], int q) {
        const unsigned char* xr = chunk(ql[q]);
        const T av = va[q * rp];
        double2 b[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) b[p] = *reinterpret_cast<const double2*>(xr + 128 * p);
#pragma unroll
        for (int p = 0; p < NP; ++p) dtile_mma<T>(c[p], av, b[p]);
      };
      for (; q + 8 <= nq; q += 8) {
        step(acc, q);
        step(odd, q + 4);
      }
      if (q + 4 <= nq) {
        step(odd, q);
        q += 4;
      }
      if (q < nq) {  // the last one to three X rows: zero operands beyond them
        const bool kv = q + t4 < nq;
        const unsigned char* xr = chunk(kv ? ql[q] : 0);
        const T av = kv ? va[q * rp] : zero_s<T>();
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          const double2 b = kv ? *reinterpret_cast<const double2*>(xr + 128 * p) : make_double2(0.0, 0.0);
          dtile_mma<T>(acc[p], av, b);
        }
      }
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int t = 0; t < 4; ++t) acc[p][t] += odd[p][t];
      double rd0 = 0.0, rd1 = 0.0;
      if (g < r) {
        const int oslot = tc.x + (int)(y0 - tc.z) + g;
        const unsigned char* xo = xs_base + (unsigned)oslot * RB;
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            dtile_epilogue<T>(a, &acc[p][2 * h],
                              reinterpret_cast<const double*>(xo + 128 * p + dtile_chunk(2 * t4 + h, oslot) * 16),
                              (y0 + g) * (RB / 8) + 16 * p + 4 * t4 + 2 * h, rd0, rd1);
      }
      if (a.want_dots) {
        if (a.row_dots) {
          write_row_dots(a.row_dots, row, rd0, rd1);
        } else {
          d0 += rd0;
          d1 += rd1;
        }
      }
    }
    __syncthreads();  // every warp is done with the tile before the next copies
  }
  if (failed && threadIdx.x == 0) {
    atomicOr(&g_pipe_status, 1u);
    // the copies of the tile that timed out may still be in flight
    mbar_wait_bounded(bar, phase);
  }
  if (a.want_dots && !a.row_dots) grid_reduce2(d0, d1, a.partials, a.counter, a.dots_out, part_base, total);
}
