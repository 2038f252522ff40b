"""Timed cases of the framework's main path: what a user's program calls, over
the sizes, types and directions that the configurations, tests and benchmark
of this repository use.

listed() / draw() give cases (plain dicts), prepare() the objects that a
program holds before the call (matrices on the device, vectors), run() one
pass through the public entry points, work() the bytes and operations of one
pass, exact() the same results in plain 64-bit torch.

Kinds of case:
  spmv       y = A x or A^H x on a random symmetric block pattern (vbg_spmv,
             vbg_spmv_adjoint): solvers' inner product with the matrix
  spmv_pair  y = A x and z = A^H x on wide complex blocks (9 to 20 orbitals an
             atom): bi-orthogonal Krylov methods on DFT-sized bases
  spmm       Y = A X for a block of vectors (vbg_spmm)
  train      sparse_apply forward and backward: gradients of the block values
             and of X
  kpm        Chebyshev moments of a TMD lattice (vbg_kpm_moments): the DOS
             workload, FP64 and FP32 bulk
  kpm_batch  moments of several disorder realisations in one recurrence
             (vbg_kpm_moments_batched)
  spgemm     thresholded C = A B on banded decaying matrices (vbg_spgemm)
  spgemm_h   the Hermitian product on complex lattices (vbg_spgemm_hermitian)
  mcweeny    a whole purification through VBCSR and mcweeny_purify
  propagate  chebyshev_propagate of complex128 state, forward and backward
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from vbcsr_b200 import _capi
from vbcsr_b200 import workloads as W
from vbcsr_b200.autograd import chebyshev_propagate, sparse_apply

_vp = C.c_void_p


def listed():
    return [
        # a small system's solver step: one launch, all latency
        dict(name="spmv_500", kind="spmv", n=500, smin=4, smax=8, nb=6, dtype="f64", adj=False),
        # the 5000-row SpMV configuration of the benchmark
        dict(name="spmv_5000", kind="spmv", n=5000, smin=4, smax=8, nb=6, dtype="f64", adj=False),
        # wide complex blocks, both directions (k-point DFT matrices)
        dict(name="spmv_pair_wide_c128", kind="spmv_pair", n=4000, smin=9, smax=20, nb=6, band=64),
        # a 4096-block geometric graph of degree ~12 with 16 right-hand sides
        dict(name="spmm_wide_k16", kind="spmm", n=4096, smin=9, smax=16, nb=6, band=64, k=16, dtype="f64"),
        # fitting a Hamiltonian's values: forward, adjoint and value gradient
        dict(name="train_k24", kind="train", n=5000, smin=4, smax=8, nb=6, k=24),
        # a small cell's DOS with the helper's default 10 vectors and 200 moments
        dict(name="kpm_small", kind="kpm", L=20, Ly=20, R=10, M=200, prec="fp64", two=True),
        # the DOS configuration: 200 x 200 cells, 64 vectors, 1024 moments
        dict(name="kpm_200_fp64", kind="kpm", L=200, Ly=200, R=64, M=1024, prec="fp64", two=True),
        # disorder averages: uneven members in one recurrence, FP32 bulk
        dict(name="kpm_batch_fp32", kind="kpm_batch", count=10, smin=40, smax=100, R=16, M=512, prec="fp32"),
        # density-matrix product of a filled band
        dict(name="spgemm_band_fp64", kind="spgemm", n=12000, smin=4, smax=8, nb=16, band=32, thr=1e-5),
        # H^2 of a lattice in a magnetic field (complex Hermitian)
        dict(name="spgemm_herm_c128", kind="spgemm_h", L=60, Ly=60, thr=1e-4),
        # purification as the README runs it: 10 iterations, threshold 1e-5
        dict(name="mcweeny_3000", kind="mcweeny", n=3000, smin=4, smax=8, nb=8, band=32, thr=1e-5, its=10, herm=False),
        # the propagation configuration with its gradient
        dict(name="propagate_grad_60", kind="propagate", L=60, Ly=60, terms=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmv_pair", "spmm", "spmm", "train", "kpm", "kpm", "kpm_batch", "spgemm",
                       "spgemm_h", "mcweeny", "propagate"])
    if kind == "spmv":
        smin, smax = rng.choice([(4, 8), (1, 4), (3, 5)])
        return dict(kind=kind, n=_log(rng, 300, 20000), smin=smin, smax=smax, nb=rng.randint(2, 8),
                    dtype=rng.choice(["f64", "f64", "c128"]), adj=rng.random() < 0.3)
    if kind == "spmv_pair":
        return dict(kind=kind, n=_log(rng, 500, 6000), smin=9, smax=rng.randint(13, 20), nb=rng.randint(4, 8),
                    band=rng.randint(16, 128))
    if kind == "spmm":
        wide = rng.random() < 0.4
        return dict(kind=kind, n=_log(rng, 800, 5000), smin=9 if wide else 3, smax=16 if wide else 8,
                    nb=rng.randint(3, 8), band=rng.choice([0, 32, 64, 128]), k=rng.randint(3, 72),
                    dtype=rng.choice(["f64", "f64", "c128"]))
    if kind == "train":
        return dict(kind=kind, n=_log(rng, 800, 8000), smin=rng.randint(1, 4), smax=8, nb=rng.randint(3, 8),
                    k=rng.randint(1, 40))
    if kind == "kpm":
        L, Ly = _log(rng, 12, 160), _log(rng, 12, 160)
        return dict(kind=kind, L=L, Ly=Ly, R=rng.choice([1, 4, 10, 16, 24, 32, 48, 64]), M=rng.randint(64, 512),
                    prec=rng.choice(["fp64", "fp32"]), two=rng.random() < 0.8)
    if kind == "kpm_batch":
        return dict(kind=kind, count=rng.randint(3, 10), smin=rng.randint(16, 40), smax=rng.randint(50, 90),
                    R=rng.choice([8, 16, 32]), M=rng.randint(64, 512), prec=rng.choice(["fp64", "fp32"]))
    if kind == "spgemm":
        return dict(kind=kind, n=_log(rng, 1000, 11000), smin=rng.choice([1, 3, 4]), smax=8, nb=rng.randint(4, 15),
                    band=rng.randint(16, 64), thr=rng.choice([1e-5, 1e-4, 1e-6]))
    if kind == "spgemm_h":
        return dict(kind=kind, L=_log(rng, 16, 60), Ly=_log(rng, 16, 60), thr=rng.choice([1e-3, 1e-4, 1e-5]))
    if kind == "mcweeny":
        return dict(kind=kind, n=_log(rng, 500, 3000), smin=4, smax=8, nb=rng.randint(4, 8), band=rng.randint(16, 32), thr=1e-5,
                    its=rng.randint(3, 10), herm=rng.random() < 0.5)
    return dict(kind=kind, L=_log(rng, 16, 60), Ly=_log(rng, 16, 60), terms=rng.randint(48, 256))


# ---------------------------------------------------------------- inputs

@functools.lru_cache(maxsize=4)
def _base(kind, key):
    """The case's block matrix before its seed enters: pattern and block norms."""
    c = dict(key)
    if kind == "kpm_batch":
        H, seg = W.block_diagonal(W.tmd_disorder_batch(c["count"], c["smin"], c["smax"], seed=5))
        return H, seg
    if kind == "kpm":
        return W.tmd_lattice(c["L"], seed=5, Ly=c["Ly"])[0], None
    if kind in ("spgemm_h", "propagate"):
        return W.tmd_lattice(c["L"], seed=5, Ly=c["Ly"], bond_phase=True)[0], None
    if c.get("band", 0) == 0:
        H = W.random_symmetric_blocks(c["n"], c["smin"], c["smax"], c["nb"], seed=5)
    else:
        decay = 4.0 if kind in ("spgemm", "mcweeny") else 32.0
        H = W.banded_decaying(c["n"], c["smin"], c["smax"], c["nb"], c["band"], decay, seed=5)
    if kind == "spmv_pair" or c.get("dtype") == "c128":
        H.values = H.values * np.exp(2j * np.pi * np.random.default_rng(6).random(H.nnz))
    return H, None


def _matrix_of(case):
    kind = case["kind"]
    return _base(kind, tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "kind"))))


def _hamiltonian(case, seed):
    """The case's matrix with every block row's basis reflected by the seed
    (Q A Q^H, Q block diagonal, I - 2 v v^H): other values everywhere, the
    same pattern, block norms and spectrum, so that every seed's results have
    the same shape."""
    H, seg = _matrix_of(case)
    cx = np.iscomplexobj(H.values)
    rng = np.random.default_rng(seed)
    off = H.slot_offsets()
    rows = np.repeat(np.arange(H.n), np.diff(H.row_ptr))
    bs = H.block_sizes
    V = rng.standard_normal((H.n, int(bs.max())))
    if cx:
        V = V + 1j * rng.standard_normal(V.shape)
    V[np.arange(V.shape[1])[None, :] >= bs[:, None]] = 0.0
    V /= np.sqrt((np.abs(V) ** 2).sum(1))[:, None]
    out = np.empty_like(H.values)
    shape = bs[rows].astype(np.int64) * 1000 + bs[H.col_ind]
    for key in np.unique(shape):
        sel = np.nonzero(shape == key)[0]
        r, k = int(key // 1000), int(key % 1000)
        at = off[sel][:, None] + np.arange(r * k)
        B = H.values[at].reshape(-1, r, k)
        u, w = V[rows[sel], :r], V[H.col_ind[sel], :k]
        B = B - 2 * u[:, :, None] * (u.conj()[:, None, :] @ B)
        B = B - 2 * (B @ w[:, :, None]) * w.conj()[:, None, :]
        out[at] = B.reshape(len(sel), -1)
    return W.BlockCSR(H.block_sizes, H.row_ptr, H.col_ind, out), seg


def _ld(k, es=8):
    """The multivectors' leading dimension: k rounded up to 64 bytes."""
    per = 64 // es
    return k if k == 1 else (k + per - 1) // per * per


def _vectors(N, k, seed, kind="normal", dtype="f64"):
    """N x k vectors on the device: normal, or +-1 for stochastic traces."""
    rng = np.random.default_rng(seed + 17)
    if kind == "sign":
        v = np.where(rng.random((N, k)) < 0.5, -1.0, 1.0)
    else:
        v = rng.standard_normal((N, k))
        if dtype == "c128":
            v = v + 1j * rng.standard_normal((N, k))
    return torch.from_numpy(v).cuda()


def _padded(V):
    ld = _ld(V.shape[1], V.element_size())
    out = torch.zeros((V.shape[0], ld), dtype=V.dtype, device=V.device)
    out[:, :V.shape[1]] = V
    return out


def _matrix(H):
    return _capi.DeviceMatrix.create(H.block_sizes, H.row_ptr, H.col_ind, H.values)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "mcweeny":
        from vbcsr_b200 import VBCSR

        H, _ = _hamiltonian(c, seed)
        return dict(c=c, H=VBCSR.from_block_csr(H.block_sizes, H.row_ptr, H.col_ind, H.values))
    H, seg = _hamiltonian(c, seed)
    st = dict(c=c)
    if kind != "propagate" and kind != "train":
        st["A"] = _matrix(H)
    if kind == "spmv":
        st["x"] = _vectors(H.N, 1, seed, dtype=c["dtype"])[:, 0].contiguous()
        st["y"] = torch.zeros_like(st["x"])
    elif kind == "spmv_pair":
        st["x"] = _vectors(H.N, 1, seed, dtype="c128")[:, 0].contiguous()
        st["y"] = torch.zeros_like(st["x"])
        st["z"] = torch.zeros_like(st["x"])
    elif kind == "spmm":
        st["X"] = _padded(_vectors(H.N, c["k"], seed, dtype=c["dtype"]))
        st["Y"] = torch.zeros_like(st["X"])
    elif kind == "train":
        st["op"] = _matrix(H)
        st["values"] = torch.from_numpy(H.values).cuda().requires_grad_(True)
        st["X"] = _vectors(H.N, c["k"], seed).requires_grad_(True)
        st["G"] = _vectors(H.N, c["k"], seed + 1)
    elif kind == "kpm":
        V = _vectors(H.N, c["R"], seed, "sign")
        st["V"] = _padded(V) if c["R"] > 1 else V
        st["mu"] = torch.zeros(c["M"], dtype=torch.float64, device="cuda")
    elif kind == "kpm_batch":
        st["V"] = _padded(_vectors(H.N, c["R"], seed, "sign"))
        st["mu"] = torch.zeros((c["count"], c["M"]), dtype=torch.float64, device="cuda")
        st["seg"] = np.ascontiguousarray(seg, dtype=np.int32)
    elif kind == "propagate":
        st["op"] = _matrix(H)
        st["values"] = torch.from_numpy(H.values).cuda().requires_grad_(True)
        psi = _vectors(H.N, 1, seed, dtype="c128")[:, 0]
        st["psi0"] = (psi / torch.linalg.vector_norm(psi)).contiguous().requires_grad_(True)
        st["g"] = _vectors(H.N, 1, seed + 1, dtype="c128")[:, 0].contiguous()
    return st


# ---------------------------------------------------------------- one pass

def _p(t):
    return _vp(t.data_ptr())


def _stream():
    return _vp(torch.cuda.current_stream().cuda_stream)


class _View:
    """A device array of a matrix as torch sees it; keeps the matrix alive."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(int(n),), typestr=typestr, data=(int(ptr), False), version=3)


def _product(M):
    """A product's values and slot offsets, in place on the device."""
    vals, offs = _vp(), _vp()
    _capi.call("vbg_matrix_device_values", M.h, C.byref(vals), C.byref(offs))
    typ = "<c16" if M.dtype_code == _capi.VBG_C128 else "<f8"
    return {"values": torch.as_tensor(_View(M, vals.value, M.nnz, typ), device="cuda"),
            "offsets": torch.as_tensor(_View(M, offs.value, M.nnzb + 1, "<i8"), device="cuda")}


def run(st):
    c, kind = st["c"], st["c"]["kind"]
    if kind == "spmv":
        _capi.call("vbg_spmv_adjoint" if c["adj"] else "vbg_spmv", st["A"].h, _p(st["x"]), _p(st["y"]), _stream())
        return st["y"]
    if kind == "spmv_pair":
        _capi.call("vbg_spmv", st["A"].h, _p(st["x"]), _p(st["y"]), _stream())
        _capi.call("vbg_spmv_adjoint", st["A"].h, _p(st["x"]), _p(st["z"]), _stream())
        return st["y"], st["z"]
    if kind == "spmm":
        _capi.call("vbg_spmm", st["A"].h, c["k"], st["X"].stride(0), _p(st["X"]), _p(st["Y"]), _stream())
        return st["Y"]
    if kind == "train":
        Y = sparse_apply(st["values"], st["X"], st["op"])
        gv, gx = torch.autograd.grad(Y, (st["values"], st["X"]), st["G"])
        return Y.detach(), gv, gx
    if kind == "kpm":
        _capi.call("vbg_kpm_moments", st["A"].h, c["R"], st["V"].stride(0) if c["R"] > 1 else 1, _p(st["V"]), c["M"],
                   int(c["prec"] == "fp32"), int(c["two"]), 1, _p(st["mu"]), _stream())
        return st["mu"]
    if kind == "kpm_batch":
        _capi.call("vbg_kpm_moments_batched", st["A"].h, c["count"], st["seg"].ctypes.data_as(C.POINTER(C.c_int)),
                   c["R"], st["V"].stride(0), _p(st["V"]), c["M"], int(c["prec"] == "fp32"), 1, 1, _p(st["mu"]),
                   _stream())
        return st["mu"]
    if kind == "spgemm":
        return _product(st["A"].spgemm(st["A"], c["thr"], torch.cuda.current_stream().cuda_stream)[0])
    if kind == "spgemm_h":
        return _product(st["A"].spgemm_hermitian(st["A"], c["thr"], torch.cuda.current_stream().cuda_stream)[0])
    if kind == "mcweeny":
        from vbcsr_b200.purification import mcweeny_purify

        r = mcweeny_purify(st["H"], threshold=c["thr"], iterations=c["its"], hermitian=c["herm"])
        return {"values": r.P.get_values(), "nnzb": r.nnzb, "trace": r.trace, "residual": r.residual}
    psi = chebyshev_propagate(st["values"], st["psi0"], st["op"], dt=100.0, scale=1.0, num_terms=c["terms"])
    gv, gp = torch.autograd.grad(psi, (st["values"], st["psi0"]), st["g"])
    return psi.detach(), gv, gp


# ------------------------------------------------- what a pass cannot avoid

def _norms(H):
    return np.sqrt(np.add.reduceat(np.abs(H.values) ** 2, H.slot_offsets()[:-1]))


def _pairs(H, norms):
    """All (slot of A_ik, slot of A_kj) pairs of A A, numpy, with their C key."""
    rows = np.repeat(np.arange(H.n), np.diff(H.row_ptr))
    ln = np.diff(H.row_ptr).astype(np.int64)[H.col_ind]
    sa = np.repeat(np.arange(H.nnzb), ln)
    within = np.arange(int(ln.sum())) - np.repeat(np.cumsum(ln) - ln, ln)
    sb = np.asarray(H.row_ptr, np.int64)[H.col_ind][sa] + within
    key = rows[sa].astype(np.int64) * H.n + H.col_ind[sb]
    return sa, sb, key, norms[sa] * norms[sb], rows


def _product_work(H, thr, upper):
    """Stored scalars of C and multiply-adds of the kept pairs (a thresholded
    A A, the symbolic keep rule and the pair skip)."""
    sa, sb, key, pn, rows = _pairs(H, _norms(H))
    bs = H.block_sizes.astype(np.int64)
    uk, inv = np.unique(key, return_inverse=True)
    kept = np.bincount(inv, weights=pn) > thr
    ok = kept[inv] & (pn >= thr / np.maximum(1, np.diff(H.row_ptr))[rows[sa]])
    ui, uj = uk // H.n, uk % H.n
    cs = bs[ui] * bs[uj]
    flops = (bs[rows[sa]] * bs[H.col_ind[sa]] * bs[H.col_ind[sb]])[ok]
    up = (rows[sa] <= H.col_ind[sb])[ok] if upper else np.ones(int(ok.sum()), bool)
    return int(cs[kept].sum()), int(kept.sum()), 2 * int(flops[up].sum())


def work(case):
    c, kind = case, case["kind"]
    H, _ = _matrix_of(c)
    n, nnzb, nnz, N = H.n, H.nnzb, H.nnz, H.N
    struct = 4.0 * nnzb + 4.0 * (n + 1)
    cx = 2 if np.iscomplexobj(H.values) else 1
    es, fl = 8 * cx, 2 * cx * cx
    if kind == "spmv":
        return dict(bytes=es * (nnz + 2.0 * N) + struct, flops=float(fl * nnz))
    if kind == "spmv_pair":  # the matrix, x, and both results
        return dict(bytes=es * (nnz + 3.0 * N) + struct, flops=2.0 * fl * nnz)
    if kind == "spmm":
        return dict(bytes=es * (nnz + 2.0 * N * c["k"]) + struct, flops=float(fl * nnz * c["k"]))
    if kind == "train":  # values, X, G in; Y, gX, gV out
        return dict(bytes=es * (2.0 * nnz + 4.0 * N * c["k"]) + struct, flops=3.0 * fl * nnz * c["k"])
    if kind in ("kpm", "kpm_batch"):
        # every step reads the matrix and two vectors and writes one
        ws = 4 if c["prec"] == "fp32" else 8
        steps = 1 + ((c["M"] - 2) // 2 if c.get("two", True) else c["M"] - 2)
        return dict(bytes=steps * (ws * (nnz + 3.0 * N * c["R"]) + struct), flops=steps * 2.0 * nnz * c["R"])
    if kind in ("spgemm", "spgemm_h"):
        cn, cb, flops = _product_work(H, c["thr"], kind == "spgemm_h")
        return dict(bytes=es * (nnz + cn) + struct + 8.0 * cb, flops=flops * cx * cx)
    if kind == "mcweeny":
        # the first product's pairs for each of the products (later ones, on
        # filled patterns, have more), the result read and written per iteration
        P = W.BlockCSR(H.block_sizes, H.row_ptr, H.col_ind, 0.1 * H.values)
        cn, cb, flops = _product_work(P, c["thr"], c["herm"])
        return dict(bytes=c["its"] * 2.0 * (es * cn + 4.0 * cb), flops=2.0 * c["its"] * flops)
    # propagate: the recurrence forward, again in the backward, its adjoint;
    # vectors and values are read once per step
    steps = 3.0 * (c["terms"] - 1)
    return dict(bytes=steps * (es * (nnz + 3.0 * N) + struct), flops=(steps + c["terms"] - 1) * fl * nnz)


def tolerance(case):
    """About four times what the paths measure against exact()."""
    kind = case["kind"]
    if kind in ("kpm", "kpm_batch"):
        # of the moments' norm, which mu_0 dominates: FP32 7e-9, FP64 1.3e-15
        # for the longest recurrence
        return {"rel": 3e-8} if case["prec"] == "fp32" else {"rel": 1e-14}
    if kind == "mcweeny":
        return {"rel": 2e-14}  # twenty products, each of them 4e-16
    if kind == "propagate":
        return {"rel": 1e-13}  # 2.7e-14: 256 steps of an unnormalised recurrence
    return {"rel": 4e-15}  # 1.9e-16 to 8e-16


# ------------------------------------------------------- plain 64-bit torch

def _coords(H):
    """Scalar row and column of every stored value (slot order)."""
    so = np.zeros(H.n + 1, np.int64)
    np.cumsum(H.block_sizes, out=so[1:])
    rows = np.repeat(np.arange(H.n), np.diff(H.row_ptr))
    r, k = H.block_sizes[rows].astype(np.int64), H.block_sizes[H.col_ind].astype(np.int64)
    blk = np.repeat(np.arange(H.nnzb), r * k)
    t = np.arange(H.nnz) - np.repeat(np.cumsum(r * k) - r * k, r * k)
    return (torch.from_numpy(so[rows][blk] + t // k[blk]).cuda(),
            torch.from_numpy(so[H.col_ind][blk] + t % k[blk]).cuda())


def _csr(H, N):
    i, j = _coords(H)
    return torch.sparse_coo_tensor(torch.stack([i, j]), torch.from_numpy(H.values).cuda(), (N, N)).coalesce().to_sparse_csr()


def _moments(A, V, M, two, seg=None):
    """mu_n = sum_r <v_r|T_n(A)|v_r> of every segment of rows."""
    def dot(a, b):
        d = (a * b).sum(1)
        if seg is None:
            return d.sum()[None]
        return torch.stack([d[seg[s]:seg[s + 1]].sum() for s in range(len(seg) - 1)])

    mu = [None] * max(M, 2)
    t0, t1 = V, A @ V
    mu[0], mu[1] = dot(V, V), dot(V, t1)
    if two:
        if M > 2:
            mu[2] = 2 * dot(t1, t1) - mu[0]
        for n in range(1, (M - 2) // 2 + 1):
            t0, t1 = t1, 2 * (A @ t1) - t0
            if 2 * n + 1 < M:
                mu[2 * n + 1] = 2 * dot(t1, t0) - mu[1]
            if 2 * n + 2 < M:
                mu[2 * n + 2] = 2 * dot(t1, t1) - mu[0]
    else:
        for n in range(2, M):
            t0, t1 = t1, 2 * (A @ t1) - t0
            mu[n] = dot(V, t1)
    return torch.stack(mu[:M], dim=1)


class _Blocks:
    """A block matrix as 8 x 8 (or wider) zero-padded blocks, sorted by key."""

    def __init__(self, bs, key, val, width):
        self.bs, self.key, self.val, self.w = bs, key, val, width
        n = len(bs)
        self.row, self.col = key // n, key % n
        cnt = torch.bincount(self.row, minlength=n)
        self.len = cnt
        self.ptr = torch.cat([torch.zeros(1, dtype=torch.int64, device=key.device), torch.cumsum(cnt, 0)])

    @classmethod
    def of(cls, H):
        w = int(H.block_sizes.max())
        bs = torch.from_numpy(H.block_sizes.astype(np.int64)).cuda()
        rows = np.repeat(np.arange(H.n), np.diff(H.row_ptr)).astype(np.int64)
        key = torch.from_numpy(rows * H.n + H.col_ind).cuda()
        r, k = H.block_sizes[rows].astype(np.int64), H.block_sizes[H.col_ind].astype(np.int64)
        blk = np.repeat(np.arange(H.nnzb), r * k)
        t = np.arange(H.nnz) - np.repeat(np.cumsum(r * k) - r * k, r * k)
        at = torch.from_numpy(blk * w * w + t // k[blk] * w + t % k[blk]).cuda()
        v = torch.zeros(H.nnzb * w * w, dtype=torch.from_numpy(H.values).dtype, device="cuda")
        v[at] = torch.from_numpy(H.values).cuda()
        return cls(bs, key, v.reshape(-1, w, w), w)

    def norms(self):
        return self.val.abs().square().sum((1, 2)).sqrt()

    def select(self, keep):
        return _Blocks(self.bs, self.key[keep], self.val[keep], self.w)

    def values(self):
        r, k = self.bs[self.row], self.bs[self.col]
        i = torch.arange(self.w, device="cuda")
        live = (i[None, :, None] < r[:, None, None]) & (i[None, None, :] < k[:, None, None])
        return self.val[live]

    def offsets(self):
        o = torch.zeros(len(self.key) + 1, dtype=torch.int64, device="cuda")
        torch.cumsum(self.bs[self.row] * self.bs[self.col], 0, out=o[1:])
        return o

    def product(self, B, thr, upper=False):
        """Thresholded product: keep C_ij iff sum_k |A_ik||B_kj| > thr, skip
        pairs below thr / blocks of A's row, drop finished blocks below thr."""
        n, nA, nB = len(self.bs), self.norms(), B.norms()
        ln = B.len[self.col]
        sa = torch.repeat_interleave(torch.arange(len(self.key), device="cuda"), ln)
        sb = B.ptr[self.col][sa] + torch.arange(len(sa), device="cuda") - (torch.cumsum(ln, 0) - ln)[sa]
        key = self.row[sa] * n + B.col[sb]
        if upper:
            up = B.col[sb] >= self.row[sa]
            sa, sb, key = sa[up], sb[up], key[up]
        pn = nA[sa] * nB[sb]
        uk, inv = torch.unique(key, return_inverse=True)
        tot = torch.zeros(len(uk), dtype=torch.float64, device="cuda").index_add_(0, inv, pn)
        kept = tot > thr
        slot = torch.cumsum(kept, 0) - 1
        ok = kept[inv] & (pn >= thr / self.len.clamp(min=1)[self.row[sa]])
        sa, sb, dst = sa[ok], sb[ok], slot[inv[ok]]
        out = torch.zeros((int(kept.sum()), self.w, self.w), dtype=self.val.dtype, device="cuda")
        for i in range(0, len(sa), 1 << 20):
            s = slice(i, i + (1 << 20))
            out.index_add_(0, dst[s], self.val[sa[s]] @ B.val[sb[s]])
        C_ = _Blocks(self.bs, uk[kept], out, self.w)
        C_ = C_.select(C_.norms() >= thr) if thr > 0 else C_
        if upper:
            d = C_.row == C_.col
            D = C_.val[d]
            C_.val[d] = 0.5 * (D + D.transpose(1, 2).conj())
            key = torch.cat([C_.key, C_.col[~d] * n + C_.row[~d]])
            val = torch.cat([C_.val, C_.val[~d].transpose(1, 2).conj()])
            o = torch.argsort(key)
            C_ = _Blocks(self.bs, key[o], val[o], self.w)
        return C_

    def plus(self, a, B, b):
        """a self + b B on the union pattern."""
        uk, inv = torch.unique(torch.cat([self.key, B.key]), return_inverse=True)
        v = torch.zeros((len(uk), self.w, self.w), dtype=self.val.dtype, device="cuda")
        v.index_add_(0, inv, torch.cat([a * self.val, b * B.val]))
        return _Blocks(self.bs, uk, v, self.w)

    def trace(self):
        return float(torch.diagonal(self.val[self.row == self.col], dim1=1, dim2=2).sum())


def _mcweeny(c, H):
    A = _Blocks.of(H)
    d = A.row == A.col
    i = torch.arange(A.w, device="cuda")
    eye = ((i[None, :] < A.bs[:, None]).double()[:, :, None] * torch.eye(A.w, dtype=torch.float64, device="cuda"))
    A.val *= 0.1
    A.val[d] += 0.5 * eye[A.row[d]]
    nnzb, trace, residual = [], [], []
    for _ in range(c["its"]):
        P2 = A.product(A, c["thr"], c["herm"])
        residual.append(float(P2.plus(1.0, A, -1.0).val.square().sum().sqrt()))
        A = P2.plus(3.0, P2.product(A, c["thr"], c["herm"]), -2.0)
        A = A.select(A.norms() >= c["thr"])
        nnzb.append(len(A.key))
        trace.append(A.trace())
    return {"values": A.values(), "nnzb": nnzb, "trace": trace, "residual": residual}


def exact(case, seed):
    c, kind = case, case["kind"]
    H, seg = _hamiltonian(c, seed)
    if kind == "kpm_batch":
        so = np.concatenate([[0], np.cumsum(H.block_sizes)])
        return _moments(_csr(H, H.N), _vectors(H.N, c["R"], seed, "sign"), c["M"], True, [int(so[s]) for s in seg])
    if kind in ("spmv", "spmv_pair"):
        A = _csr(H, H.N)
        x = _vectors(H.N, 1, seed, dtype=c.get("dtype", "c128"))

        def adjoint():
            i, j = _coords(H)
            v = torch.from_numpy(H.values).cuda().conj().resolve_conj()
            return torch.zeros_like(x[:, 0]).index_add_(0, j, v * x[i, 0])

        if kind == "spmv":
            return adjoint() if c["adj"] else (A @ x)[:, 0]
        return (A @ x)[:, 0], adjoint()
    if kind == "spmm":
        return _padded(_csr(H, H.N) @ _vectors(H.N, c["k"], seed, dtype=c["dtype"]))
    if kind == "train":
        i, j = _coords(H)
        v = torch.from_numpy(H.values).cuda()
        X, G = _vectors(H.N, c["k"], seed), _vectors(H.N, c["k"], seed + 1)
        return (torch.zeros_like(X).index_add_(0, i, v[:, None] * X[j]), (G[i] * X[j]).sum(1),
                torch.zeros_like(X).index_add_(0, j, v[:, None] * G[i]))
    if kind == "kpm":
        return _moments(_csr(H, H.N), _vectors(H.N, c["R"], seed, "sign"), c["M"], c["two"])[0]
    if kind in ("spgemm", "spgemm_h"):
        A = _Blocks.of(H)
        P = A.product(A, c["thr"], kind == "spgemm_h")
        return {"values": P.values(), "offsets": P.offsets()}
    if kind == "mcweeny":
        return _mcweeny(c, H)
    # J_n(100) from the Fourier series of exp(i 100 sin t)
    n = np.arange(c["terms"])
    J = np.fft.fft(np.exp(100j * np.sin(2 * np.pi * np.arange(2048) / 2048))).real[:c["terms"]] / 2048
    coef = np.where(n == 0, 1.0, 2.0) * (-1j) ** n * J
    i, j = _coords(H)
    v = torch.from_numpy(H.values).cuda().requires_grad_(True)
    p = _vectors(H.N, 1, seed, dtype="c128")[:, 0]
    p = (p / torch.linalg.vector_norm(p)).requires_grad_(True)
    g = _vectors(H.N, 1, seed + 1, dtype="c128")[:, 0]
    mul = lambda x: torch.zeros_like(x).index_add(0, i, v * x[j])  # noqa: E731
    t0, t1 = p, mul(p)
    psi = complex(coef[0]) * t0 + complex(coef[1]) * t1
    for m in range(2, c["terms"]):
        t0, t1 = t1, 2 * mul(t1) - t0
        psi = psi + complex(coef[m]) * t1
    gv, gp = torch.autograd.grad(psi, (v, p), g)
    return psi.detach(), gv, gp
