"""Adjoint vectors on blocks of at most 8 x 8 at their edges: few block columns
(their blocks split over the CTA's warps), more than 32 blocks in a column, more
columns than warps, blocks of 1 and 8, empty columns, with the fused epilogue.
Tolerance 1e-12 of the largest value: sums of at most 60 blocks of 8 products,
500 roundings of 1.1e-16 (a column's products all count towards its value)."""
import ctypes as C

import numpy as np
import pytest

from vbcsr_b200 import workloads as W

from .conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lo,hi,per_row", [(1, 3, 3, 0), (7, 1, 8, 3), (60, 8, 8, 50), (500, 1, 8, 6),
                                             (4000, 1, 3, 40), (9000, 1, 1, 2)])
@pytest.mark.parametrize("cplx", [False, True])
def test_fused_adjoint_step(oracle, dev, n, lo, hi, per_row, cplx):
    import torch

    from vbcsr_b200 import _capi

    from . import _gpu

    H = W.random_pattern(n, lo, hi, per_row, seed=n)
    if n == 500:  # empty block columns
        keep = np.nonzero(H.col_ind % 9 != 4)[0]
        off = H.slot_offsets()
        rows = np.repeat(np.arange(n), np.diff(H.row_ptr))
        rp = np.concatenate([[0], np.cumsum(np.bincount(rows[keep], minlength=n))]).astype(np.int32)
        H = W.BlockCSR(H.block_sizes, rp, H.col_ind[keep], np.concatenate([H.values[off[s]:off[s + 1]] for s in keep]))
    rng = np.random.default_rng(n)
    if cplx:
        H.values = H.values * np.exp(2j * np.pi * rng.random(H.nnz))
    X, P, D, A = (rng.normal(size=(H.N, 1)) + (1j * rng.normal(size=(H.N, 1)) if cplx else 0) for _ in range(4))
    dm = _gpu.dmat(H)
    x, p, d, acc = (_gpu.to_dev_mv(v, 1, H.values.dtype) for v in (X, P, D, A))
    y = torch.zeros_like(x)
    dots = torch.zeros(2, dtype=torch.float64, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    c = 0.4 - 0.2j if cplx else 0.4
    _capi.call("vbg_cheb_step_adjoint", dm.h, 1, 1, 1.7, -0.3, -1.0, ptr(x), ptr(p), ptr(y), ptr(d), ptr(dots),
               ptr(acc), float(np.real(c)), float(np.imag(c)), None)
    torch.cuda.synchronize()
    Y = 1.7 * oracle.apply(H, X, True) - 0.3 * X - P
    assert rel_err(y.cpu().numpy().reshape(Y.shape), Y) < 1e-12
    assert rel_err(acc.cpu().numpy().reshape(Y.shape), A + c * Y) < 1e-12
    ref = np.array([np.sum((D.conj() * Y).real), np.sum(np.abs(Y) ** 2)])
    assert np.abs(dots.cpu().numpy() - ref).max() < 1e-12 * np.sum(np.abs(D) * np.abs(Y) + np.abs(Y) ** 2)
