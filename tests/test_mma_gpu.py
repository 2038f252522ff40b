"""The tensor-core row apply at its edges: leading dimensions that fill no
128-byte piece or several, blocks of 1 to 24 (row tiles with a remainder, two
row groups), few rows (entries split over the CTA's warps) and many, forward
and adjoint, with the fused epilogue, against the oracle's apply and the
epilogue in numpy.  Tolerance 1e-12 of the largest value: sums of at most 13
blocks of 24 products, 300 roundings of 1.1e-16."""
import ctypes as C

import numpy as np
import pytest

from vbcsr_b200 import workloads as W

from .conftest import rel_err

pytestmark = pytest.mark.gpu


def _matrix(name):
    if name == "wide":
        return W.random_pattern(40, 7, 24, 6, seed=31)
    if name == "few":
        return W.random_symmetric_blocks(30, 4, 8, 6, seed=32)
    if name == "many":
        return W.random_pattern(4200, 1, 3, 2, seed=33)
    return W.random_pattern(60, 9, 17, 5, seed=34)


@pytest.mark.parametrize("name", ["wide", "few", "many", "all_wide"])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("k", [2, 7, 18, 33, 72])
def test_fused_step(oracle, dev, name, cplx, adjoint, k):
    import torch

    from vbcsr_b200 import _capi

    from . import _gpu

    H = _matrix(name)
    rng = np.random.default_rng(k)
    if cplx:
        H.values = H.values * np.exp(2j * np.pi * rng.random(H.nnz))
    dt = H.values.dtype

    def mv():
        v = rng.normal(size=(H.N, k))
        return v + 1j * rng.normal(size=(H.N, k)) if cplx else v

    X, P, D, A = mv(), mv(), mv(), mv()
    dm = _gpu.dmat(H)
    # the smallest legal leading dimension (16-byte rows), not the padded one
    ld = k if cplx or k % 2 == 0 else k + 1
    x, p, d, acc = (_gpu.to_dev_mv(v, ld, dt) for v in (X, P, D, A))
    y = torch.zeros_like(x)
    dots = torch.zeros(2, dtype=torch.float64, device="cuda")
    alpha, beta, gamma, c = 1.7, -0.3, -1.0, (0.4 - 0.2j if cplx else 0.4)
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    _capi.call("vbg_cheb_step_adjoint" if adjoint else "vbg_cheb_step", dm.h, k, ld, alpha, beta, gamma, ptr(x),
               ptr(p), ptr(y), ptr(d), ptr(dots), ptr(acc), float(np.real(c)), float(np.imag(c)), None)
    torch.cuda.synchronize()
    Y = alpha * oracle.apply(H, X, adjoint) + beta * X + gamma * P
    assert rel_err(y.cpu().numpy()[:, :k], Y) < 1e-12
    assert np.all(y.cpu().numpy()[:, k:] == 0)
    assert rel_err(acc.cpu().numpy()[:, :k], A + c * Y) < 1e-12
    ref = np.array([np.sum((D.conj() * Y).real), np.sum(np.abs(Y) ** 2)])
    assert np.abs(dots.cpu().numpy() - ref).max() < 1e-12 * np.sum(np.abs(D) * np.abs(Y) + np.abs(Y) ** 2)
