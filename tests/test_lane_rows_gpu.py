"""Small FP64 and complex blocks in multivector applies: where the scalar rows run
instead of the tensor-core rows, forward (rows no staged kernel takes) and
adjoint, on both sides of the rule's lines, with the fused epilogue, against
the oracle's apply.  Tolerance 1e-12 of the largest value: sums of at most 41
blocks of 5 products, 210 roundings of 1.1e-16."""
import ctypes as C

import numpy as np
import pytest

from vbcsr_b200 import workloads as W

from .conftest import rel_err

pytestmark = pytest.mark.gpu


def _step(oracle, H, k, adjoint):
    import torch

    from vbcsr_b200 import _capi

    from . import _gpu

    cplx = np.iscomplexobj(H.values)
    rng = np.random.default_rng(k)
    X, P, D, A = (rng.normal(size=(H.N, k)) + (1j * rng.normal(size=(H.N, k)) if cplx else 0) for _ in range(4))
    dm = _gpu.dmat(H)
    x, p, d, acc = (_gpu.to_dev_mv(v, k, H.values.dtype) for v in (X, P, D, A))
    y = torch.zeros_like(x)
    dots = torch.zeros(2, dtype=torch.float64, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    c = 0.4 - 0.2j if cplx else 0.4
    _capi.call("vbg_cheb_step_adjoint" if adjoint else "vbg_cheb_step", dm.h, k, k, 1.7, -0.3, -1.0, ptr(x), ptr(p),
               ptr(y), ptr(d), ptr(dots), ptr(acc), float(np.real(c)), float(np.imag(c)), None)
    torch.cuda.synchronize()
    Y = 1.7 * oracle.apply(H, X, adjoint) - 0.3 * X - P
    assert rel_err(y.cpu().numpy(), Y) < 1e-12
    assert rel_err(acc.cpu().numpy(), A + c * Y) < 1e-12
    ref = np.array([np.sum((D.conj() * Y).real), np.sum(np.abs(Y) ** 2)])
    assert np.abs(dots.cpu().numpy() - ref).max() < 1e-12 * np.sum(np.abs(D) * np.abs(Y) + np.abs(Y) ** 2)
    return _capi.adjoint_kernel(dm, k) if adjoint else _capi.apply_kernel(dm, k)


def _phases(H, seed):
    H.values = H.values * np.exp(2j * np.pi * np.random.default_rng(seed).random(H.nnz))
    return H


@pytest.mark.parametrize("cplx,k", [(False, 8), (False, 24), (False, 48), (False, 128), (True, 4), (True, 16), (True, 40)])
@pytest.mark.parametrize("n,lo,hi", [(1200, 1, 1), (1199, 1, 1), (3600, 1, 1), (3600, 1, 3), (3599, 1, 3), (10800, 1, 3),
                                     (2500, 3, 3)])
def test_adjoint(oracle, dev, cplx, k, n, lo, hi):
    H = W.random_pattern(n, lo, hi, 4, seed=n)
    if cplx:
        _phases(H, n)
    idle = k in (24, 48, 40)  # lanes without a column: a quarter (48), more (24, 40)
    rows = 3600 if idle and not cplx else 1200
    small = hi == 1 if k in (24, 40) else lo == 1  # mean block of 1, of at most 7 values
    want = "lane_rows" if small and n >= rows * (hi - lo + 1) else "rows"
    assert _step(oracle, H, k, True) == want


@pytest.mark.parametrize("cplx,k", [(False, 8), (False, 48), (False, 128), (True, 4)])
@pytest.mark.parametrize("n,lo,hi", [(2400, 1, 2), (2399, 1, 2)])
def test_forward(oracle, dev, cplx, k, n, lo, hi):
    H = W.random_pattern(n, lo, hi, 40, seed=n)
    if cplx:
        _phases(H, n)
    # (rows of a multiple of 512 bytes: the pipelined kernel; 48 columns leave lanes idle)
    want = "pipe" if k == 128 else "lane_rows" if n == 2400 and k != 48 else "rows"
    assert _step(oracle, H, k, False) == want


@pytest.mark.parametrize("cplx,k,adjoint", [(False, 2, False), (False, 4, True), (True, 2, False), (True, 2, True)])
@pytest.mark.parametrize("n", [7999, 8000])
def test_rows_of_32_bytes(oracle, dev, cplx, k, adjoint, n):
    H = W.random_pattern(n, 2, 4, 5, seed=n)
    if cplx:
        _phases(H, n)
    assert _step(oracle, H, k, adjoint) == ("lane_rows" if n == 8000 else "rows")


@pytest.mark.parametrize("k,want", [(4, "lane_rows"), (8, "rows"), (24, "lane_rows"), (48, "rows"), (32, "lane_rows"), (64, "lane_rows")])
def test_complex_adjoint_on_many_rows(oracle, dev, k, want):
    H = _phases(W.tmd_lattice(52, seed=1)[0], 5)  # 8112 block rows of 3 and 5, mean 14.3 values a block
    assert _step(oracle, H, k, True) == want


@pytest.mark.parametrize("cplx,k,n,lo,hi,want", [
    (False, 64, 500, 2, 4, "rows"), (False, 64, 2999, 3, 5, "rows"), (False, 64, 3000, 3, 5, "pipe"),
    (False, 128, 1500, 2, 4, "pipe"), (True, 32, 2499, 2, 4, "rows"), (True, 64, 1250, 2, 4, "pipe"),
    (False, 64, 5000, 8, 8, "rows")])
def test_rows_of_512_bytes_without_tiles(oracle, dev, cplx, k, n, lo, hi, want):
    H = W.random_pattern(n, lo, hi, 10 if hi == 8 else 40, seed=n)
    if cplx:
        _phases(H, n)
    assert _step(oracle, H, k, False) == want
