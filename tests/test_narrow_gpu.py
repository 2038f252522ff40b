"""Narrow multivectors on the tiled applies at their edges: rows of 128 and 256
bytes (FP64 16 and 32 columns, complex 8 and 16) on the tensor-core tiles, FP32
at 16 and 32 columns on the two-stage tiles; blocks of 1 to 8, empty block rows,
tiles with a remainder, one tile per CTA and several; and the rows that take
over where no tiles fit.  FP64 tolerance 1e-12 of the largest value: sums of at
most 41 blocks of 3 or 13 of 8 products and the epilogue, 130 roundings of
1.1e-16."""
import ctypes as C

import numpy as np
import pytest

from vbcsr_b200 import workloads as W

from .conftest import rel_err

pytestmark = pytest.mark.gpu


def _banded(n, cplx=False):
    """Blocks of 1 to 8 within six of the diagonal; every 11th block row empty."""
    H = W.banded_decaying(n, size_min=1, size_max=8, neighbours=4, band=6, seed=n)
    off = H.slot_offsets()
    rows = np.repeat(np.arange(H.n), np.diff(H.row_ptr))
    keep = np.nonzero(rows % 11 != 5)[0]
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows[keep], minlength=H.n))]).astype(np.int32)
    v = np.concatenate([H.values[off[s]:off[s + 1]] for s in keep])
    if cplx:
        v = v * np.exp(2j * np.pi * np.random.default_rng(n).random(len(v)))
    return W.BlockCSR(H.block_sizes, rp, H.col_ind[keep], v)


def _check_step(oracle, H, k, want):
    """Y = alpha A X + beta X + gamma P, dots against D, acc += c Y."""
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
    _capi.call("vbg_cheb_step", dm.h, k, k, 1.7, -0.3, -1.0, ptr(x), ptr(p), ptr(y), ptr(d), ptr(dots), ptr(acc),
               float(np.real(c)), float(np.imag(c)), None)
    torch.cuda.synchronize()
    assert _capi.apply_kernel(dm, k) == want
    Y = 1.7 * oracle.apply(H, X) - 0.3 * X - P
    assert rel_err(y.cpu().numpy(), Y) < 1e-12
    assert rel_err(acc.cpu().numpy(), A + c * Y) < 1e-12
    ref = np.array([np.sum((D.conj() * Y).real), np.sum(np.abs(Y) ** 2)])
    assert np.abs(dots.cpu().numpy() - ref).max() < 1e-12 * np.sum(np.abs(D) * np.abs(Y) + np.abs(Y) ** 2)
    # no dots, beta and gamma 0, dots with X itself
    _capi.call("vbg_cheb_step", dm.h, k, k, 1.0, 0.0, 0.0, ptr(x), None, ptr(y), None, None, None, 0.0, 0.0, None)
    Z = oracle.apply(H, X)
    assert rel_err(y.cpu().numpy(), Z) < 1e-12
    _capi.call("vbg_cheb_step", dm.h, k, k, 1.0, 0.0, 0.0, ptr(x), None, ptr(y), None, ptr(dots), None, 0.0, 0.0, None)
    torch.cuda.synchronize()
    assert abs(dots.cpu().numpy()[0] - np.sum((X.conj() * Z).real)) < 1e-12 * np.sum(np.abs(X) * np.abs(Z))
    assert _capi.device_status(clear=True) == 0


@pytest.mark.parametrize("n", [1, 37, 605, 6001])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("pieces", [1, 2])
def test_tensor_core_tiles(oracle, dev, n, cplx, pieces):
    _check_step(oracle, _banded(max(n, 1), cplx) if n > 13 else W.random_pattern(n, 5, 5, 0, seed=1,
                dtype=np.complex128 if cplx else np.float64), pieces * (8 if cplx else 16), "tile")


@pytest.mark.parametrize("cplx,k", [(False, 16), (False, 32), (False, 64), (True, 8), (True, 32)])
def test_rows_where_no_tiles_fit(oracle, dev, cplx, k):
    H = W.random_pattern(3000, 4, 8, 12, seed=5)
    if cplx:
        H.values = H.values * np.exp(2j * np.pi * np.random.default_rng(1).random(H.nnz))
    _check_step(oracle, H, k, "rows")


@pytest.mark.parametrize("cplx,k,want", [(False, 32, "rows"), (False, 64, "pipe"), (True, 16, "pipe"), (True, 64, "pipe")])
def test_small_blocks_where_no_tiles_fit(oracle, dev, cplx, k, want):
    H = W.random_pattern(3000, 1, 3, 40, seed=6)
    if cplx:
        H.values = H.values * np.exp(2j * np.pi * np.random.default_rng(1).random(H.nnz))
    _check_step(oracle, H, k, want)


@pytest.mark.parametrize("n", [37, 605, 9001])
@pytest.mark.parametrize("k", [16, 32])
def test_fp32_tiles(oracle, dev, n, k):
    """Moments of a matrix with row sums below 1.  A step's 110 roundings of
    6e-8 are 7e-6 of an entry at most, after the four steps of eight moments
    (1 + 3 + 5 + 7) times that, 1e-4; a moment adds N k > 2500 entries'
    errors of either sign over mu_0 = N k, 1/50 of it: 2e-6."""
    from vbcsr_b200 import _capi

    from . import _gpu

    H = _banded(n)
    H.values = H.values / W.gershgorin_bound(H)
    V = np.where(np.random.default_rng(k).random((H.N, k)) < 0.5, -1.0, 1.0)
    dm = _gpu.dmat(H)
    mu = _gpu.kpm_moments(dm, V, 8, precision=1)
    assert _capi.apply_kernel(dm, k, precision=1) == "tile"
    ref = oracle.kpm_moments(H, V, 8, True)
    assert np.abs(mu - ref).max() / abs(ref[0]) < 2e-6
    assert np.array_equal(mu, _gpu.kpm_moments(_gpu.dmat(H), V, 8, precision=1))
    assert _capi.device_status(clear=True) == 0


@pytest.mark.parametrize("n,lo,hi", [(37, 8, 8), (1500, 1, 2), (1501, 4, 8), (5003, 3, 5)])
@pytest.mark.parametrize("k", [16, 32])
def test_fp32_short_tiles(oracle, dev, n, lo, hi, k):
    """Random patterns, whose tiles are too short for two stages (but for the
    smallest matrix); tolerance as above, rows of 13 blocks of at most 8."""
    from vbcsr_b200 import _capi

    from . import _gpu

    H = W.random_pattern(n, lo, hi, 12, seed=n)
    H.values = (H.values - 0.5) / W.gershgorin_bound(H)
    V = np.where(np.random.default_rng(k).random((H.N, k)) < 0.5, -1.0, 1.0)
    dm = _gpu.dmat(H)
    mu = _gpu.kpm_moments(dm, V, 8, precision=1)
    assert _capi.apply_kernel(dm, k, precision=1) == "tile"
    assert n == 37 or _capi.apply_tile_rows(dm, k, precision=1) < 8
    ref = oracle.kpm_moments(H, V, 8, True)
    assert np.abs(mu - ref).max() / abs(ref[0]) < 2e-6
    assert np.array_equal(mu, _gpu.kpm_moments(_gpu.dmat(H), V, 8, precision=1))
    assert _capi.device_status(clear=True) == 0


def _chains(H, X, chains):
    """A X with every row's products added four at a time to `chains` sums in turn,
    as fused multiply-adds of 64 bits, and the sums added; and in long double."""
    so = H.scalar_offsets()
    rows, cols = W.scalar_coords(H)
    order = np.lexsort((cols, rows))  # the q-list's order: ascending columns
    rows, cols, v = rows[order], cols[order], H.values[order]
    m = np.bincount(rows, minlength=H.N)
    at = np.arange(len(rows)) - np.repeat(np.cumsum(m) - m, m)
    A = np.zeros((H.N, m.max()), np.longdouble)
    J = np.zeros((H.N, m.max()), np.int64)
    A[rows, at], J[rows, at] = v, cols
    Xl = X.astype(np.longdouble)
    s = np.zeros((chains, H.N, X.shape[1]))
    exact = np.zeros((H.N, X.shape[1]), np.longdouble)
    for q in range(m.max()):
        p = A[:, q, None] * Xl[J[:, q]]
        s[q // 4 % chains] = (s[q // 4 % chains].astype(np.longdouble) + p).astype(np.float64)
        exact += p
    assert so[-1] == H.N
    return sum(s[1:], s[0]), exact


@pytest.mark.parametrize("k", [16, 32])
def test_tensor_core_tiles_rounding(dev, k):
    """The rounding error of a tile's sums is that of two chains, which a single
    chain exceeds by a third: the root mean squares over 2156 k entries differ by
    less than a tenth between two orders of the same chain lengths."""
    from vbcsr_b200 import _capi

    from . import _gpu

    H = W.tmd_lattice(14, seed=1)[0]
    X = np.random.default_rng(k).standard_normal((H.N, k))
    dm = _gpu.dmat(H)
    y = _gpu.apply(dm, X)
    assert _capi.apply_kernel(dm, k) == "tile"
    two, exact = _chains(H, X, 2)
    one, _ = _chains(H, X, 1)
    rms = lambda a: float(np.sqrt(np.mean((a.astype(np.longdouble) - exact) ** 2)))  # noqa: E731
    assert rms(one) > 1.2 * rms(two)
    assert rms(y) < 1.1 * rms(two)


@pytest.mark.parametrize("cplx,k", [(False, 16), (False, 64), (True, 8)])
def test_short_tiles_are_not_planned(oracle, dev, cplx, k):
    """Tiles that the choice has no use for (below 8 block rows) are not built."""
    from vbcsr_b200 import _capi

    from . import _gpu

    H = W.random_pattern(1500, 2, 4, 12, seed=7)
    if cplx:
        H.values = H.values * np.exp(2j * np.pi * np.random.default_rng(1).random(H.nnz))
    rng = np.random.default_rng(k)
    X = rng.normal(size=(H.N, k)) + (1j * rng.normal(size=(H.N, k)) if cplx else 0)
    dm = _gpu.dmat(H)
    assert rel_err(_gpu.apply(dm, X), oracle.apply(H, X)) < 1e-12
    assert _capi.apply_kernel(dm, k) == ("pipe" if cplx else "rows")
    assert _capi.apply_tile_rows(dm, k) == 0
