"""Outer products on a pattern at the edges of their forms: one operand a lane
(8 real, 4 complex columns), four (32 and 16), the general form beyond; a few
rows (a row's blocks over several warps), one round of warps, two rounds, many;
rows that start off a 16-byte boundary; against the products in numpy.
Tolerance 1e-12 of the largest value: sums of at most 40 products."""
import ctypes as C

import numpy as np
import pytest

from vbcsr_b200 import workloads as W

pytestmark = pytest.mark.gpu

_ROWS = {"few": (37, 8), "wave": (1190, 9), "two": (2400, 4), "many": (9600, 1), "thin": (2400, 1)}


@pytest.mark.parametrize("rows", list(_ROWS))
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("k", [1, 4, 5, 8, 9, 16, 17, 32, 33])
def test_sddmm(dev, rows, cplx, k):
    import torch

    from vbcsr_b200 import _capi

    from . import _gpu

    n, per = _ROWS[rows]
    H = W.random_pattern(n, 1, 8, per, seed=n, dtype=np.complex128 if cplx else np.float64)
    rng = np.random.default_rng(k)
    ld = k + (k % 2 if k % 3 else 0)  # odd and even leading dimensions
    mv = lambda: rng.normal(size=(H.N, ld)) + (1j * rng.normal(size=(H.N, ld)) if cplx else 0)  # noqa: E731
    G, X, old = mv(), mv(), rng.normal(size=H.nnz) * (1 + (0.5j if cplx else 0))
    alpha = 1.5 - 0.5j if cplx else 1.5
    r, c = W.scalar_coords(H)
    want = old + alpha * np.sum(G[r, :k] * X[c, :k].conj(), axis=1)
    dm = _gpu.dmat(H)
    g, x, out = (torch.from_numpy(v).cuda() for v in (G, X, old.copy()))
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    _capi.call("vbg_sddmm", dm.h, k, ld, ptr(g), ptr(x), float(np.real(alpha)), float(np.imag(alpha)), ptr(out), None)
    torch.cuda.synchronize()
    assert np.abs(out.cpu().numpy() - want).max() < 1e-12 * np.abs(want).max()
