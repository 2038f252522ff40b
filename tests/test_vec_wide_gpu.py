"""Vectors on matrices whose blocks are all over 8 (a kernel of its own) at
its edges: blocks up to 41 (two rounds of 32 outputs), a few rows (entries
split over the CTA's warps) and more, real and complex, both directions, the
fused epilogue with dots; and mixed sizes (the general kernel's wide rows).
Tolerance 1e-12 of the largest value: sums of at most 250 products."""
import ctypes as C

import numpy as np
import pytest

from vbcsr_b200 import workloads as W

from .conftest import rel_err

pytestmark = pytest.mark.gpu

_CASES = {"few": (20, 9, 41, 5), "one": (1, 33, 33, 1), "many": (3700, 9, 11, 3), "mixed": (50, 1, 40, 5)}


@pytest.mark.parametrize("name", list(_CASES))
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("adjoint", [False, True])
def test_wide_vector(oracle, dev, name, cplx, adjoint):
    import torch

    from vbcsr_b200 import _capi

    from . import _gpu

    n, lo, hi, per = _CASES[name]
    H = W.random_pattern(n, lo, hi, per, seed=41, dtype=np.complex128 if cplx else np.float64)
    rng = np.random.default_rng(3)

    def vec():
        v = rng.normal(size=H.N)
        return v + 1j * rng.normal(size=H.N) if cplx else v

    x, p, d = vec(), vec(), vec()
    dm = _gpu.dmat(H)
    ref = oracle.apply(H, x, adjoint)
    assert rel_err(_gpu.apply(dm, x, adjoint), ref) < 1e-12
    xd, pd, dd = (torch.from_numpy(v).cuda() for v in (x, p, d))
    yd = torch.zeros_like(xd)
    dots = torch.zeros(2, dtype=torch.float64, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    _capi.call("vbg_cheb_step_adjoint" if adjoint else "vbg_cheb_step", dm.h, 1, 1, 1.3, -0.2, -1.0, ptr(xd), ptr(pd),
               ptr(yd), ptr(dd), ptr(dots), None, 0.0, 0.0, None)
    torch.cuda.synchronize()
    y = 1.3 * ref - 0.2 * x - p
    assert rel_err(yd.cpu().numpy(), y) < 1e-12
    want = np.array([np.sum((d.conj() * y).real), np.sum(np.abs(y) ** 2)])
    assert np.abs(dots.cpu().numpy() - want).max() < 1e-12 * np.sum(np.abs(d) * np.abs(y) + np.abs(y) ** 2)


@pytest.mark.parametrize("name", list(_CASES))
def test_wide_vector_fp32(oracle, dev, name):
    """FP32 moments of one vector.  A step's 250 roundings of 6e-8 are 1.5e-5 of
    an entry at most, the three steps of six moments (1 + 3 + 5) times that,
    1.4e-4; a moment adds N > 30 entries' errors of either sign over mu_0 = N."""
    from . import _gpu

    n, lo, hi, per = _CASES[name]
    H = W.random_pattern(n, lo, hi, per, seed=41)
    H.values = (H.values - 0.5) / W.gershgorin_bound(H)
    V = np.where(np.random.default_rng(3).random((H.N, 1)) < 0.5, -1.0, 1.0)
    mu = _gpu.kpm_moments(_gpu.dmat(H), V, 6, precision=1)
    ref = oracle.kpm_moments(H, V, 6, True)
    assert np.abs(mu - ref).max() / abs(ref[0]) < 3e-5
