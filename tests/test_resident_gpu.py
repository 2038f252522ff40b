"""Vector recurrences with the matrix resident in shared memory against the
same recurrence in numpy on the oracle's apply: the series with its
checkpoints, and the column form with sources in both directions.  Sizes: one
CTA, a few block rows per CTA, rows of different lengths, non-symmetric
patterns; fewer steps than the resident kernel takes and a matrix that does
not fit run the step-by-step form.  Tolerance 1e-11 of the largest value:
recurrences of up to 40 steps on spectra inside [-1, 1] (rounding grows with
the step count, 1e-13 measured on the CPU)."""
import ctypes as C

import numpy as np
import pytest

from vbcsr_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _matrix(name):
    if name == "lattice":
        return W.tmd_lattice(9, seed=5, Ly=7, bond_phase=True)[0]
    if name == "one_row":
        H = W.random_pattern(1, 8, 8, 1, seed=6, dtype=np.complex128)
    elif name == "real":
        H = W.random_pattern(400, 1, 8, 7, seed=7)
    else:
        H = W.random_pattern(333, 1, 8, 5, seed=8, dtype=np.complex128)
    H.values = H.values / W.gershgorin_bound(H)
    return H


def _ptr(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def _vec(H, rng):
    v = rng.normal(size=H.N)
    return v + 1j * rng.normal(size=H.N) if np.iscomplexobj(H.values) else v


@pytest.mark.parametrize("name", ["lattice", "one_row", "real", "random"])
@pytest.mark.parametrize("M,K", [(40, 0), (33, 16), (12, 1), (17, 5), (4, 16)])
def test_series_and_checkpoints(oracle, dev, name, M, K):
    import torch

    from vbcsr_b200 import _capi

    from . import _gpu

    H = _matrix(name)
    rng = np.random.default_rng(M)
    v = _vec(H, rng)
    c = rng.normal(size=M) + (1j * rng.normal(size=M) if np.iscomplexobj(v) else 0.0)
    scale, center = 1.1, 0.05
    t = [v, (oracle.apply(H, v) - center * v) / scale]
    while len(t) < M:
        t.append(2 * (oracle.apply(H, t[-1]) - center * t[-1]) / scale - t[-2])
    psi = sum(ci * ti for ci, ti in zip(c, t[:M]))
    dm = _gpu.dmat(H)
    vd = torch.from_numpy(v).cuda()
    out = torch.empty_like(vd)
    n_ck = (M - 1) // K if K else 0
    ck = torch.full((max(2 * n_ck, 1), H.N), 7.0, dtype=vd.dtype, device="cuda")
    cf = np.ascontiguousarray(np.stack([np.real(c), np.imag(c)], axis=1))
    for _ in range(2):
        _capi.call("vbg_cheb_series", dm.h, 1, 1, _ptr(vd), M, cf.ctypes.data_as(C.c_void_p), scale, center, _ptr(out),
                   K, _ptr(ck), None)
        torch.cuda.synchronize()
        assert np.abs(out.cpu().numpy() - psi).max() < 1e-11 * np.abs(psi).max()
        for j in range(n_ck):
            n = (j + 1) * K
            for w in (0, 1):
                assert np.abs(ck[2 * j + w].cpu().numpy() - t[n - w]).max() < 1e-11 * np.abs(t[n - w]).max()
    assert _capi.device_status(clear=True) == 0


@pytest.mark.parametrize("name", ["lattice", "one_row", "real", "random"])
@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("steps", [0, 2, 4, 19])
@pytest.mark.parametrize("with_prev", [False, True])
def test_columns(oracle, dev, name, adjoint, steps, with_prev):
    import torch

    from vbcsr_b200 import _capi

    from . import _gpu

    H = _matrix(name)
    rng = np.random.default_rng(steps)
    x0, x1, g = _vec(H, rng), _vec(H, rng), _vec(H, rng)
    coef = rng.normal(size=(steps, 5)) * 0.5
    ys, p = [x0], x1 if with_prev else np.zeros_like(x1)
    for a, b, gm, re, im in coef:
        cc = re + 1j * im if np.iscomplexobj(x0) else re
        y = a * oracle.apply(H, ys[-1], adjoint) + b * ys[-1] + gm * p + cc * g
        p = ys[-1]
        ys.append(y)
    dm = _gpu.dmat(H)
    x0d, x1d, gd = (torch.from_numpy(v).cuda() for v in (x0, x1, g))
    # columns backwards, the last vector outside: ncol = steps + 1 - 1
    ncol = max(steps, 1)
    cols = torch.full((H.N, ncol + 2), 3.0, dtype=x0d.dtype, device="cuda")
    last, before = torch.zeros_like(x0d), torch.zeros_like(x0d)
    _capi.call("vbg_cheb_columns", dm.h, int(adjoint), _ptr(x0d), _ptr(x1d) if with_prev else None, steps,
               coef.ctypes.data_as(C.c_void_p), _ptr(gd), _ptr(cols), cols.stride(0), ncol, ncol - 1, -1, _ptr(last),
               _ptr(before), None)
    torch.cuda.synchronize()
    scale = max(np.abs(y).max() for y in ys)
    got = cols.cpu().numpy()
    for s in range(ncol):
        assert np.abs(got[:, ncol - 1 - s] - ys[s]).max() < 1e-11 * scale, s
    assert np.all(got[:, ncol:] == 3.0)
    assert np.abs(last.cpu().numpy() - ys[-1]).max() < 1e-11 * scale
    if steps or with_prev:
        assert np.abs(before.cpu().numpy() - (ys[-2] if steps else x1)).max() < 1e-11 * scale
    assert _capi.device_status(clear=True) == 0


def test_matrix_that_does_not_fit(dev):
    """37 MB of values: the series runs step by step, as with a forced kernel."""
    import torch

    from vbcsr_b200 import _capi

    from . import _gpu

    H = W.tmd_lattice(68, seed=9, bond_phase=True)[0]
    dm = _gpu.dmat(H)
    rng = np.random.default_rng(1)
    v = torch.from_numpy(_vec(H, rng)).cuda()
    cf = np.ascontiguousarray(rng.normal(size=(9, 2)))
    outs = []
    for forced in (0, 1):
        _capi.set_option("apply.vec_kernel", forced)
        try:
            out = torch.empty_like(v)
            _capi.call("vbg_cheb_series", dm.h, 1, 1, _ptr(v), 9, cf.ctypes.data_as(C.c_void_p), 1.0, 0.0, _ptr(out), 0,
                       None, None)
            torch.cuda.synchronize()
            outs.append(out.cpu().numpy())
        finally:
            _capi.set_option("apply.vec_kernel", 0)
    assert np.abs(outs[0] - outs[1]).max() < 1e-12 * np.abs(outs[1]).max()


def _series(dm, v, cf):
    import torch

    from vbcsr_b200 import _capi

    out = torch.empty_like(v)
    _capi.call("vbg_cheb_series", dm.h, 1, 1, _ptr(v), len(cf), cf.ctypes.data_as(C.c_void_p), 1.0, 0.0, _ptr(out), 0,
               None, None)
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("name", ["lattice", "one_row", "real", "random"])
@pytest.mark.parametrize("adjoint", [False, True])
def test_resident_once_the_steps_repay_the_plan(oracle, dev, name, adjoint):
    """Recurrences of seven steps run step by step until the matrix has run
    enough of them, then as one launch, in the direction asked for, with the
    same results."""
    import torch

    from vbcsr_b200 import _capi

    from . import _gpu

    H = _matrix(name)
    rng = np.random.default_rng(5)
    x = _vec(H, rng)
    dm = _gpu.dmat(H)
    xd = torch.from_numpy(x).cuda()
    steps = 7
    coef = np.ascontiguousarray(np.tile([1.9, -0.1, -1.0, 0.0, 0.0], (steps, 1)))
    p, y = np.zeros_like(x), x
    for _ in range(steps):
        p, y = y, 1.9 * oracle.apply(H, y, adjoint) - 0.1 * y - p
    calls = 0
    while not _capi.recurrence_resident(dm, adjoint):
        assert calls * steps < 12 + H.nnzb // 1500 + steps, "never resident"
        last = torch.empty_like(xd)
        _capi.call("vbg_cheb_columns", dm.h, int(adjoint), _ptr(xd), None, steps, coef.ctypes.data_as(C.c_void_p), None,
                   None, 0, 0, 0, 0, _ptr(last), None, None)
        torch.cuda.synchronize()
        assert np.abs(last.cpu().numpy() - y).max() < 1e-11 * np.abs(y).max()
        calls += 1
    assert calls > 1
    assert not _capi.recurrence_resident(dm, not adjoint)


def test_long_series_is_resident_at_once(dev):
    import torch

    from vbcsr_b200 import _capi

    from . import _gpu

    dm = _gpu.dmat(_matrix("lattice"))
    v = torch.from_numpy(_vec(_matrix("lattice"), np.random.default_rng(1))).cuda()
    _series(dm, v, np.ones((9, 2)))
    assert not _capi.recurrence_resident(dm)
    _series(dm, v, np.ones((64, 2)))
    assert _capi.recurrence_resident(dm)


def test_matrix_that_does_not_fit_is_never_resident(dev):
    import torch

    from vbcsr_b200 import _capi

    from . import _gpu

    H = W.tmd_lattice(68, seed=9, bond_phase=True)[0]
    dm = _gpu.dmat(H)
    v = torch.from_numpy(_vec(H, np.random.default_rng(1))).cuda()
    for _ in range(2):
        _series(dm, v, np.ones((256, 2)))
    assert not _capi.recurrence_resident(dm) and not _capi.recurrence_resident(dm, True)
