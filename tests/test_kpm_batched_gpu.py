"""Batched KPM: many Hamiltonians of uneven size in one device recurrence
(vbg_kpm_moments_batched) against the per-matrix FP64 moment loop on the same
vectors (1e-12 relative to mu_0) and the oracle, and the FP32 bulk batch's
DOS error (<= 1e-5)."""
import numpy as np
import pytest

from vbcsr_b200 import kpm as K
from vbcsr_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _batch(seed=4):
    return [W.tmd_lattice(L, seed=seed + L, disorder=1.0)[0] for L in (3, 7, 5, 4, 6)]


@pytest.mark.parametrize("R", [16, 64])
@pytest.mark.parametrize("two_moment", [True, False])
def test_batched_matches_single(dev, oracle, R, two_moment):
    from . import _gpu

    Hs = _batch()
    rng = np.random.default_rng(R)
    vecs = [np.where(rng.random((h.N, R)) < 0.5, -1.0, 1.0) for h in Hs]
    M = 40
    mu, sizes = K.batched_kpm_moments(Hs, M, precision="fp64", two_moment=two_moment, vectors=vecs)
    assert mu.shape == (len(Hs), M)
    for i, h in enumerate(Hs):
        ref = _gpu.kpm_moments(_gpu.dmat(h), vecs[i], M, 0, two_moment)
        assert np.abs(mu[i] - ref).max() / abs(ref[0]) < 1e-12, i
        assert sizes[i] == h.N
    o = oracle.kpm_moments(Hs[1], vecs[1], M, two_moment)
    assert np.abs(mu[1] - o).max() / abs(o[0]) < 1e-12


def test_batched_fp32_dos_error(dev):
    Hs = _batch(seed=9)
    M = 128
    mu64, sizes = K.batched_kpm_moments(Hs, M, num_random_vecs=16, precision="fp64", seed=3)
    mu32, _ = K.batched_kpm_moments(Hs, M, num_random_vecs=16, precision="fp32", seed=3)
    for i in range(len(Hs)):
        _, d64 = K.dos_from_moments(mu64[i] / (16 * sizes[i]), 300)
        _, d32 = K.dos_from_moments(mu32[i] / (16 * sizes[i]), 300)
        assert np.abs(d32 - d64).max() / np.abs(d64).max() < 1e-5


def test_batched_graph_replay_and_layout_change(dev):
    Hs = _batch(seed=11)
    a, _ = K.batched_kpm_moments(Hs, 24, seed=1, use_graph=True)
    b, _ = K.batched_kpm_moments(Hs, 24, seed=1, use_graph=True)
    assert np.array_equal(a, b)
    c, _ = K.batched_kpm_moments(Hs[:3], 24, seed=1, use_graph=True)
    assert c.shape == (3, 24)


def test_device_status_clean(dev):
    from vbcsr_b200 import _capi

    assert _capi.device_status(clear=True) == 0


@pytest.mark.parametrize("precision", [0, 1])
def test_segment_sums_over_chunk_edges(dev, precision):
    """Per-segment sums at the edges of the 512-row chunks: an empty segment,
    exactly one chunk, a single row, a whole number of chunks and a
    remainder.  The recurrence itself does not depend on the segments, so a
    segment's moment is the plain one restricted to its rows (FP64 sums
    1e-12 of mu_0; FP32 vectors 1e-5, one rounding of 6e-8 per step and
    element)."""
    import ctypes as C

    import torch

    from vbcsr_b200 import _capi

    H, _ = W.tmd_lattice(30, seed=8)
    seg = np.array([0, 0, 512, 513, 1537, H.n], np.int32)
    R, M = 16, 9
    V = np.where(np.random.default_rng(2).random((H.N, R)) < 0.5, -1.0, 1.0)
    i, j = W.scalar_coords(H)
    A = torch.sparse_coo_tensor(np.stack([i, j]), H.values, (H.N, H.N)).to_sparse_csr()
    Vt = torch.from_numpy(V)
    ts = [Vt, A @ Vt]
    while len(ts) < M:
        ts.append(2 * (A @ ts[-1]) - ts[-2])
    so = H.scalar_offsets()[seg]
    ref = np.array([[float((Vt * t)[a:b].sum()) for t in ts] for a, b in zip(so[:-1], so[1:])])
    dm = _capi.DeviceMatrix.create(H.block_sizes, H.row_ptr, H.col_ind, H.values)
    Vd = Vt.cuda().contiguous()
    mu = torch.full((len(seg) - 1, M), -1.0, dtype=torch.float64, device="cuda")
    for _ in range(2):  # the second call replays the graph (its counters were reset)
        _capi.call("vbg_kpm_moments_batched", dm.h, len(seg) - 1, seg.ctypes.data_as(C.POINTER(C.c_int)), R, R,
                   C.c_void_p(Vd.data_ptr()), M, precision, 0, 1, C.c_void_p(mu.data_ptr()), None)
        torch.cuda.synchronize()
        err = np.abs(mu.cpu().numpy() - ref).max(axis=1) / np.maximum(ref[:, 0], 1.0)
        assert err.max() < (1e-5 if precision else 1e-12), err
