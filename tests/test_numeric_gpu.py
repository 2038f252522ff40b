"""The tensor-core numeric phase of the SpGEMM at its edges, against the
oracle: dense bands (all J columns per pass) and sparse products (each
column's own pairs), an odd number of rows (the last pair has one row), a
single row, rows spanning more than the window table (binary search), one row
with several hundred blocks (does not fit shared memory: the item kernel),
blocks of 1 and of 8, empty rows.  Patterns equal but for blocks within 1e-10
of the threshold, values to 1e-12 of the largest (sums of at most 8 x 400
products)."""
import numpy as np
import pytest

from vbcsr_b200 import workloads as W

from .test_spgemm_gpu import assert_same_result

pytestmark = pytest.mark.gpu


def _pattern(n, size, pairs, seed, cplx):
    """A matrix of the given (row, column) blocks."""
    rng = np.random.default_rng(seed)
    bsz = rng.integers(size[0], size[1] + 1, size=n)
    so = np.zeros(n + 1, np.int64)
    np.cumsum(bsz, out=so[1:])
    key = np.unique(np.array([i * n + j for i, j in pairs], np.int64))
    r, c = key // n, key % n
    D = rng.normal(size=(so[-1], so[-1]))
    return W.from_dense_blocks(bsz, r, c, D + 1j * rng.normal(size=D.shape) if cplx else D)


def _matrix(name, cplx):
    if name == "dense_band":
        n = 61
        return _pattern(n, (1, 8), [(i, j) for i in range(n) for j in range(max(0, i - 12), min(n, i + 13))], 1, cplx)
    if name == "one_row":
        return _pattern(1, (8, 8), [(0, 0)], 2, cplx)
    if name == "eights":
        return _pattern(20, (8, 8), [(i, (i + k) % 20) for i in range(20) for k in (0, 1, 5)], 3, cplx)
    if name == "empty_rows":
        return _pattern(31, (1, 4), [(i, (7 * i + k) % 31) for i in range(0, 31, 3) for k in range(4)], 4, cplx)
    if name == "long_row":  # row 0 and column 0 full
        n = 420
        return _pattern(n, (1, 3), [(0, j) for j in range(n)] + [(j, 0) for j in range(n)] + [(j, j) for j in range(n)],
                        5, cplx)
    H = W.random_pattern(1401, 1, 5, 3, seed=6, dtype=np.complex128 if cplx else np.float64)  # far columns
    return H


@pytest.mark.parametrize("name", ["dense_band", "one_row", "eights", "empty_rows", "long_row", "far"])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("thr", [0.0, 0.5])
def test_product(oracle, dev, name, cplx, thr):
    from . import _gpu

    A = _matrix(name, cplx)
    dA = _gpu.dmat(A)
    C, stats = dA.spgemm(dA, thr)
    O, ostats = oracle.spgemm(A, A, thr)
    assert stats[0] == ostats[0]
    assert_same_result(C.to_blockcsr(), O, thr)


@pytest.mark.parametrize("cplx", [False, True])
def test_hermitian_product_of_a_dense_band(oracle, dev, cplx):
    from . import _gpu

    A = _matrix("dense_band", cplx)
    D = A.to_dense()
    so = A.scalar_offsets()
    rows = np.repeat(np.arange(A.n), np.diff(A.row_ptr))
    A = W.from_dense_blocks(A.block_sizes, rows, A.col_ind, D + D.conj().T)
    assert so[-1] == A.N
    dA = _gpu.dmat(A)
    C, _ = dA.spgemm_hermitian(dA, 0.3)
    O, _ = oracle.spgemm_hermitian(A, A, 0.3)
    assert_same_result(C.to_blockcsr(), O, 0.3)
