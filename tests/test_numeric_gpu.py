"""The tensor-core numeric phase of the SpGEMM at its edges, against the
oracle: dense bands (all J columns per pass) and sparse products (each
column's own pairs), an odd number of rows (the last pair has one row), a
single row, rows spanning more than the window table (binary search), one row
of several hundred blocks, blocks of 1 and of 8, empty rows; and row pairs on
both sides of what the forms' shared memory holds, up to the item kernel.  Patterns equal but for blocks within 1e-10
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


def _form(A):
    """The form the kernel's rules choose for A A: shared memory of the longest
    merged row pair at eight and sixteen warps against an SM's and half an SM's."""
    cx = np.iscomplexobj(A.values)
    es, J = (16, 2) if cx else (8, 4)
    rows = [A.col_ind[A.row_ptr[i]:A.row_ptr[i + 1]] for i in range(A.n)]
    off = A.slot_offsets()
    merged = max(len(np.union1d(rows[i], rows[min(i + 1, A.n - 1)])) for i in range(0, A.n, 2))
    vals = max(off[A.row_ptr[min(i + 2, A.n)]] - off[A.row_ptr[i]] for i in range(0, A.n, 2))
    kc = max(16, (merged + 15) // 16 * 16)
    size = {w: (vals * es + 15) // 16 * 16 + kc * (36 + (4 * J + 1) * w) + 2048 + 1024 for w in (8, 16)}
    ln = np.diff(A.row_ptr)
    pairs = sum(int(ln[r].sum()) for r in rows)
    c = sum(len(np.unique(np.concatenate([rows[k] for k in r]))) if len(r) else 0 for r in rows)
    dense = pairs * A.n >= 0.45 * c * A.nnzb
    if size[8] > 226 * 1024:
        return "items"
    if not dense:
        return "sparse"
    if size[16] > 226 * 1024 and A.n < 8 * 148:  # fewer than four rounds of CTAs
        return "items"
    return "dense 8 x 2" if size[8] <= 113 * 1024 else "dense 16" if size[16] <= 226 * 1024 else "dense 8"


@pytest.mark.parametrize("cplx,n,extra,want", [
    (False, 90, 0, "dense 8 x 2"), (False, 120, 0, "dense 16"), (False, 180, -1004, "dense 8"),
    (False, 180, -1003, "items"), (False, 220, 0, "items"), (False, 220, -1100, "items"),
    (True, 40, 0, "dense 8 x 2"), (True, 80, 0, "dense 16"), (True, 104, -1080, "dense 8"), (True, 130, 0, "items"),
    (False, 180, 400, "sparse"), (False, 220, 400, "items"), (True, 104, 400, "sparse"), (True, 130, 400, "items")])
@pytest.mark.parametrize("thr", [0.0, 40.0])
def test_long_rows_of_every_form(oracle, dev, cplx, n, extra, want, thr):
    """Two full rows of n blocks of 8 above a diagonal, alone or with -extra rows of
    a diagonal block each (dense by the rule), and beside `extra` rows of eight
    (sparse); the threshold lies among the blocks' norms (8 to 100)."""
    from . import _gpu

    m = n + abs(extra)
    pairs = [(i, j) for i in (0, 1) for j in range(n)] + [(i, i) for i in range(m)]
    if extra > 0:
        pairs += [(i, n + (i * k) % extra) for i in range(n, m) for k in (3, 7, 11, 19, 23, 31, 37)]
    key = np.unique(np.array([i * m + j for i, j in pairs], np.int64))
    rng = np.random.default_rng(n)
    rows, cols = key // m, key % m
    v = rng.normal(size=len(key) * 64)
    if cplx:
        v = v + 1j * rng.normal(size=len(v))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))]).astype(np.int32)
    A = W.BlockCSR(np.full(m, 8, np.int64), rp, cols.astype(np.int32), v)
    assert _form(A) == want
    dA = _gpu.dmat(A)
    C, stats = dA.spgemm(dA, thr)
    O, ostats = oracle.spgemm(A, A, thr)
    assert stats[0] == ostats[0] and (thr == 0.0 or 0 < len(O.col_ind) < C.nnzb + len(O.col_ind))
    assert_same_result(C.to_blockcsr(), O, thr)
