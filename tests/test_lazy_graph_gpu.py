"""Matrices whose graph is read from the device on first use: products, sums,
filters and duplicates give the structure they have at that moment, the graph
stays one object while the pattern does, and values come back the same by
every way."""
import numpy as np
import pytest

from vbcsr_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture()
def pair():
    from vbcsr_b200 import VBCSR

    H = W.banded_decaying(60, neighbours=3, band=8, seed=2)
    return H, VBCSR.from_block_csr(H.block_sizes, H.row_ptr, H.col_ind, H.values)


def test_product_then_filter(pair, dev):
    H, A = pair
    D = H.to_dense()
    C = A.spmm(A, 0.0)
    assert C.shape == A.shape and C.nnz == len(C.get_values())
    full = C.local_block_nnz
    assert np.allclose(C.to_dense(), D @ D, rtol=0, atol=1e-12 * np.abs(D @ D).max())
    E = A.spmm(A, 0.0)  # its graph not asked for before the filter
    E.filter_blocks(0.5)
    assert E.local_block_nnz < full and len(E.col_ind) == E.local_block_nnz == int(E.row_ptr[-1])
    g = E.graph
    E.scale(2.0)
    E.axpby(1.0, E.duplicate(), 1.0)  # same pattern: the same graph
    assert E.graph is g
    E.axpby(1.0, A, 1.0)  # a union: another one
    assert len(E.col_ind) == E.local_block_nnz
    v = E.create_vector()
    v.from_numpy(np.ones(H.N))
    assert np.allclose(E.mult(v).to_numpy(), E.to_dense() @ np.ones(H.N))


def test_duplicates_and_values(pair, dev):
    H, A = pair
    A.scale(1.0)  # on the device
    B = A.duplicate()
    B.shift(1.0)
    assert np.array_equal(A.get_values(), H.values)
    assert np.allclose(B.to_dense(), H.to_dense() + np.eye(H.N), rtol=0, atol=1e-15)
    shared = A.duplicate(independent_graph=False)
    assert shared.graph is A.graph and B.graph is not A.graph
    assert np.array_equal(shared.col_ind, H.col_ind) and np.array_equal(shared.row_ptr, H.row_ptr)
    B.fill(3.0)  # a host change after the device's
    assert np.all(B.get_values() == 3.0) and B.matrix_kind == A.matrix_kind
    T = A.transpose()
    assert np.array_equal(T.to_dense(), H.to_dense().T)
    assert T.get_block(0, 0).shape == (H.block_sizes[0], H.block_sizes[0])


@pytest.mark.parametrize("n", [60, 2500])  # below and above the megabyte that get_values keeps
def test_values_again_after_changes(n, dev):
    from vbcsr_b200 import VBCSR

    H = W.banded_decaying(n, neighbours=4, band=8, seed=3)
    assert (H.nnz * 8 > 1 << 20) == (n == 2500)
    A = VBCSR.from_block_csr(H.block_sizes, H.row_ptr, H.col_ind, H.values)
    A.scale(2.0)
    first = A.get_values()
    assert np.array_equal(first, 2.0 * H.values) and np.array_equal(A.get_values(), first)
    first[:] = 0.0  # the caller's own array
    assert np.array_equal(A.get_values(), 2.0 * H.values)
    A.scale(0.5)
    assert np.array_equal(A.get_values(), H.values)
    assert np.array_equal(A.get_block(1, 1).ravel(), H.values[H.slot_offsets()[H.row_ptr[1] + list(
        H.col_ind[H.row_ptr[1]:H.row_ptr[2]]).index(1)]:][:A.get_block(1, 1).size])
    A.fill(3.0)
    assert np.all(A.get_values() == 3.0)
    A.scale(2.0)
    assert np.all(A.get_values() == 6.0)
