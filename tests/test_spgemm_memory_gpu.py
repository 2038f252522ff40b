"""A product whose one-pass symbolic list does not fit what device memory is left
counts first and writes in a second pass, with the same result."""
import numpy as np
import pytest

from vbcsr_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_symbolic_list_without_memory(dev):
    """16000 single values a row of 121: 14500 columns a row by the bound, 0.9 GB
    of list, beside 0.3 GB of tables; 0.7 GB are left."""
    import torch

    from vbcsr_b200 import _capi

    n, per = 16000, 120
    rng = np.random.default_rng(1)
    rows = np.repeat(np.arange(n), per)
    key = np.unique(np.concatenate([rows * n + rng.integers(0, n, n * per), np.arange(n) * (n + 1)]))
    rows, cols = key // n, key % n
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    v = np.where(rows == cols, 1.0, 1e-6)
    H = W.BlockCSR(np.ones(n, np.int64), rp, cols.astype(np.int32), v)
    dm = _capi.DeviceMatrix.create(H.block_sizes, H.row_ptr, H.col_ind, H.values)

    def product():
        C, stats = dm.spgemm(dm, 0.5)
        out = C.to_blockcsr()
        return out.col_ind, out.values, stats[:3]

    want = product()
    assert np.array_equal(want[0], np.arange(n)) and np.abs(want[1] - 1.0).max() < 1e-9
    torch.cuda.synchronize()
    _capi.call("vbg_memory_trim")
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(max(free - 700 * 2**20, 0), dtype=torch.uint8, device="cuda")
    try:
        got = product()
    finally:
        del hog
        torch.cuda.empty_cache()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]) and got[2] == want[2]
