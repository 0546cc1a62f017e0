"""Pointers of matrices with wide empty ranges: gaps around the widths that a thread
(32 entries), a warp and a whole tile (4,096) write, at both ends and in between,
bit-exact for rows and columns; and 8M columns whose nonzeros sit in 64 of them,
which must not be slower than the same nonzeros spread out."""
import time

import numpy as np
import pytest

from gpu_util import dev

pytestmark = pytest.mark.gpu


def _check(torch, m, n, row, col, rows=True):
    from spmx import SpmspvHandle
    nnz = len(row)
    val = np.arange(nnz, dtype=np.float32)
    h = SpmspvHandle(m, n, nnz)
    h.InputCOO(nnz, dev(row, torch), dev(col, torch), dev(val, torch))
    h.ToCSC()
    h.check_device_error()
    by_row = np.lexsort((col, row))
    rp, cl, vl = (t.cpu().numpy() for t in h.get_csr())
    assert np.array_equal(rp, np.searchsorted(row[by_row], np.arange(m + 1)))
    assert np.array_equal(cl, col[by_row]) and np.array_equal(vl, val[by_row])
    by_col = by_row[np.argsort(col[by_row], kind="stable")]
    rw, cp, cv = (t.cpu().numpy() for t in h.get_csc())
    assert np.array_equal(cp, np.searchsorted(col[by_col], np.arange(n + 1)))
    assert np.array_equal(rw, row[by_col]) and np.array_equal(cv, val[by_col])


@pytest.mark.parametrize("extent", [31, 32, 33, 64, 4094, 4095, 4096, 4097, 8190, 8191, 8192, 8193, 20000])
def test_gaps(torch_cuda, extent):
    at = [[0], [extent - 1], [extent // 2], [0, extent - 1], [min(31, extent - 1)], [min(32, extent - 1)],
          [extent // 3, extent // 3 + 1], [max(extent - 4097, 0), extent - 1], [max(extent - 33, 0)],
          sorted({min(k, extent - 1) for k in (4095, 4096, 8191, 8192, 12287, 12290)})]
    rng = np.random.default_rng(extent)
    for used in at:
        for nnz in (1, 5, 131, 3000):
            here = rng.choice(used, nnz).astype(np.int32)
            other = rng.integers(0, 50, nnz).astype(np.int32)
            _check(torch_cuda, 50, extent, other, here)
            _check(torch_cuda, extent, 50, here, other)


def _columns(kind, n):
    rng = np.random.default_rng(3)
    return {"first": np.arange(64), "last": np.arange(n - 64, n), "clusters": np.r_[np.arange(32), np.arange(n - 32, n)],
            "spread": np.sort(rng.choice(n, 64, replace=False))}[kind]


@pytest.mark.parametrize("kind", ["first", "last", "clusters", "spread"])
def test_eight_million(torch_cuda, kind):
    torch = torch_cuda
    from spmx import SpmspvHandle
    n, nnz, small = 1 << 23, 1 << 20, 5000
    rng = np.random.default_rng(5)
    here = rng.choice(_columns(kind, n), nnz).astype(np.int32)
    even = (np.arange(nnz) * 8).astype(np.int32)
    other = rng.integers(0, small, nnz).astype(np.int32)
    _check(torch, small, n, other, here)
    _check(torch, n, small, here, other)

    def best(col):
        h = SpmspvHandle(small, n, nnz)
        h.InputCOO(nnz, dev(other, torch), dev(col, torch))
        ts = []
        for _ in range(12):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            h.ToCSC()
            ts.append(time.perf_counter() - t0)
        return min(ts)

    # host time of a synchronous call, best of twelve; a gap per thread took 12 to 160 times as long
    assert best(here) < 8 * best(even)
