"""Infinities, NaNs of either sign, overflowing products, cancelled and negative
zeros through the dense double rows of the sorted write-back and of the bucket
method: a row is listed if and only if a nonzero reaches it, and its sum is that
of the rounded products."""
import numpy as np
import pytest

from gpu_util import make_handle, set_sparse

pytestmark = pytest.mark.gpu

SPECIAL = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, -np.nan, 3e38, -3e38, 1e-30, -1e-30], np.float32)


@pytest.mark.parametrize("full_row", [False, True])  # combined per warp where a row may take many products
def test_rows(torch_cuda, full_row):
    from spmx.gen import Csr
    torch = torch_cuda
    m, n = 5000, 40000
    rng = np.random.default_rng(3)
    rows = np.r_[rng.integers(0, m - 1, 3 * n // 2), np.full(n if full_row else 0, m - 1)]
    cols = np.r_[rng.integers(0, n, 3 * n // 2), np.arange(n)[:n if full_row else 0]]
    key = np.unique(rows * n + cols)
    key = key[key // n % 7 != 3]  # rows without a nonzero
    rows, cols = key // n, (key % n).astype(np.int32)
    val = SPECIAL[rng.integers(0, len(SPECIAL), len(rows))]
    # three quarters of the rows from zeros alone, so that sums of zeros are there too
    quiet = rows % 4 != 0
    val[quiet] = SPECIAL[rng.integers(0, 4, int(quiet.sum()))]
    A = Csr(m, n, np.searchsorted(rows, np.arange(m + 1)).astype(np.int32), cols, val)
    h = make_handle(A, torch, hola=False)
    xkey = np.sort(rng.choice(n, 36000, replace=False)).astype(np.int32)
    xval = SPECIAL[rng.integers(0, len(SPECIAL), len(xkey))]
    xval[rng.random(len(xkey)) < 0.7] = np.float32(-0.0)
    keep = set_sparse(h, xkey, xval, torch)
    x = np.zeros(n, np.float32)
    x[xkey] = xval
    used = np.isin(cols, xkey)
    with np.errstate(all="ignore"):
        prod = val[used] * x[cols[used]]
        e = np.zeros(m)
        np.add.at(e, rows[used], prod.astype(np.float64))
        mag = np.zeros(m)
        np.add.at(mag, rows[used], np.abs(prod.astype(np.float64)))
        e32 = e.astype(np.float32)
    touched = np.unique(rows[used])
    assert 1000 < len(touched) < m and np.isnan(e32).any() and np.isinf(e32).any()
    assert (e32[touched] == 0).any() and (not full_row or touched[-1] == m - 1)
    for bucket in (False, True):
        y = torch.full((m,), 3.0, device="cuda")
        yk = torch.full((m,), -1, dtype=torch.int32, device="cuda")
        yv = torch.full((m,), 3.0, device="cuda")
        k = h.CscBasedBucketSpmspv(1.0, y, yk, yv) if bucket else h.spmspv_csc(2, 1, 1.0, y, yk, yv)
        assert np.array_equal(yk[:k].cpu().numpy(), touched)
        for got, want, size in ((y.cpu().numpy(), e32, mag), (yv[:k].cpu().numpy(), e32[touched], mag[touched])):
            assert np.array_equal(np.isnan(got), np.isnan(want))
            ok = np.isfinite(want)
            assert np.array_equal(got[~ok & ~np.isnan(want)], want[~ok & ~np.isnan(want)])
            # doubles in any order: exact but for the last rounding
            assert np.all(np.abs(got[ok].astype(np.float64) - want[ok]) <= 2.0 ** -23 * np.abs(want[ok]) +
                          2.0 ** -40 * size[ok])
    h.check_device_error()
    assert keep
