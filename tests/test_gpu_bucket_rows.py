"""The bucket SpMSpV: bucket counts asked for from 1 to 4,000, rows of many pairs, x
sizes around 512 and 4,096 entries, a row out of range, and its outputs in every
combination."""
import numpy as np
import pytest

from conftest import rand_csr
from gpu_util import dev, make_handle, set_sparse
import oracle.oracle as orc

pytestmark = pytest.mark.gpu
RTOL = 1e-5


@pytest.fixture(scope="module")
def mat():
    rng = np.random.default_rng(1)
    lens = rng.integers(0, 4, 300000)
    lens[5] = lens[299999] = 3000  # rows that many columns meet
    return rand_csr(300000, 9000, lens=lens, seed=2)


@pytest.mark.parametrize("k", [1, 511, 512, 513, 4097, 9000])
@pytest.mark.parametrize("buckets", [1, 37, 256, 1024, 1025, 4000])
def test_buckets(torch_cuda, mat, k, buckets):
    torch = torch_cuda
    h = make_handle(mat, torch, hola=False)
    rng = np.random.default_rng(k)
    key = np.sort(rng.choice(mat.n, k, replace=False)).astype(np.int32)
    val = rng.uniform(-1, 1, k).astype(np.float32)
    keep = set_sparse(h, key, val, torch)
    colptr, row, cval = mat.to_csc()
    y64, mag, touched = orc.spmspv_csc_f64(mat.m, colptr, row, cval, key, val)
    rows = np.flatnonzero(touched)
    y = torch.full((mat.m,), 3.0, device="cuda")
    yk, yv = torch.empty(mat.m, dtype=torch.int32, device="cuda"), torch.empty(mat.m, device="cuda")
    for outs in ((y, yk, yv), (None, yk, yv), (y, None, None)):
        n = h.CscBasedBucketSpmspv(1.0, *outs, buckets=buckets)
        assert n == len(rows)
        if outs[0] is not None:
            assert orc.within_tol(y.cpu().numpy(), y64, mag, RTOL)[0]
        if outs[1] is not None:
            assert np.array_equal(yk[:n].cpu().numpy(), rows)
            assert orc.within_tol(yv[:n].cpu().numpy(), y64[rows], mag[rows], RTOL)[0]
    h.check_device_error()
    assert keep


def test_row_out_of_range(torch_cuda):
    torch = torch_cuda
    from spmx import SpmspvHandle, SpmxError
    h = SpmspvHandle(100, 3, 6)
    row, colptr = np.array([1, 100, 5, -1, 5, 99], np.int32), np.array([0, 2, 4, 6], np.int32)
    t = [dev(a, torch) for a in (row, colptr, np.ones(6, np.float32))]
    h.InputCSC(6, *t)
    keep = set_sparse(h, np.arange(3, dtype=np.int32), np.ones(3, np.float32), torch)
    y = torch.empty(100, device="cuda")
    assert h.CscBasedBucketSpmspv(1.0, y) == 3
    e = np.zeros(100, np.float32)
    e[[1, 5, 99]] = 1, 2, 1
    assert np.array_equal(y.cpu().numpy(), e)
    with pytest.raises(SpmxError):
        h.check_device_error()
    assert keep
