"""Repeated x keys whose long columns make more chunks than the queue holds (it is
sized for distinct keys): the chunks beyond it are worked where they are found, in
the dense and in the sorted write-back; against the FP64 oracle."""
import numpy as np
import pytest

from gpu_util import make_handle, set_sparse
import oracle.oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [57, 58, 3000])
def test_more_chunks_than_the_queue(torch_cuda, k):
    from spmx.gen import Csr
    torch = torch_cuda
    # one column of 4,096 nonzeros (32 chunks of 128) among 116,000 in columns of 29:
    # the queue holds nnz / 64 + 1 = 1,877 chunks, 58 copies of the column make 1,856
    m, n, long_len = 6000, 4001, 4096
    rng = np.random.default_rng(k)
    cols = np.r_[np.full(long_len, 7), np.repeat(np.delete(np.arange(n), 7), 29)]
    rows = np.r_[rng.choice(m, long_len, replace=False),
                 (rng.integers(0, m, n - 1)[:, None] + np.arange(29) * 101).ravel() % m]
    order = np.lexsort((cols, rows))
    rowptr = np.zeros(m + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=m), out=rowptr[1:])
    A = Csr(m, n, rowptr, cols[order].astype(np.int32), rng.uniform(-1, 1, len(rows)).astype(np.float32))
    h = make_handle(A, torch, hola=False)
    key = np.full(k, 7, np.int32)
    key[::11] = rng.integers(0, n, len(key[::11]))
    val = rng.uniform(-1, 1, k).astype(np.float32)
    keep = set_sparse(h, key, val, torch)
    y64, mag, _ = orc.spmspv_csc_f64(m, *A.to_csc(), key, val)
    y = torch.full((m,), 3.0, device="cuda")
    for variant in (1, 2):
        h.spmspv_csc(variant, 0, 1.0, y)
        # every product is rounded once, every addition once: k + 29 of them at most per row
        assert np.all(np.abs(y.cpu().numpy() - y64) <= (k + 30) * 2.0 ** -24 * mag)
    h.check_device_error()
    assert keep
