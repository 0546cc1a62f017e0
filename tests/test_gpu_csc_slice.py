"""The one-launch SpMSpV of a handful of x entries against the FP64 oracle: row
counts around a slice (4,096), x of 1 to 33 entries (32 is its limit), repeated
and unordered keys, a key out of range, an unaligned y, columns whose product
with x_nnz is at the limit of 2,048 and above, and calls chained without a wait."""
import numpy as np
import pytest

from conftest import rand_csr
from gpu_util import dev, make_handle, set_sparse
import oracle.oracle as orc

pytestmark = pytest.mark.gpu
RTOL = 1e-5


@pytest.mark.parametrize("m", [1, 4095, 4096, 4097, 70001])
@pytest.mark.parametrize("k", [1, 2, 31, 32, 33])
def test_slice(torch_cuda, m, k):
    torch = torch_cuda
    rng = np.random.default_rng(m + k)
    lens = rng.integers(0, 3, m) if m < 70001 else (rng.random(m) < 0.05).astype(int)
    lens[-1] = 2
    A = rand_csr(m, 200, lens=lens, seed=m)
    h = make_handle(A, torch, hola=False)
    h.selector_inputs()  # the longest column becomes known
    colptr, row, cval = A.to_csc()
    keys = [np.sort(rng.choice(A.n, k, replace=False)), rng.integers(0, A.n, k)]
    bufs, expect, keep = [], [], []
    for key in keys:
        key = key.astype(np.int32)
        val = rng.uniform(-1, 1, k).astype(np.float32)
        keep.append(set_sparse(h, key, val, torch))
        for off in (0, 1):
            b = torch.full((m + 1,), 4.0, device="cuda")
            h.spmspv_csc(0, 0, -1.5, b[off:off + m], sync=False)
            bufs.append((b, off))
            y64, mag, _ = orc.spmspv_csc_f64(m, colptr, row, cval, key, val, -1.5)
            expect.append((y64, mag))
    for (b, off), (y64, mag) in zip(bufs, expect):
        assert orc.within_tol(b[off:off + m].cpu().numpy(), y64, mag, RTOL)[0]
        assert float(b[m if off == 0 else 0]) == 4.0  # nothing beside y
    h.check_device_error()


@pytest.mark.parametrize("longest", [2048, 2049])
def test_limit_of_products(torch_cuda, longest):
    torch = torch_cuda
    lens = np.zeros(5000, int)
    lens[:longest] = 1
    A = rand_csr(5000, 1, lens=lens, seed=1)
    h = make_handle(A, torch, hola=False)
    h.selector_inputs()
    keep = set_sparse(h, np.zeros(1, np.int32), np.full(1, 2.0, np.float32), torch)
    y = torch.empty(A.m, device="cuda")
    h.spmspv_csc(0, 0, 1.0, y, sync=False)
    e = np.zeros(A.m)
    e[:longest] = 2.0 * A.val
    assert np.allclose(y.cpu().numpy(), e, rtol=1e-6, atol=0) and keep


def test_key_out_of_range(torch_cuda):
    torch = torch_cuda
    from spmx import SpmxError
    A = rand_csr(300, 50, density=0.05, seed=3)
    h = make_handle(A, torch, hola=False)
    h.selector_inputs()
    key, val = np.array([3, 50, 7, -1], np.int32), np.ones(4, np.float32)
    keep = set_sparse(h, key, val, torch)
    y = torch.empty(A.m, device="cuda")
    h.spmspv_csc(0, 0, 1.0, y, sync=False)
    y64, mag, _ = orc.spmspv_csc_f64(A.m, *A.to_csc(), key[[0, 2]], val[:2])
    assert orc.within_tol(y.cpu().numpy(), y64, mag, RTOL)[0] and keep
    with pytest.raises(SpmxError):
        h.check_device_error()
