"""The adjoint without outputs: both gradients are optional, and a call that asks
for neither launches nothing and leaves no error, on matrices of short rows, of
long rows and of both, with and without a CSC."""
import numpy as np
import pytest

from conftest import rand_csr
from gpu_util import make_handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("csc", [False, True])
@pytest.mark.parametrize("lens", [np.full(3000, 5), np.full(300, 100), np.r_[np.full(3000, 5), 900]])
@pytest.mark.parametrize("limit", [None, 0, 10, 4000])
def test_no_outputs(torch_cuda, lens, csc, limit):
    torch = torch_cuda
    from spmx import _lib
    A = rand_csr(len(lens), 2500, lens=lens, seed=4)
    h = make_handle(A, torch, csc=csc)
    x, dy = torch.ones(A.n, device="cuda"), torch.ones(A.m, device="cuda")
    before = _lib.lib.spmx_launch_count()
    if limit is None:
        h.spmv_backward(x, dy)
    else:
        h.spmv_backward_auto(x, dy, limit)
    assert _lib.lib.spmx_launch_count() == before
    h.check_device_error()
    # each output alone is what it is beside the other
    dx, dvals = torch.empty(A.n, device="cuda"), torch.empty(A.nnz, device="cuda")
    h.spmv_backward(x, dy, dx)
    h.spmv_backward(x, dy, None, dvals)
    assert np.array_equal(dvals.cpu().numpy(), np.ones(A.nnz, np.float32))
    e = np.zeros(A.n)
    np.add.at(e, A.col, A.val.astype(np.float64))
    mag = np.zeros(A.n)
    np.add.at(mag, A.col, np.abs(A.val.astype(np.float64)))
    assert np.all(np.abs(dx.cpu().numpy() - e) <= 1e-5 * mag)
    h.check_device_error()
