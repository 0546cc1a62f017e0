"""A matrix without rows: where the sparse adjoint is asked for, the gradients are
zeros, from the entry points and through autograd."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 300])
def test_no_rows(torch_cuda, n):
    torch = torch_cuda
    from spmx.autograd import SparseMatrix
    rowptr = torch.zeros(1, dtype=torch.int32, device="cuda")
    op = SparseMatrix(0, n, rowptr, torch.zeros(0, dtype=torch.int32, device="cuda"), sparse_grad="sparse")
    vals = torch.zeros(0, device="cuda", requires_grad=True)
    x = torch.ones(n, device="cuda", requires_grad=True)
    if n:
        y = op(vals, x)
        dvals, dx = torch.autograd.grad(y, (vals, x), torch.zeros(0, device="cuda"))
        assert y.shape == (0,) and dvals.shape == (0,)
        assert dx.shape == (n,) and not dx.any()
    dx = torch.full((n,), 5.0, device="cuda")
    op.h.spmv_backward_auto(x.detach(), torch.zeros(0, device="cuda"), 1, dx)
    assert not dx.any()
    op.h.check_device_error()
