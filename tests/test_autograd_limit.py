"""The count of dy's nonzeros below which autograd takes the sparse adjoint says
what `count < threshold * m` says, for every threshold that can be compared."""
import math

import pytest


@pytest.mark.parametrize("threshold", [0.05, 0.0, -0.0, -1.0, 1.0, 1.0 + 1e-12, 2.0, 1e-9, 0.3, 1, 0, 1e300,
                                       float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("m", [0, 1, 2, 3, 10, 20, 1000])
def test_limit(threshold, m):
    from spmx.autograd import _sparse_limit
    limit = _sparse_limit("auto", threshold, m)
    assert isinstance(limit, int) and 0 <= limit <= m + 1
    for count in range(m + 1):
        assert (count < limit) == (count < threshold * m), count
    assert _sparse_limit("sparse", threshold, m) == m + 1
    assert not math.isnan(limit)


@pytest.mark.gpu
@pytest.mark.parametrize("threshold", [float("inf"), float("nan"), float("-inf"), 0.05])
@pytest.mark.parametrize("nz", [0, 7, 400])
def test_backward(torch_cuda, threshold, nz):
    import numpy as np
    from conftest import rand_csr
    from gpu_util import dev
    from spmx.autograd import SparseMatrix
    torch = torch_cuda
    A = rand_csr(400, 300, lens=np.full(400, 4), seed=1)
    op = SparseMatrix(A.m, A.n, dev(A.rowptr, torch), dev(A.col, torch), sparse_threshold=threshold)
    vals = dev(A.val, torch).requires_grad_(True)
    x = torch.linspace(-1, 1, A.n, device="cuda").requires_grad_(True)
    dy = torch.zeros(A.m, device="cuda")
    dy[:nz] = 0.5
    dvals, dx = torch.autograd.grad(op(vals, x), (vals, x), dy)
    e = dy.cpu().numpy()[np.repeat(np.arange(A.m), 4)]
    assert np.allclose(dvals.cpu().numpy(), e * x.detach().cpu().numpy()[A.col], rtol=2e-7, atol=0)
    dx64, mag = np.zeros(A.n), np.zeros(A.n)
    np.add.at(dx64, A.col, A.val.astype(np.float64) * e)
    np.add.at(mag, A.col, np.abs(A.val.astype(np.float64) * e))
    assert np.all(np.abs(dx.cpu().numpy() - dx64) <= 1e-5 * mag)
