"""The adjoint that chooses on the device: with one nonzero of dy fewer than the
limit, at the limit and above, against the sparse and the dense entry points'
FP64 values, with and without a CSC, and through autograd inside a CUDA graph."""
import numpy as np
import pytest

from conftest import rand_csr
from gpu_util import dev, make_handle
import oracle.oracle as orc

pytestmark = pytest.mark.gpu
RTOL = 1e-5


@pytest.mark.parametrize("csc", [False, True])
@pytest.mark.parametrize("nz", [0, 1, 99, 100, 101, 3000])
@pytest.mark.parametrize("limit", [100, 3001, 0])
def test_auto(torch_cuda, csc, nz, limit):
    torch = torch_cuda
    lens = np.random.default_rng(3).integers(0, 9, 3000)
    lens[77] = 600
    A = rand_csr(3000, 2777, lens=lens, seed=8)
    h = make_handle(A, torch, csc=csc, hola=False)
    rng = np.random.default_rng(nz)
    x = rng.standard_normal(A.n).astype(np.float32)
    dy = np.zeros(A.m, np.float32)
    dy[rng.choice(A.m, nz, replace=False)] = rng.standard_normal(nz)
    row = np.repeat(np.arange(A.m), lens)
    dv64 = dy[row].astype(np.float64) * x[A.col]
    dx64, mag = np.zeros(A.n), np.zeros(A.n)
    np.add.at(dx64, A.col, A.val.astype(np.float64) * dy[row])
    np.add.at(mag, A.col, np.abs(A.val.astype(np.float64) * dy[row]))
    xd, dyd = dev(x, torch), dev(dy, torch)
    buf = torch.full((A.nnz + 1,), 5.0, device="cuda")
    dx = torch.full((A.n,), 5.0, device="cuda")
    for dvals in (buf[:A.nnz], buf[1:], None):
        h.spmv_backward_auto(xd, dyd, limit, dx, dvals)
        assert orc.within_tol(dx.cpu().numpy(), dx64, mag, RTOL)[0]
        if dvals is not None:
            assert np.allclose(dvals.cpu().numpy(), dv64, rtol=2e-7, atol=0)
    h.spmv_backward_auto(xd, dyd, limit, None, buf[1:])
    assert np.allclose(buf[1:].cpu().numpy(), dv64, rtol=2e-7, atol=0)
    h.check_device_error()


def test_autograd_in_a_graph(torch_cuda):
    """The backward no longer reads anything back, so it can be captured, and a
    replay follows dy from one side of the limit to the other."""
    torch = torch_cuda
    from spmx.autograd import SparseMatrix
    A = rand_csr(2000, 2000, lens=np.full(2000, 5), seed=2)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        op = SparseMatrix(A.m, A.n, dev(A.rowptr, torch), dev(A.col, torch))
        vals, dy = dev(A.val, torch).requires_grad_(True), torch.zeros(A.m, device="cuda")
        x = torch.randn(A.n, device="cuda", requires_grad=True)
        torch.autograd.grad(op(vals, x), (vals, x), dy)
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            dvals, dx = torch.autograd.grad(op(vals, x), (vals, x), dy)
        row = np.repeat(np.arange(A.m), 5)
        for nz in (2000, 10, 2000, 0):
            dy.zero_()
            dy[:nz] = 1.5
            g.replay()
            s.synchronize()
            e = dy.cpu().numpy()[row]
            assert np.allclose(dvals.cpu().numpy(), e * x.detach().cpu().numpy()[A.col], rtol=2e-7, atol=0)
            dx64, mag = np.zeros(A.n), np.zeros(A.n)
            np.add.at(dx64, A.col, A.val.astype(np.float64) * e)
            np.add.at(mag, A.col, np.abs(A.val.astype(np.float64) * e))
            assert orc.within_tol(dx.cpu().numpy(), dx64, mag, RTOL)[0]
