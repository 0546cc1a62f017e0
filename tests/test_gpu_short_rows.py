"""The chunks of short rows of the Hola SpMV and of the CSR adjoint: rows at the
limit (32 nonzeros), rows across chunk ends, empty rows at both ends, matrices
with no long chunk, some, and mostly long ones, ragged last chunks, columns and
values that are not 16-byte aligned; against FP64."""
import numpy as np
import pytest

from conftest import rand_csr
from gpu_util import dev, make_handle
import oracle.oracle as orc

pytestmark = pytest.mark.gpu
RTOL = 1e-5


def _lens(kind):
    rng = np.random.default_rng(11)
    if kind == "limit":        # every row exactly at the limit: all chunks short
        return np.full(200, 32)
    if kind == "five":         # a stencil's rows, a last chunk of a few nonzeros
        return np.full(4100, 5)
    if kind == "ragged":       # 0 to 32, empty rows first and last
        return np.concatenate([np.zeros(700, int), rng.integers(0, 33, 3001), np.zeros(1500, int)])
    if kind == "ones":         # 2,048 rows per chunk
        return np.ones(6145, int)
    if kind == "over":         # one nonzero over the limit in one row: one long chunk
        lens = np.full(1000, 16)
        lens[500] = 33
        return lens
    if kind == "mixed":        # long rows in half of the matrix, one longer than a chunk
        lens = np.concatenate([rng.integers(0, 9, 3000), rng.integers(20, 400, 60)])
        lens[3001] = 5000
        return lens
    lens = rng.integers(0, 40, 2000)  # mostly long chunks: the scan takes the whole matrix
    lens[::20] = 300
    return lens


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("kind", ["limit", "five", "ragged", "ones", "over", "mixed", "mostly-long"])
def test_short_rows(torch_cuda, kind, shift):
    torch = torch_cuda
    from spmx import SpmspvHandle
    lens = _lens(kind)
    A = rand_csr(len(lens), 6000, lens=lens, seed=4)
    h = SpmspvHandle(A.m, A.n, A.nnz)
    # shift: the arrays start 4 bytes past a 16-byte boundary
    rp, cl, vl = dev(A.rowptr, torch), dev(np.r_[np.zeros(shift, np.int32), A.col], torch)[shift:], \
        dev(np.r_[np.zeros(shift, np.float32), A.val], torch)[shift:]
    h.InputCSR(A.nnz, rp, cl, vl)
    rng = np.random.default_rng(5)
    x = rng.standard_normal(A.n).astype(np.float32)
    dy = rng.standard_normal(A.m).astype(np.float32)
    dy[::7] = 0.0
    xd, dyd = dev(x, torch), dev(dy, torch)
    h.set_x(xd)
    y64, mag = orc.spmv_f64(A.rowptr, A.col, A.val, x)
    y = torch.empty(A.m, device="cuda")
    bits = dev(np.packbits(np.r_[(x > 0), np.zeros(-A.n % 32, bool)], bitorder="little").view(np.int32), torch)
    h.set_bitvector(bits, bits.numel())
    g64, gmag = orc.spmv_f64(A.rowptr, A.col, A.val, np.where(x > 0, x, 0).astype(np.float32))
    h.holaPreprocess()
    for _ in range(2):  # the second call finds the counters of split rows as the first left them
        y.fill_(7.0)
        h.holaspmv(1.0, y)
        assert orc.within_tol(y.cpu().numpy(), y64, mag, RTOL)[0]
        h.holaspmspv(1.0, y)
        assert orc.within_tol(y.cpu().numpy(), g64, gmag, RTOL)[0]
    row = np.repeat(np.arange(A.m), lens)
    dv64 = dy[row].astype(np.float64) * x[A.col]
    dx64, dmag = np.zeros(A.n), np.zeros(A.n)
    np.add.at(dx64, A.col, A.val.astype(np.float64) * dy[row])
    np.add.at(dmag, A.col, np.abs(A.val.astype(np.float64) * dy[row]))
    dx, dvals = torch.empty(A.n, device="cuda"), torch.empty(A.nnz + 1, device="cuda")
    for out in (dvals[:A.nnz], dvals[1:]):
        h.spmv_backward(xd, dyd, dx, out)
        assert np.allclose(out.cpu().numpy(), dv64, rtol=2e-7, atol=0)
        assert orc.within_tol(dx.cpu().numpy(), dx64, dmag, RTOL)[0]
    h.spmv_backward(xd, dyd, dx, None)
    assert orc.within_tol(dx.cpu().numpy(), dx64, dmag, RTOL)[0]
    h.spmv_backward(xd, dyd, None, dvals[1:])
    assert np.allclose(dvals[1:].cpu().numpy(), dv64, rtol=2e-7, atol=0)
    h.check_device_error()
