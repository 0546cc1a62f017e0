"""The sorted write-back through dense rows in double: row counts around a
tile of 2,048 rows, columns beyond the cut for long
ones, rows reached with a sum of zero, every combination of outputs, more
products than nonzeros (repeated x keys: refused), and both sides of the row
count above which few products are sorted instead; against the FP64 oracle."""
import numpy as np
import pytest

from conftest import rand_csr
from gpu_util import make_handle, set_sparse
import oracle.oracle as orc

pytestmark = pytest.mark.gpu
RTOL = 1e-5


def _check(torch, A, h, variant, key, val, outputs="all"):
    set_sparse(h, key, val, torch)
    y = torch.full((A.m,), 3.0, device="cuda") if outputs != "keyval" else None
    yk = torch.full((A.m,), -1, dtype=torch.int32, device="cuda") if outputs != "y" else None
    yv = torch.zeros(A.m, device="cuda") if outputs in ("all", "keyval") else None
    n = h.spmspv_csc(variant, 1, 1.5, y, yk, yv)
    h.check_device_error()
    y64, mag, touched = orc.spmspv_csc_f64(A.m, *A.to_csc(), key, val, alpha=1.5)
    rows = np.nonzero(touched)[0]
    assert n == len(rows)
    if y is not None:
        assert orc.within_tol(y.cpu().numpy(), y64, mag, RTOL)[0]
    if yk is not None:
        assert np.array_equal(yk[:n].cpu().numpy(), rows) and (yk[n:] == -1).all()
    if yv is not None:
        assert orc.within_tol(yv[:n].cpu().numpy(), y64[rows], mag[rows], RTOL)[0]


@pytest.mark.parametrize("m", [1, 15, 17, 2047, 2048, 2049, 4097])
@pytest.mark.parametrize("variant,outputs", [(0, "keyval"), (1, "all"), (2, "y"), (2, "key")])
def test_edges(torch_cuda, m, variant, outputs):
    torch = torch_cuda
    A = rand_csr(m, 60, lens=np.arange(m) % 9, seed=m)  # columns of up to 400: long ones too
    if A.nnz == 0:
        A = rand_csr(m, 60, lens=np.full(m, 2), seed=m)
    h = make_handle(A, torch, hola=False)
    rng = np.random.default_rng(m)
    for k in (1, 7, 60):
        key = np.sort(rng.choice(60, k, replace=False)).astype(np.int32)
        _check(torch, A, h, variant, key, rng.uniform(-1, 1, k).astype(np.float32), outputs)


def test_zero_sums_are_listed(torch_cuda):
    torch = torch_cuda
    A = rand_csr(500, 40, lens=np.full(500, 2), seed=1)
    A.val[:] = 1.0
    h = make_handle(A, torch, hola=False)
    key = np.arange(40, dtype=np.int32)
    val = np.where(key % 2, 1.0, -1.0).astype(np.float32)
    val[:4] = [0.0, -0.0, 1e-40, -1e-40]
    _check(torch, A, h, 1, key, val)


@pytest.mark.parametrize("variant", [0, 1, 2])
def test_repeated_keys_beyond_the_nonzeros(torch_cuda, variant):
    torch = torch_cuda
    from spmx import SpmxError
    lens = np.zeros(40, np.int64)
    lens[7] = 3
    A = rand_csr(40, 50, lens=lens, seed=5)
    h = make_handle(A, torch, hola=False)
    y = torch.zeros(A.m, device="cuda")
    set_sparse(h, np.full(4, A.col[0], np.int32), np.ones(4), torch)
    with pytest.raises(SpmxError):
        h.spmspv_csc(variant, 1, 1.0, y)
    _check(torch, A, h, variant, np.full(3, A.col[0], np.int32), np.ones(3, np.float32))
    empty = np.setdiff1d(np.arange(50), A.col).astype(np.int32)
    _check(torch, A, h, variant, empty, np.ones(len(empty), np.float32))


@pytest.mark.parametrize("m", [1 << 23, (1 << 23) + 1])
@pytest.mark.parametrize("k", [3, 64])
@pytest.mark.parametrize("variant", [1, 3])
def test_many_rows(torch_cuda, m, k, variant):
    from spmx.gen import Csr
    torch = torch_cuda
    rng = np.random.default_rng(k)
    nnz = 2_200_000
    rows = np.sort(rng.choice(m, nnz, replace=False))
    rowptr = np.zeros(m + 1, np.int32)
    rowptr[1:] = np.cumsum(np.bincount(rows, minlength=m))
    A = Csr(m, 64, rowptr, rng.integers(0, 64, nnz).astype(np.int32), rng.uniform(-1, 1, nnz).astype(np.float32))
    h = make_handle(A, torch, hola=False)
    key = np.sort(rng.choice(64, k, replace=False)).astype(np.int32)
    _check(torch, A, h, variant, key, rng.uniform(-1, 1, k).astype(np.float32), "keyval")
    _check(torch, A, h, variant, key, rng.uniform(-1, 1, k).astype(np.float32), "all")


@pytest.mark.parametrize("csr", [True, False])
@pytest.mark.parametrize("k", [32768, 32769, 40000])
def test_full_rows(torch_cuda, k, csr):
    """Rows of every column, with and without the row lengths being known: from
    32,769 products of a row on, those of a warp are combined."""
    from gpu_util import dev
    from spmx import SpmspvHandle
    from spmx.gen import Csr
    torch = torch_cuda
    m, n = 300, 40000
    rng = np.random.default_rng(k)
    full = np.zeros((m, n), bool)
    full[[0, 17, 299]] = True
    full[rng.integers(0, m, 2 * n), rng.integers(0, n, 2 * n)] = True
    r, c = np.nonzero(full)
    rowptr = np.r_[0, np.cumsum(full.sum(1))].astype(np.int32)
    A = Csr(m, n, rowptr, c.astype(np.int32), rng.uniform(-1, 1, len(c)).astype(np.float32))
    if csr:
        h = make_handle(A, torch, hola=False)
    else:
        colptr, row, cval = (dev(t, torch) for t in A.to_csc())
        h = SpmspvHandle(m, n, A.nnz)
        h.InputCSC(A.nnz, row, colptr, cval)
    key = np.sort(rng.choice(n, k, replace=False)).astype(np.int32)
    _check(torch, A, h, 2, key, rng.uniform(-1, 1, k).astype(np.float32))
