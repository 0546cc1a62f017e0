"""The load-balanced CSC SpMSpV with dense y: columns around the cut (128) and
the chunk of long columns, x sizes around the entries per warp (148 SMs x 64
warps per power of two), repeated and unordered keys, an unaligned y; against
the FP64 oracle, with the bin count it leaves behind."""
import numpy as np
import pytest

from gpu_util import dev, make_handle, set_sparse
import oracle.oracle as orc

pytestmark = pytest.mark.gpu
RTOL = 1e-5


def _matrix(n):
    from spmx.gen import Csr
    rng = np.random.default_rng(n)
    lens = rng.integers(0, 7, n)
    lens[:9] = (0, 1, 127, 128, 129, 255, 256, 257, 4000)
    m = 5003
    rows = np.concatenate([rng.choice(m, k, replace=False) for k in lens])
    cols = np.repeat(np.arange(n), lens)
    order = np.lexsort((cols, rows))
    rowptr = np.zeros(m + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=m), out=rowptr[1:])
    return Csr(m, n, rowptr, cols[order].astype(np.int32), rng.uniform(-1, 1, len(rows)).astype(np.float32))


@pytest.fixture(scope="module")
def mat():
    return _matrix(40000)


@pytest.mark.parametrize("k", [1, 9, 31, 9471, 9472, 9473, 18945, 37889, 40000])
@pytest.mark.parametrize("order", ["sorted", "reversed", "repeated"])
def test_flat(torch_cuda, mat, k, order):
    torch = torch_cuda
    h = make_handle(mat, torch, hola=False)
    rng = np.random.default_rng(k)
    key = np.concatenate([np.arange(min(k, 9)), 9 + rng.choice(mat.n - 9, max(k - 9, 0), replace=False)])
    key = np.sort(key)[:: -1 if order == "reversed" else 1]
    if order == "repeated":
        key[k // 2:] = key[: k - k // 2]
    key = np.ascontiguousarray(key, np.int32)
    val = rng.uniform(-1, 1, k).astype(np.float32)
    set_x = set_sparse(h, key, val, torch)
    buf = torch.full((mat.m + 1,), 7.0, device="cuda")
    colptr, row, cval = mat.to_csc()
    y64, mag, _ = orc.spmspv_csc_f64(mat.m, colptr, row, cval, key, val)
    for y in (buf[:mat.m], buf[1:]):  # 16-byte aligned and not
        for variant in (1, 2):
            h.spmspv_csc(variant, 0, 1.0, y, sync=False)
            assert orc.within_tol(y.cpu().numpy(), y64, mag, RTOL)[0], (variant, order)
    h.check_device_error()
    del set_x


def test_longest_column_follows_the_matrix(torch_cuda, mat):
    """The kernel for long columns is left out where the selector knows that
    there are none; a new matrix on the handle has to be looked at again."""
    torch = torch_cuda
    colptr, row, cval = mat.to_csc()
    short = np.flatnonzero(np.diff(colptr) <= 128)
    h = make_handle(mat, torch, hola=False)
    lens = np.diff(colptr)[short]
    # the same number of nonzeros in columns of at most 4
    flat = np.arange(mat.nnz)
    c0 = np.minimum(np.arange(mat.n + 1) * 4, mat.nnz).astype(np.int32)
    c0[-1] = mat.nnz
    if c0[-1] - c0[-2] > 128:
        pytest.skip("matrix too dense for columns of 4")
    r0 = (flat % mat.m).astype(np.int32)
    short_csc = [dev(a, torch) for a in (r0, c0, cval)]
    h.InputCSC(mat.nnz, *short_csc)
    key, val = np.arange(12, dtype=np.int32), np.ones(12, np.float32)
    keep = set_sparse(h, key, val, torch)
    y = torch.empty(mat.m, device="cuda")
    h.selector_inputs()  # the longest column becomes known: 4
    h.spmspv_csc(1, 0, 1.0, y, sync=False)
    y64, mag, _ = orc.spmspv_csc_f64(mat.m, c0, r0, cval, key, val)
    assert orc.within_tol(y.cpu().numpy(), y64, mag, RTOL)[0]
    h.ToCSC()  # columns of up to 4,000 again
    h.spmspv_csc(1, 0, 1.0, y, sync=False)
    y64, mag, _ = orc.spmspv_csc_f64(mat.m, colptr, row, cval, key, val)
    assert orc.within_tol(y.cpu().numpy(), y64, mag, RTOL)[0]
    assert len(lens) and keep
