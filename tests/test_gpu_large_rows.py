"""The sorted write-back and the bucket method above 8M rows, where few products are
expected and they go through their own kernels (pairs and radix sort; buckets) and
not through dense rows: every work distribution, bucket counts from one to more
than the method takes, every combination of outputs, a row that 20,000 columns
meet, the last row, and a row count that no bucket size divides."""
import numpy as np
import pytest

from gpu_util import make_handle, set_sparse
import oracle.oracle as orc

pytestmark = pytest.mark.gpu

M, N, NNZ, HUB = (1 << 23) + 12345, 200000, 600000, 4000001
OUTPUTS = ["all", "keyval", "y", "key", "val"]


@pytest.fixture(scope="module")
def mat(torch_cuda):
    from spmx.gen import Csr
    # all of x's columns together: 600,000 expected products, fewer than M / 4
    assert N * NNZ < M / 4 * N
    rng = np.random.default_rng(0)
    hub_cols = np.arange(0, N, 10)
    rows = np.r_[np.full(len(hub_cols), HUB), [0, M - 1, M - 1], rng.integers(0, M, NNZ - len(hub_cols) - 3)]
    cols = np.r_[hub_cols, [5, 5, N - 1], rng.integers(0, N, NNZ - len(hub_cols) - 3)]
    key = np.unique(rows * N + cols)
    rows, cols = key // N, (key % N).astype(np.int32)
    rowptr = np.searchsorted(rows, np.arange(M + 1)).astype(np.int32)
    A = Csr(M, N, rowptr, cols, rng.uniform(-1, 1, len(cols)).astype(np.float32))
    return A, A.to_csc(), make_handle(A, torch_cuda, hola=False)


def _case(torch, mat, k, seed):
    A, (colptr, row, cval), h = mat
    rng = np.random.default_rng(seed)
    key = np.sort(np.r_[5, rng.choice(np.delete(np.arange(N), 5), k - 1, replace=False)]).astype(np.int32)
    val = rng.uniform(-1, 1, k).astype(np.float32)
    keep = set_sparse(h, key, val, torch)
    y64, mag, touched = orc.spmspv_csc_f64(M, colptr, row, cval, key, val)
    reached = row[np.repeat(np.isin(np.arange(N), key), np.diff(colptr))]
    # one rounding per product and one per addition
    bound = (np.bincount(reached, minlength=M) + 2) * 2.0 ** -24 * mag
    return h, y64, bound, np.flatnonzero(touched), keep


def _run(torch, run, outputs, y64, bound, rows):
    y = torch.full((M,), 3.0, device="cuda") if outputs in ("all", "y") else None
    yk = torch.full((M,), -1, dtype=torch.int32, device="cuda") if outputs in ("all", "keyval", "key") else None
    yv = torch.full((M,), 9.0, device="cuda") if outputs in ("all", "keyval", "val") else None
    n = run(y, yk, yv)
    assert n == len(rows)
    if y is not None:
        assert np.all(np.abs(y.cpu().numpy() - y64) <= bound)
    if yk is not None:
        assert np.array_equal(yk[:n].cpu().numpy(), rows) and bool((yk[n:] == -1).all())
    if yv is not None:
        assert np.all(np.abs(yv[:n].cpu().numpy() - y64[rows]) <= bound[rows]) and bool((yv[n:] == 9.0).all())


@pytest.mark.parametrize("k", [1, 3, 4097, N])
@pytest.mark.parametrize("variant", [0, 1, 2])
def test_sorted(torch_cuda, mat, variant, k):
    h, y64, bound, rows, keep = _case(torch_cuda, mat, k, k)
    for outputs in ("all", "keyval", "y"):
        _run(torch_cuda, lambda y, yk, yv: h.spmspv_csc(variant, 1, 1.0, y, yk, yv), outputs, y64, bound, rows)
    h.check_device_error()
    assert keep


@pytest.mark.parametrize("k", [1, 4097, N])
@pytest.mark.parametrize("buckets", [0, 1, 1030, 4000, 16384])
def test_buckets(torch_cuda, mat, buckets, k):
    h, y64, bound, rows, keep = _case(torch_cuda, mat, k, k + 1)
    for outputs in OUTPUTS:
        _run(torch_cuda, lambda y, yk, yv: h.CscBasedBucketSpmspv(1.0, y, yk, yv, buckets=buckets), outputs, y64,
             bound, rows)
    h.check_device_error()
    assert keep


def test_more_buckets_than_the_method_takes(torch_cuda, mat):
    from spmx import SpmxError
    h, _, _, _, keep = _case(torch_cuda, mat, 3, 1)
    y = torch_cuda.empty(M, device="cuda")
    with pytest.raises(SpmxError):
        h.CscBasedBucketSpmspv(1.0, y, buckets=40000)
    assert keep
