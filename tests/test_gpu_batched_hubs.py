"""Batched SpMSpV rows around the hub limit (384 nonzeros), which whole CTAs
take: 384, 385 and more rows above it than there are CTAs, with vector counts
that are and are not multiples of 4 and above 256, fewer and more batch entries
than columns; against FP64."""
import numpy as np
import pytest

from conftest import rand_csr
from gpu_util import dev, make_handle
import oracle.oracle as orc

pytestmark = pytest.mark.gpu
RTOL = 1e-5


@pytest.mark.parametrize("nvec", [1, 6, 64, 260])
@pytest.mark.parametrize("hubs", [0, 3, 900])
@pytest.mark.parametrize("options", [0, 3])
def test_hub_rows(torch_cuda, nvec, hubs, options):
    torch = torch_cuda
    rng = np.random.default_rng(nvec + hubs)
    lens = rng.integers(0, 12, 1500)
    lens[100:105] = (511, 512, 40, 384, 385)
    lens[200:200 + hubs] = 513 + rng.integers(0, 60, hubs)
    A = rand_csr(1500, 1600, lens=lens, seed=6)
    h = make_handle(A, torch, hola=False)
    h.set_batch_options(options)
    size = rng.integers(1, 90, nvec)
    xptr = np.r_[0, np.cumsum(size)].astype(np.int32)
    xkey = np.concatenate([np.sort(rng.choice(A.n, k, replace=False)) for k in size]).astype(np.int32)
    xval = rng.standard_normal(len(xkey)).astype(np.float32)
    vec = np.repeat(np.arange(nvec), size)
    xp, xk, xv = (dev(a, torch) for a in (xptr, xkey, xval))
    dY = rng.standard_normal((A.m, nvec)).astype(np.float32)
    Y = torch.full((A.m, nvec), 9.0, device="cuda")
    dxval, dvals = torch.full((len(xkey),), 9.0, device="cuda"), torch.full((A.nnz,), 9.0, device="cuda")
    for _ in range(2):
        h.spmspv_batched(xp, xk, xv, 0.5, Y)
        h.spmspv_batched_backward(xp, xk, xv, 0.5, dev(dY, torch), dxval, dvals)
    h.check_device_error()
    X = np.zeros((A.n, nvec))
    X[xkey, vec] = xval
    row = np.repeat(np.arange(A.m), lens)
    a64 = A.val.astype(np.float64)
    D = np.zeros((A.m, A.n))
    D[row, A.col] = a64
    assert orc.within_tol(Y.cpu().numpy().ravel(), 0.5 * (D @ X).ravel(), 0.5 * (abs(D) @ abs(X)).ravel(), RTOL)[0]
    e = 0.5 * np.einsum("kv,kv->k", X[A.col], dY[row].astype(np.float64))
    mag = 0.5 * np.einsum("kv,kv->k", abs(X[A.col]), abs(dY[row]).astype(np.float64))
    assert orc.within_tol(dvals.cpu().numpy(), e, mag, RTOL)[0]
    g, gm = 0.5 * (D.T @ dY)[xkey, vec], 0.5 * (abs(D.T) @ abs(dY))[xkey, vec]
    assert orc.within_tol(dxval.cpu().numpy(), g, gm, RTOL)[0]


@pytest.mark.parametrize("m", [130_000, 131_073, 200_001])
def test_row_chunk_sizes(torch_cuda, m):
    """Row chunks between the smallest (128) and the largest weight: row counts
    on both sides of the first size above 128 (a row weighs its nonzeros + 32)."""
    torch = torch_cuda
    lens = np.random.default_rng(m).integers(0, 3, m)
    rowptr = np.r_[0, np.cumsum(lens)].astype(np.int32)
    from spmx.gen import Csr
    rng = np.random.default_rng(7)
    A = Csr(m, 50, rowptr, rng.integers(0, 50, rowptr[-1]).astype(np.int32),
            rng.standard_normal(rowptr[-1]).astype(np.float32))
    h = make_handle(A, torch, csc=False, hola=False)
    nvec = 3
    X = rng.standard_normal((50, nvec)).astype(np.float32)
    xptr = np.arange(nvec + 1, dtype=np.int32) * 50
    xkey, xval = np.tile(np.arange(50, dtype=np.int32), nvec), np.ascontiguousarray(X.T).ravel()
    xp, xk, xv = (dev(a, torch) for a in (xptr, xkey, xval))
    dY = rng.standard_normal((m, nvec)).astype(np.float32)
    Y, dvals = torch.full((m, nvec), 9.0, device="cuda"), torch.full((A.nnz,), 9.0, device="cuda")
    h.spmspv_batched(xp, xk, xv, 1.0, Y)
    h.spmspv_batched_backward(xp, xk, xv, 1.0, dev(dY, torch), None, dvals)
    h.check_device_error()
    row = np.repeat(np.arange(m), lens)
    prod = A.val[:, None].astype(np.float64) * X[A.col]
    want, mag = np.zeros((m, nvec)), np.zeros((m, nvec))
    np.add.at(want, row, prod)
    np.add.at(mag, row, np.abs(prod))
    assert orc.within_tol(Y.cpu().numpy(), want, mag, RTOL)[0]
    each = dY[row].astype(np.float64) * X[A.col]
    assert orc.within_tol(dvals.cpu().numpy(), each.sum(1), np.abs(each).sum(1), RTOL)[0]
