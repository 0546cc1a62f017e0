"""Two matrices through InputCOO on one handle, whose arrays stay where they are:
the batched SpMSpV, its adjoint, both BFS and the format conversions follow the
second matrix; and values, then a pattern without values, then values again."""
import numpy as np
import pytest

from gpu_util import dev
from test_gpu_reinput import _stars
import oracle.oracle as orc

pytestmark = pytest.mark.gpu
N, NVEC = 3000, 5


def _coo(torch, g, vals, seed):
    row = np.repeat(np.arange(N, dtype=np.int32), np.diff(g.rowptr))
    p = np.random.default_rng(seed).permutation(g.nnz)
    return [dev(row[p], torch), dev(g.col[p], torch)] + ([dev(vals[p], torch)] if vals is not None else [])


def _bfs(torch, h, g):
    srcs = [0, 9, 2999, 1700]
    lv = torch.full((len(srcs) * N,), -7, dtype=torch.int32, device="cuda")
    h.bfs_batched(srcs, lv)
    one = torch.full((N,), -7, dtype=torch.int32, device="cuda")
    h.bfs(9, one)
    expect = [orc.bfs_queue(N, g.rowptr, g.col, s)[0] for s in srcs]
    assert np.array_equal(lv.cpu().numpy().reshape(len(srcs), N), np.array(expect))
    assert np.array_equal(one.cpu().numpy(), expect[1])
    h.check_device_error()


def _products(torch, h, g, vals):
    """forward and backward of a batch, and a sorted product, against 64 bits"""
    rng = np.random.default_rng(7)
    lens = [0, 1, 40, 700, 3000]
    xkey = np.concatenate([np.sort(rng.choice(N, k, replace=False)) for k in lens]).astype(np.int32)
    xval = rng.uniform(-1, 1, len(xkey)).astype(np.float32)
    xptr = np.r_[0, np.cumsum(lens)].astype(np.int32)
    X = np.zeros((N, NVEC))
    for v in range(NVEC):
        X[xkey[xptr[v]:xptr[v + 1]], v] = xval[xptr[v]:xptr[v + 1]]
    D = np.zeros((N, N))
    row = np.repeat(np.arange(N), np.diff(g.rowptr))
    D[row, g.col] = vals
    most = int(np.diff(g.rowptr).max())  # the longest row, and the longest column of this symmetric pattern
    eps = 2.0 ** -24
    xd = [dev(t, torch) for t in (xptr, xkey, xval)]
    Y = torch.full((N, NVEC), 5.0, device="cuda")
    h.spmspv_batched(*xd, 1.0, Y)
    assert np.all(np.abs(Y.cpu().numpy() - D @ X) <= (most + 12) * eps * (np.abs(D) @ np.abs(X)))
    dY = rng.uniform(-1, 1, (N, NVEC)).astype(np.float32)
    dxval = torch.full((len(xkey),), 5.0, device="cuda")
    dvals = torch.full((g.nnz,), 5.0, device="cuda")
    h.spmspv_batched_backward(*xd, 1.0, dev(dY, torch), dxval, dvals)
    vec = np.repeat(np.arange(NVEC), lens)
    assert np.all(np.abs(dxval.cpu().numpy() - (D.T @ dY)[xkey, vec]) <=
                  (most + 12) * eps * (np.abs(D).T @ np.abs(dY))[xkey, vec])
    assert np.all(np.abs(dvals.cpu().numpy() - (dY @ X.T)[row, g.col]) <=
                  (NVEC + 4) * eps * (np.abs(dY) @ np.abs(X).T)[row, g.col])
    h.set_sparse_x(*xd[1:], lens[3] + lens[2])  # entries of two vectors: some keys twice
    x64 = np.zeros(N)
    np.add.at(x64, xkey[:740], xval[:740].astype(np.float64))
    mag = np.zeros(N)
    np.add.at(mag, xkey[:740], np.abs(xval[:740]).astype(np.float64))
    y = torch.full((N,), 5.0, device="cuda")
    h.spmspv_csc(1, 1, 1.0, y)
    assert np.all(np.abs(y.cpu().numpy() - D @ x64) <= 4 * eps * (np.abs(D) @ mag))
    h.check_device_error()


def test_second_matrix(torch_cuda):
    torch = torch_cuda
    from spmx import SpmspvHandle
    graphs = [_stars(N, (0, 1, 2), 900, 1), _stars(N, (7, 1800, 2999), 900, 2)]
    h = SpmspvHandle(N, N, graphs[0].nnz)
    for i in (0, 1, 0):
        g = graphs[i]
        vals = np.random.default_rng(i + 5).uniform(-1, 1, g.nnz).astype(np.float32)
        h.InputCOO(g.nnz, *_coo(torch, g, vals, i))
        h.ToCSC()
        _bfs(torch, h, g)
        _products(torch, h, g, vals)
        rp, cl, vl = (t.cpu().numpy() for t in h.get_csr())
        assert np.array_equal(rp, g.rowptr) and np.array_equal(cl, g.col) and np.array_equal(vl, vals)


def test_values_then_a_pattern(torch_cuda):
    torch = torch_cuda
    from spmx import SpmspvHandle, SpmxError
    graphs = [_stars(N, (0, 1, 2), 900, 1), _stars(N, (7, 1800, 2999), 900, 2)]
    h = SpmspvHandle(N, N, graphs[0].nnz)
    for i, with_values in ((0, True), (1, False), (1, True), (0, False), (1, True)):
        g = graphs[i]
        vals = np.random.default_rng(i).uniform(-1, 1, g.nnz).astype(np.float32) if with_values else None
        h.InputCOO(g.nnz, *_coo(torch, g, vals, i))
        h.ToCSC()
        _bfs(torch, h, g)
        if with_values:
            _products(torch, h, g, vals)
        else:
            h.set_x(torch.ones(N, device="cuda"))
            for run in (lambda: h.naivespmv(1.0, torch.empty(N, device="cuda")),
                        lambda: h.CscBasedNoSortNaiveSpmspv(1.0, torch.empty(N, device="cuda"))):
                with pytest.raises(SpmxError):
                    run()
        rp, cl, vl = (t.cpu().numpy() for t in h.get_csr())
        assert np.array_equal(rp, g.rowptr) and np.array_equal(cl, g.col)
        if with_values:
            assert np.array_equal(vl, vals)
