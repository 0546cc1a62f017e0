"""One handle fed a second pattern, in the device arrays of the first or in others:
tables that the handle keeps for a matrix (the hubs of the multi-source BFS, the
chunks of Hola and of the adjoint) are those of the matrix it holds now, also where
the second input comes right before a capture."""
import numpy as np
import pytest

from conftest import rand_csr, sym_graph
from gpu_util import dev
import oracle.oracle as orc

pytestmark = pytest.mark.gpu


def _stars(n, hubs, leaves, seed):
    """hubs of `leaves` leaves each (over and under the chunk of 256 edges) and a
    random core, n vertices, as many edges whatever the hubs' numbers"""
    rng = np.random.default_rng(seed)
    edges = {(min(h, v), max(h, v)) for h in hubs for v in rng.permutation(n)[:leaves + 1] if v != h}
    edges = set(sorted(edges)[:len(hubs) * leaves - 100])
    while len(edges) < len(hubs) * leaves + 900:
        a, b = map(int, rng.integers(0, n, 2))
        if a != b:
            edges.add((min(a, b), max(a, b)))
    return sym_graph(n, sorted(edges))


def _check(torch, h, g, srcs, lv, run):
    lv.fill_(-7)
    run()
    torch.cuda.synchronize()
    h.check_device_error()
    got = lv.cpu().numpy().reshape(len(srcs), g.n)
    for s, src in enumerate(srcs):
        assert np.array_equal(got[s], orc.bfs_queue(g.n, g.rowptr, g.col, src)[0]), src


@pytest.mark.parametrize("capture", [False, True])
def test_bfs_hubs_follow_the_pattern(torch_cuda, capture):
    torch = torch_cuda
    from spmx import SpmspvHandle
    n, srcs = 3000, [5, 17, 2900, 0, 640]
    first, second = _stars(n, (0, 1, 2), 900, 1), _stars(n, (7, 1800, 2999), 900, 2)
    assert first.nnz == second.nnz and max(np.diff(first.rowptr)) > 512 and max(np.diff(second.rowptr)) > 512
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        h = SpmspvHandle(n, n, first.nnz)
        rp, cl = dev(first.rowptr, torch), dev(first.col, torch)
        lv = torch.empty(len(srcs) * n, dtype=torch.int32, device="cuda")
        h.InputCSR(first.nnz, rp, cl)
        _check(torch, h, first, srcs, lv, lambda: h.bfs_batched(srcs, lv))
        rp.copy_(dev(second.rowptr, torch))
        cl.copy_(dev(second.col, torch))
        h.InputCSR(second.nnz, rp, cl)
        if capture:
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                h.bfs_batched(srcs, lv, sync=False)
            _check(torch, h, second, srcs, lv, graph.replay)
            _check(torch, h, second, srcs, lv, graph.replay)
        _check(torch, h, second, srcs, lv, lambda: h.bfs_batched(srcs, lv))


NNZ = 24000
PATTERNS = {  # 3,000 rows, 12 chunks of 2,048 nonzeros
    "short": np.full(3000, 8),                                           # every chunk by rows
    "mixed": np.r_[np.full(2000, 7), 5000, np.full(998, 5), 10],         # both kinds, a row over four chunks
    "long": np.r_[np.full(7, 3000), np.zeros(2899, int), np.full(93, 32), 24],  # the scan alone
}


def _hola_check(torch, h, A, x, dy, y, dx, dvals, run):
    for t in (y, dx, dvals):
        t.fill_(5.0)
    run()
    torch.cuda.synchronize()
    h.check_device_error()
    xn, dn = x.cpu().numpy(), dy.cpu().numpy()
    y64, mag = orc.spmv_f64(A.rowptr, A.col, A.val, xn)
    assert orc.within_tol(y.cpu().numpy(), y64, mag, 1e-5)[0]
    e = dn[np.repeat(np.arange(A.m), np.diff(A.rowptr))]
    assert np.allclose(dvals.cpu().numpy(), e.astype(np.float64) * xn[A.col], rtol=2e-7, atol=0)
    dx64, dmag = np.zeros(A.n), np.zeros(A.n)
    np.add.at(dx64, A.col, A.val.astype(np.float64) * e)
    np.add.at(dmag, A.col, np.abs(A.val.astype(np.float64) * e))
    assert orc.within_tol(dx.cpu().numpy(), dx64, dmag, 1e-5)[0]


@pytest.mark.parametrize("how", ["csr", "csr captured", "coo", "same arrays"])
@pytest.mark.parametrize("first,second", [("short", "mixed"), ("mixed", "short"), ("short", "long"), ("long", "short"),
                                          ("long", "mixed")])
def test_hola_tables_follow_the_pattern(torch_cuda, first, second, how):
    torch = torch_cuda
    from spmx import SpmspvHandle
    n = 6000
    mats = [rand_csr(3000, n, lens=PATTERNS[k], seed=i) for i, k in enumerate((first, second))]
    assert all(A.nnz == NNZ for A in mats)
    rng = np.random.default_rng(1)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        x, dy = (dev(rng.uniform(-1, 1, k).astype(np.float32), torch) for k in (n, 3000))
        y, dx, dvals = (torch.empty(k, device="cuda") for k in (3000, n, NNZ))
        h = SpmspvHandle(3000, n, NNZ)

        def run():
            h.holaspmv(1.0, y)
            h.spmv_backward(x, dy, dx, dvals)

        def as_coo(A):
            row = np.repeat(np.arange(3000, dtype=np.int32), np.diff(A.rowptr))
            p = rng.permutation(NNZ)
            return [dev(t[p], torch) for t in (row, A.col, A.val)]

        h.set_x(x)
        if how == "coo":
            h.InputCOO(NNZ, *as_coo(mats[0]))
        else:
            rp, cl, vl = (dev(t, torch) for t in (mats[0].rowptr, mats[0].col, mats[0].val))
            h.InputCSR(NNZ, rp, cl, vl)
        h.holaPreprocess()
        _hola_check(torch, h, mats[0], x, dy, y, dx, dvals, run)
        if how == "coo":
            h.InputCOO(NNZ, *as_coo(mats[1]))
        elif how == "same arrays":
            for t, s in ((rp, mats[1].rowptr), (cl, mats[1].col), (vl, mats[1].val)):
                t.copy_(dev(s, torch))
            h.InputCSR(NNZ, rp, cl, vl)
            h.holaPreprocess()
        else:
            h.InputCSR(NNZ, *(dev(t, torch) for t in (mats[1].rowptr, mats[1].col, mats[1].val)))
        if how == "csr captured":
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                run()
            for _ in range(2):
                _hola_check(torch, h, mats[1], x, dy, y, dx, dvals, graph.replay)
        for _ in range(2):
            _hola_check(torch, h, mats[1], x, dy, y, dx, dvals, run)
