"""One handle fed a second pattern through the device arrays of the first: tables
that the handle keeps for a matrix (the hubs of the multi-source BFS) are those of
the matrix it holds now, also where the second input comes right before a capture."""
import numpy as np
import pytest

from conftest import sym_graph
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
