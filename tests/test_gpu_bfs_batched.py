"""The multi-source BFS at the edges of its level planes (levels 15, 16 and 17),
of its hub chunks (256 edges), of the 32- and 64-bit source words and of both
layouts: bit-exact against one queue BFS per source."""
import numpy as np
import pytest

from conftest import sym_graph
from gpu_util import make_handle
import oracle.oracle as orc

pytestmark = pytest.mark.gpu


def _graph(kind):
    if kind == "path15":    # deepest level 15: the last that the planes hold
        return sym_graph(16, [(i, i + 1) for i in range(15)])
    if kind == "path16":
        return sym_graph(17, [(i, i + 1) for i in range(16)])
    if kind == "hubs":      # degrees 255..513 around the chunk, a tail of 40 levels, isolated vertices
        edges, at = [], 4
        for hub, leaves in enumerate((255, 256, 257, 513)):
            edges += [(hub, at + i) for i in range(leaves)]
            edges += [(hub, (hub + 1) % 4)] if hub < 3 else []
            at += leaves
        edges += [(at + i, at + i + 1) for i in range(40)] + [(3, at)]
        return sym_graph(at + 46, edges)
    rng = np.random.default_rng(5)  # a dense core that several sources reach at once
    e = rng.integers(0, 701, (9000, 2))
    return sym_graph(701, [tuple(map(int, p)) for p in e if p[0] != p[1]])


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("kind,ns", [("path15", 3), ("path16", 2), ("hubs", 1), ("hubs", 31), ("hubs", 33),
                                     ("hubs", 64), ("core", 32), ("core", 63), ("core", 64)])
def test_levels(torch_cuda, kind, ns, layout):
    torch = torch_cuda
    g = _graph(kind)
    h = make_handle(g, torch, csc=False, hola=False)
    srcs = [0] + np.random.default_rng(ns).integers(0, g.n, ns - 1).tolist()
    for _ in range(2):  # the second run starts from what the first left behind
        lv = torch.full((ns * g.n,), -7, dtype=torch.int32, device="cuda")
        depth = h.bfs_batched(srcs, lv, layout=layout)
        h.check_device_error()
        got = lv.cpu().numpy().reshape((ns, g.n) if layout else (g.n, ns))
        got = got if layout else got.T
        deepest = 0
        for s, src in enumerate(srcs):
            e, ed = orc.bfs_queue(g.n, g.rowptr, g.col, int(src))
            assert np.array_equal(got[s], e), (s, src)
            deepest = max(deepest, ed)
        assert depth == deepest
