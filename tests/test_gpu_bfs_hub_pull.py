"""Hubs of the multi-source pull whose chunks outnumber the warps of the grid: a
warp then reads an accumulator that it and others have added to, level after
level.  Bit-exact against one queue BFS per source."""
import numpy as np
import pytest

from gpu_util import make_handle
import oracle.oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("ns", [2, 33, 64])
def test_many_hub_chunks(torch_cuda, ns, layout):
    from spmx.gen import Csr
    torch = torch_cuda
    # 24 hubs adjacent to nearly all of 40,000 vertices: some 3,650 chunks of 256 edges
    # beside 1,256 warps; everything is reached by level 3
    n, hubs = 40000, 24
    rng = np.random.default_rng(ns)
    hub_of = np.repeat(np.arange(hubs), n - hubs)
    leaf = np.tile(np.arange(hubs, n), hubs)
    keep = rng.random(len(leaf)) < 0.97
    a = np.r_[hub_of[keep], rng.integers(hubs, n, 3 * n)]
    b = np.r_[leaf[keep], rng.integers(hubs, n, 3 * n)]
    key = np.unique(np.r_[a * n + b, b * n + a][np.r_[a, b] != np.r_[b, a]])
    rowptr = np.zeros(n + 1, np.int32)
    rowptr[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    g = Csr(n, n, rowptr, (key % n).astype(np.int32), None)
    h = make_handle(g, torch, csc=False, hola=False)
    srcs = rng.integers(0, n, ns).tolist()
    expect = [orc.bfs_queue(n, g.rowptr, g.col, int(s)) for s in srcs]
    for _ in range(3):
        lv = torch.full((ns * n,), -7, dtype=torch.int32, device="cuda")
        depth = h.bfs_batched(srcs, lv, layout=layout)
        h.check_device_error()
        got = lv.cpu().numpy().reshape((ns, n) if layout else (n, ns))
        got = got if layout else got.T
        for s in range(ns):
            assert np.array_equal(got[s], expect[s][0]), s
        assert depth == max(d for _, d in expect)
