"""A dense2sparse of one handle on a stream of its own beside the calls that compact
inside (the sorted write-back, the bucket method, the adjoint that chooses on the
device): neither sees the other's counts."""
import numpy as np
import pytest

from gpu_util import make_handle, set_sparse
import oracle.oracle as orc

pytestmark = pytest.mark.gpu
RTOL = 1e-5


def test_beside_dense2sparse(torch_cuda):
    torch = torch_cuda
    from spmx import gen
    A = gen.zipf_rows(200_000, 1.5, 16, 2000, seed=4)
    h = make_handle(A, torch, hola=False)
    colptr, row, cval = A.to_csc()
    rng = np.random.default_rng(2)
    key = np.sort(rng.choice(A.n, 5000, replace=False)).astype(np.int32)
    val = rng.uniform(-1, 1, len(key)).astype(np.float32)
    y64, mag, touched = orc.spmspv_csc_f64(A.m, colptr, row, cval, key, val)
    rows = np.flatnonzero(touched)
    # 5M entries to host memory: about a millisecond of writes
    size = 5_000_001
    big = torch.rand(size, device="cuda") + 0.5
    big[::3] = 0.0
    want_key = np.flatnonzero(big.cpu().numpy())
    hk, hv = torch.empty(size, dtype=torch.int32).pin_memory(), torch.empty(size).pin_memory()
    hc = torch.zeros(1, dtype=torch.int32).pin_memory()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    h.set_stream(s1)
    keep = set_sparse(h, key, val, torch)
    y = torch.empty(A.m, device="cuda")
    yk, yv = torch.empty(A.m, dtype=torch.int32, device="cuda"), torch.empty(A.m, device="cuda")
    x = torch.linspace(-1, 1, A.n, device="cuda")
    dy = torch.zeros(A.m, device="cuda")
    dy[::50] = 0.5
    dx = torch.empty(A.n, device="cuda")
    e = np.repeat(dy.cpu().numpy(), np.diff(A.rowptr)).astype(np.float64)
    dx64, dmag = np.zeros(A.n), np.zeros(A.n)
    np.add.at(dx64, A.col, A.val * e)
    np.add.at(dmag, A.col, np.abs(A.val * e))
    torch.cuda.synchronize()

    def check_y(n):
        assert n is None or n == len(rows)
        assert np.array_equal(yk[:len(rows)].cpu().numpy(), rows)
        assert orc.within_tol(yv[:len(rows)].cpu().numpy(), y64[rows], mag[rows], RTOL)[0]
        assert orc.within_tol(y.cpu().numpy(), y64, mag, RTOL)[0]

    for rep in range(4):
        for call in ("sorted", "buckets", "adjoint"):
            hk.zero_()
            hc.zero_()
            h.set_stream(s2)
            h.dense2sparse_to_host(size, big, hk, hv, hc)
            h.set_stream(s1)
            n = None
            for _ in range(5):
                if call == "sorted":
                    n = h.spmspv_csc(2, 1, 1.0, y, yk, yv)
                elif call == "buckets":
                    h.spmspv_csc(3, 1, 1.0, y, yk, yv, sync=False)
                else:
                    h.spmv_backward_auto(x, dy, A.m // 20, dx)
            torch.cuda.synchronize()
            h.check_device_error()
            if call == "adjoint":
                assert orc.within_tol(dx.cpu().numpy(), dx64, dmag, RTOL)[0]
            else:
                check_y(n)
            c = int(hc[0])
            assert c == len(want_key) and np.array_equal(hk[:c].numpy(), want_key), (rep, call)
            assert np.array_equal(hv[:c].numpy(), big.cpu().numpy()[want_key])
    assert keep
