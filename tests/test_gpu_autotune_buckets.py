"""The tuner leaves the bucket count alone where the bucket method goes through
dense rows and ignores it, and times it where the bucket kernels run."""
import numpy as np
import pytest

from conftest import rand_csr
from gpu_util import make_handle

pytestmark = pytest.mark.gpu


def _buckets(h, path):
    h.autotune(path)
    return int(open(path).read().split()[8])


@pytest.mark.parametrize("m,n", [(500, 700), (20000, 15000), (3000, 3000), (60000, 2000), (1000, 50000), (9000, 9000)])
def test_left_alone(torch_cuda, tmp_path, m, n):
    A = rand_csr(m, n, lens=np.random.default_rng(m).integers(0, 9, m), seed=n)
    assert _buckets(make_handle(A, torch_cuda, hola=False), str(tmp_path / "tune.txt")) == 256


def test_timed_above_the_row_scan(torch_cuda, tmp_path):
    from spmx.gen import Csr
    m, nnz = (1 << 23) + 5, 300000
    rng = np.random.default_rng(2)
    rows = np.sort(rng.choice(m, nnz, replace=False))
    rowptr = np.searchsorted(rows, np.arange(m + 1)).astype(np.int32)
    A = Csr(m, 5000, rowptr, rng.integers(0, 5000, nnz).astype(np.int32), np.ones(nnz, np.float32))
    h = make_handle(A, torch_cuda, hola=False)
    assert _buckets(h, str(tmp_path / "tune.txt")) in (64, 256, 1024)
    h.check_device_error()
