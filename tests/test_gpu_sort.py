"""The radix sort at the edges of its tiles (1,024, 2,048 and 4,096 items), of the
sizes where the tile changes, and of its digit widths, through COO -> CSR and
CSR -> CSC: bit-exact against a stable host sort."""
import numpy as np
import pytest

from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nnz", [
    (1, 1), (2, 3), (100, 1023), (127, 1024), (129, 1025), (300, 4095), (65535, 4097), (65536, 20000),
    (65537, 303103), (3, 303104), (1 << 20, 303105), (5000, 2424831), (131072, 2424832), (999983, 2424833)])
def test_sorts_at_tile_edges(torch_cuda, n, nnz):
    torch = torch_cuda
    from spmx import SpmspvHandle
    rng = np.random.default_rng(nnz)
    row = rng.integers(0, n, nnz).astype(np.int32)
    col = np.minimum(rng.zipf(1.3, nnz) - 1, n - 1).astype(np.int32)  # long runs of equal digits
    val = rng.standard_normal(nnz).astype(np.float32)
    h = SpmspvHandle(n, n, nnz)
    h.InputCOO(nnz, dev(row, torch), dev(col, torch), dev(val, torch))
    h.ToCSC()
    h.check_device_error()
    by_row = np.lexsort((col, row))
    by_col = by_row[np.argsort(col[by_row], kind="stable")]
    ends = np.arange(n + 1)
    rp, cl, vl = (t.cpu().numpy() for t in h.get_csr())
    assert np.array_equal(rp, np.searchsorted(row[by_row], ends))
    assert np.array_equal(cl, col[by_row]) and np.array_equal(vl, val[by_row])
    rw, cp, cv = (t.cpu().numpy() for t in h.get_csc())
    assert np.array_equal(cp, np.searchsorted(col[by_col], ends))
    assert np.array_equal(rw, row[by_col]) and np.array_equal(cv, val[by_col])
