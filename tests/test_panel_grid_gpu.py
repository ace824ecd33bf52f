"""Grid-wide panel kernel at the edges of its row slices, rows per thread and leaf
widths: bit-identical to the cluster kernel in FP32, LAPACK's pivots in FP64."""
import numpy as np
import pytest
from scipy.linalg import lapack

from tests.common import dev, host2d
from tests.test_panel_cluster_gpu import clear_pivots, factor

pytestmark = pytest.mark.gpu


@pytest.fixture
def grid_handle(hd, monkeypatch):
    def make(rows):
        monkeypatch.setenv("HDBF_PANEL_ROWS", str(rows))
        h = hd.Handle()
        monkeypatch.delenv("HDBF_PANEL_ROWS")
        h.set_panel_kernel(1)
        return h
    return make


# rows per CTA and leaf widths that reach 1, 2, 3 and 6 rows a thread
SHAPES = [(1, 256, 64), (2, 64, 64), (63, 64, 64), (255, 256, 128), (257, 256, 127), (700, 300, 64),
          (1025, 512, 64), (1500, 512, 33), (1537, 768, 64), (1700, 768, 32), (2100, 1100, 32),
          (3100, 1536, 31), (3100, 4096, 16), (3100, 64, 64), (2500, 90, 65)]


@pytest.mark.parametrize("n,rows,nb", SHAPES)
def test_grid_bitwise_cluster(hd, handle, grid_handle, torch_cuda, n, rows, nb):
    A = clear_pivots(n, n, np.float32)
    d, ipiv, info = factor(torch_cuda, hd, grid_handle(rows), A, nb)
    handle.set_panel_kernel(0)
    d2, ipiv2, info2 = factor(torch_cuda, hd, handle, A, nb)
    assert info == info2 == 0
    np.testing.assert_array_equal(ipiv, ipiv2)
    assert torch_cuda.equal(d, d2)


@pytest.mark.parametrize("n,rows,nb", [(n, rows, max(1, nb // 2)) for n, rows, nb in SHAPES])
def test_grid_fp64(hd, grid_handle, torch_cuda, n, rows, nb):
    A = clear_pivots(n, n, np.float64)
    d, ipiv, info = factor(torch_cuda, hd, grid_handle(rows), A, nb, "double_blocked_getrf_double")
    lu, piv, _ = lapack.dgetrf(A)
    assert info == 0
    np.testing.assert_array_equal(ipiv - 1, piv)
    F = host2d(d, n, n, n)
    # as for the cluster kernel: a small multiple of n u of the largest entry
    assert np.abs(F - lu).max() <= 8 * max(n, 16) * 2.0 ** -53 * np.abs(lu).max()
