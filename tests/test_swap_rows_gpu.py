"""Row interchanges on both sides of every line of their launch shapes (swaps per
thread, CTAs per SM, one launch or two), against the swaps one by one."""
import numpy as np
import pytest

from tests.common import dev, host2d, ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [530, 1300, 3000, 6100])
@pytest.mark.parametrize("k", [1, 128, 129, 256, 257, 448, 449, 512, 513])
def test_swaps(hd, torch_cuda, dtype, n, k):
    rng = np.random.default_rng(n + k)
    panel = 7  # the swaps' first row and the panel's first column
    m = n - panel
    piv = np.arange(k) + (rng.random(k) * (m - np.arange(k))).astype(int)
    piv[::5] = rng.permutation(piv)[: len(piv[::5])].clip(np.arange(k)[::5])  # repeated rows
    A = np.arange(n * n, dtype=np.int64).reshape(n, n).astype(dtype)
    # the pivots count from the panel's first row, and come back counting from row 1
    dA, dp = dev(torch_cuda, A), dev(torch_cuda, (piv + 1).astype(np.int32))
    name = "launch_apply_getrf_panel_pivots" + ("" if dtype == np.float32 else "_double")
    hd.call(name, ptr(dA), n, n, panel, k, ptr(dp), torch_cuda.cuda.current_stream().cuda_stream)
    torch_cuda.cuda.synchronize()
    row = np.arange(n)
    for i, p in enumerate(piv):
        row[[panel + i, panel + p]] = row[[panel + p, panel + i]]
    want = A[row]
    want[:, panel:panel + k] = A[:, panel:panel + k]
    np.testing.assert_array_equal(host2d(dA, n, n, n), want)
    np.testing.assert_array_equal(dp.cpu().numpy(), piv + 1 + panel)
