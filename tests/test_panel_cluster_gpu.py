"""Cluster panel kernel at the edges of its row slices, sub-panels and leaf
widths: bit-identical to the grid-wide kernel in FP32, LAPACK's pivots in FP64."""
import numpy as np
import pytest
from scipy.linalg import lapack

from tests.common import dev, host2d, info_tensor, ptr

pytestmark = pytest.mark.gpu


def clear_pivots(n, seed, dtype):
    """U[-1,1) plus one strong entry per column in shuffled rows: pivots that no
    rounding can change."""
    rng = np.random.default_rng(seed)
    A = rng.uniform(-1, 1, (n, n))
    A[rng.permutation(n), np.arange(n)] += 2 * n ** 0.5 * rng.choice([-1, 1], n)
    return A.astype(dtype)


def factor(torch, hd, handle, A, nb, name="double_blocked_getrf"):
    n = A.shape[0]
    d, info = dev(torch, A), info_tensor(torch)
    ipiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    hd.call(name, handle.ptr, ptr(d), n, n, nb, nb, 0, 0, ptr(ipiv), ptr(info))
    torch.cuda.synchronize()
    assert handle.device_errors() == 0
    return d, ipiv.cpu().numpy(), int(info.item())


@pytest.mark.parametrize("n,nb", [(1, 128), (15, 128), (16, 128), (17, 17), (33, 128), (100, 31),
                                  (255, 128), (256, 128), (257, 100), (272, 128), (512, 127),
                                  (513, 128), (1024, 128), (2049, 128), (4097, 128), (8193, 64)])
def test_cluster_bitwise_grid(hd, handle, torch_cuda, n, nb):
    A = clear_pivots(n, n, np.float32)
    out = {}
    for mode in (0, 1):
        handle.set_panel_kernel(mode)
        out[mode] = factor(torch_cuda, hd, handle, A, nb)
    handle.set_panel_kernel(0)
    assert out[0][2] == out[1][2] == 0
    np.testing.assert_array_equal(out[0][1], out[1][1])
    assert torch_cuda.equal(out[0][0], out[1][0])


@pytest.mark.parametrize("n,nb", [(1, 64), (7, 64), (8, 64), (9, 9), (65, 33), (256, 64), (257, 63),
                                  (1000, 64), (2049, 64), (4100, 64)])
def test_cluster_fp64(hd, handle, torch_cuda, n, nb):
    A = clear_pivots(n, n, np.float64)
    d, ipiv, info = factor(torch_cuda, hd, handle, A, nb, "double_blocked_getrf_double")
    lu, piv, _ = lapack.dgetrf(A)
    assert info == 0
    np.testing.assert_array_equal(ipiv - 1, piv)
    F = host2d(d, n, n, n)
    # both are backward stable; the factors of this well-conditioned matrix
    # agree to a small multiple of n u relative to their largest entry
    assert np.abs(F - lu).max() <= 8 * max(n, 16) * 2.0 ** -53 * np.abs(lu).max()


@pytest.mark.parametrize("case", ["zero_column", "subnormal", "ties", "nan"])
def test_cluster_special_values(hd, handle, torch_cuda, case):
    n = 300
    A = clear_pivots(n, 5, np.float32)
    if case == "zero_column":
        A[:, 20] = 0.0
    elif case == "subnormal":
        A[:, 3] = 0.0
        A[100, 3] = 1e-40
    elif case == "ties":
        A[:, 0] = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    else:
        A[40, 30] = np.nan
    out = {}
    for mode in (0, 1):
        handle.set_panel_kernel(mode)
        out[mode] = factor(torch_cuda, hd, handle, A, 128)
    handle.set_panel_kernel(0)
    if case == "nan":  # valid pivots and NaN factors, as the grid-wide kernel gives
        ipiv = out[0][1]
        assert (ipiv >= np.arange(1, n + 1)).all() and (ipiv <= n).all()
        assert torch_cuda.isnan(out[0][0]).any()
        return
    assert out[0][2] == out[1][2] == (21 if case == "zero_column" else 0)
    np.testing.assert_array_equal(out[0][1], out[1][1])
    same = (out[0][0] == out[1][0]) | (torch_cuda.isnan(out[0][0]) & torch_cuda.isnan(out[1][0]))
    assert bool(same.all())


def test_cluster_wait_limit(hd, handle, torch_cuda):
    """With a limit of one poll the cluster's waits may run out; the call then
    reports a timeout, and either way the handle factors correctly afterwards."""
    A = clear_pivots(2048, 1, np.float32)
    d, info = dev(torch_cuda, A), info_tensor(torch_cuda)
    ipiv = torch_cuda.zeros(2048, dtype=torch_cuda.int32, device="cuda")
    try:
        handle.set_wait_limit(1)
        hd.call("double_blocked_getrf", handle.ptr, ptr(d), 2048, 2048, 128, 128, 0, 0, ptr(ipiv),
                ptr(info))
        torch_cuda.cuda.synchronize()
        assert handle.device_errors() in (0, 6)  # 6: timeout
    finally:
        handle.set_wait_limit(0)
    got = factor(torch_cuda, hd, handle, A, 128)
    handle.set_panel_kernel(1)
    want = factor(torch_cuda, hd, handle, A, 128)
    handle.set_panel_kernel(0)
    np.testing.assert_array_equal(got[1], want[1])
    assert torch_cuda.equal(got[0], want[0])
