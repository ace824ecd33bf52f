"""Rounding of the TRSM leaves: the products are summed by themselves before they meet
the right-hand side, FP32 and FP64, right side (Cholesky panels) and left (LU)."""
import numpy as np
import pytest

from tests.common import dev, host2d, info_tensor, ptr

pytestmark = pytest.mark.gpu


def near_identity(n, eps, dtype, rng):
    """Unit lower, off-diagonal entries of at most `eps`."""
    L = np.tril(rng.uniform(-eps, eps, (n, n)), -1).astype(dtype)
    L[np.diag_indices(n)] = 1.0
    return L


def bound(n, eps, unit, want):
    """Per entry: one rounding at the size of x for each of the ceil(n / 64) subtractions
    and for the copy through the inverted diagonal block, in which 63 products of at most
    eps |x| are rounded at no more than the size of x times n eps; the sums themselves
    round at 64 eps |x| a term."""
    tiles = (n + 63) // 64
    small = 64 * 64 * eps * tiles
    return unit * np.abs(want).max() * (tiles + 2 + 2 * small)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,rows", [(64, 500), (65, 100), (128, 33), (256, 1500), (130, 7001),
                                    (700, 300)])
def test_right_side(hd, handle, torch_cuda, dtype, n, rows):
    rng = np.random.default_rng(n + rows)
    unit, eps = (2.0 ** -24, 2.0 ** -16) if dtype == np.float32 else (2.0 ** -53, 2.0 ** -40)
    L = near_identity(n, eps, dtype, rng)
    B = rng.uniform(0.5, 1.0, (rows, n)).astype(dtype)
    dL, dB = dev(torch_cuda, L), dev(torch_cuda, B)
    name = "trsm_right_lower_transpose" + ("" if dtype == np.float32 else "_double")
    hd.call(name, handle.ptr, rows, n, ptr(dL), n, ptr(dB), rows)
    torch_cuda.cuda.synchronize()
    handle.check(name)
    # X = B (I + E^T)^{-1}; the series leaves (n eps)^5 out
    wide = np.float64 if dtype == np.float32 else np.longdouble
    E = np.tril(L, -1).astype(wide)
    X = B.astype(wide)
    for _ in range(4):
        X = B.astype(wide) - X @ E.T
    err = np.abs(host2d(dB, rows, rows, n).astype(wide) - X)
    assert float(err.max()) <= bound(n, eps, unit, X)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,b", [(512, 256), (1000, 200)])
def test_left_side(hd, handle, torch_cuda, dtype, n, b):
    """The rows of U that an LU without pivoting solves for, beside a near-identity panel."""
    rng = np.random.default_rng(n + b)
    unit, eps = (2.0 ** -24, 2.0 ** -16) if dtype == np.float32 else (2.0 ** -53, 2.0 ** -40)
    A = np.tril(rng.uniform(-eps, eps, (n, n)), -1).astype(dtype)
    A[np.diag_indices(n)] = 1.0
    A[:b, b:] = rng.uniform(0.5, 1.0, (b, n - b)).astype(dtype)
    dA, info = dev(torch_cuda, A), info_tensor(torch_cuda)
    name = "blocked_right_looking_getrf_npvt" + ("" if dtype == np.float32 else "_double")
    hd.call(name, handle.ptr, ptr(dA), n, n, b, ptr(info))
    torch_cuda.cuda.synchronize()
    handle.check(name)
    got = host2d(dA, n, n, n)
    wide = np.float64 if dtype == np.float32 else np.longdouble
    E = np.tril(got[:b, :b], -1).astype(wide)
    B = A[:b, b:].astype(wide)
    X = B
    for _ in range(4):
        X = B - E @ X
    err = np.abs(got[:b, b:].astype(wide) - X)
    assert float(err.max()) <= bound(b, eps, unit, X)
