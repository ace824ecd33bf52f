"""Diagonal-tile Cholesky (64 x 64, one launch) at its panel edges, on failing
tiles and outside the range of its fast pivots."""
import numpy as np
import pytest

from tests.common import dev, host2d, info_tensor, ptr

pytestmark = pytest.mark.gpu


def spd(n, scale=1.0, seed=0):
    rng = np.random.default_rng(seed + n)
    G = rng.uniform(-1, 1, (n, n))
    return ((G @ G.T / n + np.eye(n)) * scale).astype(np.float32)


def factor(torch, hd, handle, A, n):
    d, info = dev(torch, A), info_tensor(torch)
    hd.call("double_blocked_potrf", handle.ptr, ptr(d), n, n, 64, 64, ptr(info))
    torch.cuda.synchronize()
    return host2d(d, n, n, n), int(info.item())


@pytest.mark.parametrize("n", [1, 7, 8, 9, 16, 23, 56, 57, 63, 64, 65, 72, 130])
@pytest.mark.parametrize("scale", [1.0, 1e-36, 1e33])
def test_tile_factor(torch_cuda, hd, handle, n, scale):
    A = spd(n, scale)
    F, info = factor(torch_cuda, hd, handle, A, n)
    assert info == 0
    L = np.tril(F).astype(np.float64)
    # backward error of a Cholesky factor: (n + 1) u |L||L^T|, u = 2^-24, twice
    # for the reciprocal square roots
    bound = 2 * (n + 1) * 2.0 ** -24 * (np.abs(L) @ np.abs(L).T)
    assert (np.abs(np.tril(L @ L.T - A)) <= bound).all()


@pytest.mark.parametrize("col", [0, 1, 7, 8, 9, 31, 40, 63])
@pytest.mark.parametrize("value", [-1.0, 0.0, np.nan])
def test_tile_failure(torch_cuda, hd, handle, col, value):
    n = 96
    A = spd(n)
    A[col, col] = value
    F, info = factor(torch_cuda, hd, handle, A, n)
    assert info == col + 1
    # the leading columns are factored, rows below the tile included
    k = col
    L = np.tril(F)[:, :k].astype(np.float64)
    R = np.tril(L @ L[:k].T - A[:, :k].astype(np.float64))
    bound = 4 * (n + 1) * 2.0 ** -24 * (np.abs(L) @ np.abs(L[:k]).T)
    assert (np.abs(R) <= bound)[~np.isnan(R)].all() and not np.isnan(R[:col]).any()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("half", [32, 16])
@pytest.mark.parametrize("diag", [1.0, 1.7])
def test_inverse_residual(hd, handle, torch_cuda, dtype, half, diag):
    """Inverse of a 64 x 64 tile whose second diagonal block is ill conditioned while the
    inverse below it is not: a column solved by substitution has |L W - I| <= (n + 3) u |L|
    |W| entry by entry (each entry a chain of at most n operations, a reciprocal and a
    multiplication by it), whatever the condition of the blocks.  With B = I the solve
    returns the inverse itself."""
    rng = np.random.default_rng(half)
    n, unit = 64, 2.0 ** -24 if dtype == np.float32 else 2.0 ** -53
    L = np.eye(n) * diag
    for b in range(0, n, 2 * half):
        L11 = np.tril(rng.uniform(-0.5, 0.5, (half, half)), -1) + diag * np.eye(half)
        L22 = np.tril(np.full((half, half), -0.5 * diag), -1) + diag * np.eye(half)
        Y = rng.uniform(-1, 1, (half, half))
        L[b:b + half, b:b + half] = L11
        L[b + half:b + 2 * half, b + half:b + 2 * half] = L22
        L[b + half:b + 2 * half, b:b + half] = -L22 @ Y @ L11
    L = L.astype(dtype)
    dL, dB = dev(torch_cuda, L), dev(torch_cuda, np.eye(n, dtype=dtype))
    name = "trsm_right_lower_transpose" + ("" if dtype == np.float32 else "_double")
    hd.call(name, handle.ptr, n, n, ptr(dL), n, ptr(dB), n)
    torch_cuda.cuda.synchronize()
    handle.check(name)
    W = host2d(dB, n, n, n).T.astype(np.longdouble)
    Lw = L.astype(np.longdouble)
    assert (np.triu(W, 1) == 0).all()
    bound = (n + 3) * unit * (np.abs(Lw) @ np.abs(W))
    assert (np.abs(Lw @ W - np.eye(n)) <= bound).all()


@pytest.mark.parametrize("n", [8, 64, 200, 700])
@pytest.mark.parametrize("k", [50, 55, 61])
def test_scaled_matrix_same_bits(hd, handle, torch_cuda, n, k):
    """4^k A has the factor 2^k L, bit for bit: every operation scales exactly as long as
    nothing overflows (and nothing underflows here), whatever path the pivots take."""
    A = spd(n)
    assert A.max() * 4.0 ** k < 2.0 ** 125

    def run(M):
        d, info = dev(torch_cuda, M), info_tensor(torch_cuda)
        hd.call("double_blocked_potrf", handle.ptr, ptr(d), n, n, 256, 64, ptr(info))
        torch_cuda.cuda.synchronize()
        handle.check()
        assert info.item() == 0
        return np.tril(host2d(d, n, n, n))

    want = run(A) * np.float32(2.0 ** k)
    np.testing.assert_array_equal(run(A * np.float32(4.0 ** k)), want)
