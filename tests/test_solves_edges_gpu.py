"""Wavefront solves and pivot permutations at their block edges."""
import numpy as np
import pytest
from scipy.linalg import lapack

from tests.common import dev, host2d, ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 128, 129, 200, 255, 256, 257, 513, 1000, 1537])
@pytest.mark.parametrize("nrhs", [1, 8, 9, 17, 33])
def test_getrs_potrs(hd, handle, torch_cuda, n, nrhs):
    """FP32 solves on LAPACK's factors: residual within 3 n u |L||U||x| (Higham,
    Theorem 9.4), four times for the block inverses."""
    rng = np.random.default_rng(n + nrhs)
    A = rng.uniform(-1, 1, (n, n)).astype(np.float32)
    A[rng.permutation(n), np.arange(n)] += 2 * n ** 0.5
    B = rng.standard_normal((n, nrhs)).astype(np.float32)
    lu, piv, _ = lapack.sgetrf(A)
    dF, dB = dev(torch_cuda, lu), dev(torch_cuda, B)
    dp = dev(torch_cuda, (piv + 1).astype(np.int32))
    st = hd.call("hdbf_sgetrs", handle.ptr, ptr(dF), n, n, ptr(dp), nrhs, ptr(dB), n)
    torch_cuda.cuda.synchronize()
    assert st == 0 and handle.device_errors() == 0
    X = host2d(dB, n, n, nrhs).astype(np.float64)
    L = np.tril(lu.astype(np.float64), -1) + np.eye(n)
    U = np.triu(lu.astype(np.float64))
    P = np.arange(n)
    for i, p in enumerate(piv):
        P[[i, p]] = P[[p, i]]
    bound = 12 * (n + 2) * 2.0 ** -24 * (np.abs(L) @ (np.abs(U) @ np.abs(X)))
    assert (np.abs(L @ (U @ X) - B[P]) <= bound).all()

    S = np.tril(rng.uniform(-1, 1, (n, n)))
    S = S + S.T + (2 * n ** 0.5 + 1) * np.eye(n)
    c = lapack.spotrf(S.astype(np.float32), lower=1)[0]
    dF, dB = dev(torch_cuda, c), dev(torch_cuda, B)
    st = hd.call("hdbf_spotrs", handle.ptr, ptr(dF), n, n, nrhs, ptr(dB), n)
    torch_cuda.cuda.synchronize()
    assert st == 0
    X = host2d(dB, n, n, nrhs).astype(np.float64)
    L = np.tril(c.astype(np.float64))
    bound = 12 * (n + 2) * 2.0 ** -24 * (np.abs(L) @ (np.abs(L).T @ np.abs(X)))
    assert (np.abs(L @ (L.T @ X) - B) <= bound).all()


def solve_bound(T, x, b, order, block=64):
    """What a block substitution with inverted diagonal blocks may leave of T x - b, T
    triangular and its block rows solved in `order`: each row's products summed and
    subtracted, 66 u |T||x|, then the inverse applied to what is left of b, y, whose own
    residual and products are 131 u |D||D^-1||y|."""
    u, n = 2.0 ** -24, len(T)
    out = np.zeros_like(b)
    done = np.zeros(n, bool)
    for i in order:
        rows = slice(i * block, min(n, (i + 1) * block))
        y = b[rows] - T[rows][:, done] @ x[done]
        D = T[rows, rows]
        out[rows] = (66 * u * (np.abs(T[rows][:, done]) @ np.abs(x[done]) + np.abs(b[rows]))
                     + 131 * u * (np.abs(D) @ (np.abs(np.linalg.inv(D)) @ np.abs(y))))
        done[rows] = True
    return out


@pytest.mark.parametrize("nrhs", [1, 8, 17])
@pytest.mark.parametrize("case", ["lower", "upper", "lower_t"])
def test_block_cancellation(hd, handle, torch_cuda, nrhs, case):
    """A diagonal block with a large inverse behind a coupling that nearly cancels the
    right-hand side: the inverse must meet the difference, not its two terms."""
    n, h = 128, 64
    rng = np.random.default_rng(nrhs)
    ill = np.eye(h) + np.tril(np.full((h, h), -0.15), -1)
    T = np.eye(n)
    tail, head = slice(h, n), slice(0, h)
    T[tail, head] = 1024 * rng.uniform(-1, 1, (h, h))
    if case == "lower_t":  # its transpose couples the first block to the second
        T[head, head] = ill
    else:
        T[tail, tail] = ill
    if case == "upper":
        T = T[::-1, ::-1].copy()
    T = T.astype(np.float32).astype(np.float64)
    x = rng.uniform(0.5, 1, (n, nrhs))
    if case == "lower_t":
        B = (T @ (T.T @ x)).astype(np.float32)
        dF, dB = dev(torch_cuda, T.astype(np.float32)), dev(torch_cuda, B)
        st = hd.call("hdbf_spotrs", handle.ptr, ptr(dF), n, n, nrhs, ptr(dB), n)
    else:
        B = (T @ x).astype(np.float32)
        # packed factors, the other one the identity: a unit diagonal is both's
        dF, dB = dev(torch_cuda, T.astype(np.float32)), dev(torch_cuda, B)
        dp = dev(torch_cuda, np.arange(1, n + 1, dtype=np.int32))
        st = hd.call("hdbf_sgetrs", handle.ptr, ptr(dF), n, n, ptr(dp), nrhs, ptr(dB), n)
    torch_cuda.cuda.synchronize()
    assert st == 0 and handle.device_errors() == 0
    X, Bw = host2d(dB, n, n, nrhs).astype(np.float64), B.astype(np.float64)
    if case == "lower_t":
        z = T.T @ X
        bound = (np.abs(T) @ solve_bound(T.T, X, np.linalg.solve(T, Bw), [1, 0])
                 + solve_bound(T, z, Bw, [0, 1]))
        # z is the first solve's result up to the second one's residual
        assert (np.abs(T @ z - Bw) <= 1.01 * bound).all()
    else:
        bound = solve_bound(T, X, Bw, [0, 1] if case == "lower" else [1, 0])
        assert (np.abs(T @ X - Bw) <= bound).all()
