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
