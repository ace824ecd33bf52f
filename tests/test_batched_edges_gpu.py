"""Batched factor-and-solve at the edges of its panels, sub-panels and row blocks,
every launch shape: backward error of the factors and solutions, LAPACK's pivots,
and what it leaves on failure."""
import numpy as np
import pytest
from scipy.linalg import lapack

from hygondoubleblockedfactorizations_b200.batch import DeviceBatch

pytestmark = pytest.mark.gpu

NS_CHOL = [1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 40, 63, 64, 65, 97, 129, 160, 161, 257, 500, 512]
NS_LU = NS_CHOL[:-2] + [385, 513, 767, 768]


def fill(torch, b, seed):
    """Well-conditioned SPD systems, and general ones whose pivots are clear."""
    rng = np.random.default_rng(seed)
    A, r = [], []
    for op, n in zip(b.ops, b.ns):
        n = int(n)
        M = rng.uniform(-1, 1, (n, n))
        if op == 0:
            M = np.tril(M) + np.tril(M, -1).T + (1.5 * n ** 0.5 + 1) * np.eye(n)
        else:
            M[rng.permutation(n), np.arange(n)] += 2 * n ** 0.5 * rng.choice([-1, 1], n)
        A.append(M.astype(np.float32))
        r.append(rng.standard_normal(n).astype(np.float32))
    b.A.copy_(torch.from_numpy(np.concatenate([M.ravel(order="F") for M in A])))
    b.b.copy_(torch.from_numpy(np.concatenate(r)))
    return A, r


@pytest.mark.parametrize("variant", range(6))
def test_orders(hd, handle, torch_cuda, variant):
    ops = np.array([0] * len(NS_CHOL) + [1] * len(NS_LU), np.int32)
    b = DeviceBatch(torch_cuda, ops, np.array(NS_CHOL + NS_LU, np.int32))
    A, rhs = fill(torch_cuda, b, 11)
    assert b.run(handle, variant) == 0
    torch_cuda.cuda.synchronize()
    assert not b.info.cpu().numpy().any()
    for i, (op, n) in enumerate(zip(ops, b.ns)):
        n = int(n)
        F = b.matrix(i).cpu().numpy().astype(np.float64)
        x = b.rhs(i).cpu().numpy().astype(np.float64)
        M = A[i].astype(np.float64)
        u = 2.0 ** -24
        if op == 0:
            L = np.tril(F)
            np.testing.assert_array_equal(np.triu(F, 1), np.triu(M, 1))
            E, bound = np.tril(L @ L.T - M), np.abs(L) @ np.abs(L).T
            W = bound
        else:
            L, U = np.tril(F, -1) + np.eye(n), np.triu(F)
            piv = b.pivots(i).cpu().numpy() - 1
            np.testing.assert_array_equal(piv, lapack.sgetrf(A[i])[1])
            P = np.arange(n)
            for j, p in enumerate(piv):
                P[[j, p]] = P[[p, j]]
            E, bound = L @ U - M[P], np.abs(L) @ np.abs(U)
            W = np.empty_like(bound)
            W[P] = bound
        # Higham, Theorems 10.3 and 9.3: n u |L||L^T|, n u |L||U|; twice for the
        # reciprocals in place of divisions
        assert (np.abs(E) <= 2 * (n + 2) * u * bound).all(), (i, n)
        # and the solves (Theorem 9.4 and its Cholesky twin): 3 n u |L||U||x|
        res = np.abs(M @ x - rhs[i])
        assert (res <= 4 * (3 * n + 3) * u * (W @ np.abs(x)) + 1e-30).all(), (i, n)


@pytest.mark.parametrize("variant", [0, 2, 5])
def test_failures(hd, handle, torch_cuda, variant):
    """A failing Cholesky reports its column, factors the ones before it and keeps
    its right-hand side; a singular LU reports its first zero pivot."""
    ops = np.array([0, 0, 0, 1, 0], np.int32)
    ns = np.array([70, 200, 50, 60, 48], np.int32)
    b = DeviceBatch(torch_cuda, ops, ns)
    A, rhs = fill(torch_cuda, b, 5)
    for i, col, val in ((0, 37, -1.0), (1, 64, 0.0), (2, 9, np.nan)):
        A[i][col, col] = val
    A[3][:, 20] = 0.0
    A[4] *= np.float32(1e-34)  # pivots outside the fast range
    b.A.copy_(torch_cuda.from_numpy(np.concatenate([M.ravel(order="F") for M in A])))
    assert b.run(handle, variant) == 0
    torch_cuda.cuda.synchronize()
    assert b.info.cpu().numpy().tolist() == [38, 65, 10, 21, 0]
    for i, col in ((0, 37), (1, 64), (2, 9)):
        np.testing.assert_array_equal(b.rhs(i).cpu().numpy(), rhs[i])
        L = np.tril(b.matrix(i).cpu().numpy())[:, :col].astype(np.float64)
        E = np.abs(L[:col] @ L[:col].T - A[i][:col, :col].astype(np.float64))
        bound = 2 * (ns[i] + 2) * 2.0 ** -24 * (np.abs(L[:col]) @ np.abs(L[:col]).T)
        assert (np.tril(E) <= bound).all()
    L = np.tril(b.matrix(4).cpu().numpy()).astype(np.float64)
    bound = 2 * (48 + 2) * 2.0 ** -24 * (np.abs(L) @ np.abs(L).T)
    assert (np.abs(np.tril(L @ L.T - A[4].astype(np.float64))) <= bound).all()


@pytest.mark.parametrize("variant", range(6))
def test_lu_nan_pivots(hd, handle, torch_cuda, variant):
    """The first maximum as reference LAPACK's ISAMAX finds it: a NaN on the diagonal is
    never beaten, a NaN below it never chosen."""
    where = [(0, 0), (5, 0), (40, 30), (30, 30), (99, 99), (17, 16)]
    n = 100
    b = DeviceBatch(torch_cuda, np.ones(len(where), np.int32), np.full(len(where), n, np.int32))
    A, _ = fill(torch_cuda, b, 7)
    for i, (r, c) in enumerate(where):
        # strong entries on the diagonal: without the NaN no row moves
        A[i] = (np.random.default_rng(i).uniform(-1, 1, (n, n)) + 4 * n * np.eye(n)).astype(
            np.float32)
        A[i][r, c] = np.nan
    b.A.copy_(torch_cuda.from_numpy(np.concatenate([M.ravel(order="F") for M in A])))
    assert b.run(handle, variant) == 0
    torch_cuda.cuda.synchronize()
    for i, (r, c) in enumerate(where):
        M = A[i].astype(np.float64)
        piv = []
        with np.errstate(invalid="ignore"):
            for j in range(n):
                p = j
                for q in range(j + 1, n):
                    if abs(M[q, j]) > abs(M[p, j]):
                        p = q
                piv.append(p)
                M[[j, p]] = M[[p, j]]
                M[j + 1:, j] /= M[j, j]
                M[j + 1:, j + 1:] -= np.outer(M[j + 1:, j], M[j, j + 1:])
        np.testing.assert_array_equal(b.pivots(i).cpu().numpy() - 1, piv)


@pytest.mark.parametrize("op", [0, 1])
@pytest.mark.parametrize("variant", range(6))
def test_solve_divides(hd, handle, torch_cuda, op, variant):
    """Diagonal systems over the whole range of exponents, subnormal pivots among them:
    the solution is the division's, exact here (b = d times a small integer, zero among
    them; Cholesky: d a power of four)."""
    n = 70
    b = DeviceBatch(torch_cuda, np.full(2, op, np.int32), np.full(2, n, np.int32))
    k = np.arange(n)
    d = np.float32(2.0) ** np.where(op, -148 + 4 * k, 2 * (-73 + 2 * k)).astype(np.float64)
    d = d[d < 2.0 ** 120][np.arange(n) % (d < 2.0 ** 120).sum()].astype(np.float32)
    assert (d > 0).all() and (d < 2.0 ** -126).any()
    x = (k % 5).astype(np.float32)
    want = np.concatenate([x, x])
    b.A.copy_(torch_cuda.from_numpy(np.concatenate([np.diag(d).ravel()] * 2)))
    b.b.copy_(torch_cuda.from_numpy(np.concatenate([d * x] * 2)))
    assert b.run(handle, variant) == 0
    torch_cuda.cuda.synchronize()
    assert not b.info.cpu().numpy().any()
    np.testing.assert_array_equal(b.b.cpu().numpy(), want)
