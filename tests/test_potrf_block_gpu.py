"""Diagonal-block Cholesky on one cluster at every tile count and ragged edges, and
failures in any tile."""
import numpy as np
import pytest

from tests.common import dev, host2d, info_tensor, ptr

pytestmark = pytest.mark.gpu


def spd(n, seed=0):
    rng = np.random.default_rng(seed + n)
    G = rng.uniform(-1, 1, (n, n))
    return (G @ G.T / n + np.eye(n)).astype(np.float32)


def factor(torch, hd, handle, A, lda):
    n = A.shape[0]
    buf = np.full((lda, n), np.nan, np.float32)
    buf[:n] = A
    d, info = dev(torch, buf), info_tensor(torch)
    hd.call("double_blocked_potrf", handle.ptr, ptr(d), lda, n, 1024, 1024, ptr(info))
    torch.cuda.synchronize()
    handle.check()
    assert handle.device_errors() == 0
    return host2d(d, lda, n, n), int(info.item())


@pytest.mark.parametrize("n", [65, 127, 128, 129, 191, 193, 256, 257, 320, 385, 449, 511, 512, 577,
                               640, 705, 769, 833, 960, 1023, 1024])
@pytest.mark.parametrize("pad", [0, 1])
def test_block(hd, handle, torch_cuda, n, pad):
    A = spd(n)
    F, info = factor(torch_cuda, hd, handle, A, n + pad)
    assert info == 0
    np.testing.assert_array_equal(np.triu(F, 1), np.triu(A, 1))
    L = np.tril(F).astype(np.float64)
    # (n + 1) u |L||L^T| (Higham, Theorem 10.3), twice for the tile inverses of
    # these well-conditioned blocks
    bound = 2 * (n + 1) * 2.0 ** -24 * (np.abs(L) @ np.abs(L).T)
    assert (np.abs(np.tril(L @ L.T - A)) <= bound).all()


@pytest.mark.parametrize("n,col", [(200, 70), (256, 255), (512, 0), (512, 300), (1000, 640),
                                   (1000, 999)])
def test_block_failure(hd, handle, torch_cuda, n, col):
    A = spd(n)
    A[col, col] = -1.0
    F, info = factor(torch_cuda, hd, handle, A, n)
    assert info == col + 1
    done = col // 64 * 64  # whole tile columns before the failing one
    L = np.tril(F)[:, :done].astype(np.float64)
    bound = 2 * (n + 1) * 2.0 ** -24 * (np.abs(L) @ np.abs(L[:done]).T)
    assert (np.abs(np.tril(L @ L[:done].T - A[:, :done])) <= bound).all()
    again, info = factor(torch_cuda, hd, handle, spd(n, 3), n)  # the handle goes on
    assert info == 0


@pytest.mark.parametrize("n,nb,b,col", [(1000, 512, 256, 100), (700, 1024, 200, 300),
                                        (1100, 512, 1024, 64), (300, 128, 64, 5)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_failure_depends_on_the_matrix_alone(hd, torch_cuda, n, nb, b, col, dtype):
    """What is left behind a failed Cholesky is the same on a new handle and on one that
    has factored something else in between."""
    name = "double_blocked_potrf" + ("" if dtype == np.float32 else "_double")

    def run(h, A):
        d, info = dev(torch_cuda, A.astype(dtype)), info_tensor(torch_cuda)
        hd.call(name, h.ptr, ptr(d), len(A), len(A), nb, b, ptr(info))
        torch_cuda.cuda.synchronize()
        h.check(name)
        return d.cpu().numpy(), int(info.item())

    bad = spd(n)
    bad[col, col] = -1.0
    out = []
    for other in (None, 3.0 * spd(n, 5), 0.1 * spd(n, 6)):
        h = hd.Handle(torch_cuda.cuda.current_stream().cuda_stream)
        if other is not None:
            assert run(h, other)[1] == 0
        out.append(run(h, bad))
        h.close()
    assert all(info == col + 1 for _, info in out)
    np.testing.assert_array_equal(out[1][0], out[0][0])
    np.testing.assert_array_equal(out[2][0], out[0][0])
