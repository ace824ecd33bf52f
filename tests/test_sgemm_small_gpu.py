"""Small-update GEMM (64 x 64 tiles, K shared by a cluster) at the edges of its
tiles, slabs and K ranges, aligned and not, against FP64."""
import numpy as np
import pytest

from tests.common import dev, host2d, ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (3, 65, 31), (64, 64, 32), (65, 63, 33), (130, 70, 127),
                                   (64, 64, 128), (192, 64, 512), (257, 129, 520), (100, 300, 1025),
                                   (2048, 64, 511), (1500, 500, 64)])
@pytest.mark.parametrize("pad", [0, 1, 4])
@pytest.mark.parametrize("lower", [False, True])
def test_small_update(hd, handle, torch_cuda, M, N, K, pad, lower):
    if lower:
        N = M = min(M, 700)
    rng = np.random.default_rng(M * 7 + N * 3 + K)

    def put(rows, cols):
        X = np.full((rows + pad, cols), np.nan, np.float32)
        X[:rows] = rng.uniform(-1, 1, (rows, cols))
        return X

    A, C = put(M, K), put(M, N)
    B = A if lower else put(N, K)
    dA, dB, dC = dev(torch_cuda, A), dev(torch_cuda, B), dev(torch_cuda, C)
    if lower:
        hd.call("syrk_lower_update", handle.ptr, N, K, ptr(dA), M + pad, ptr(dC), M + pad)
    else:
        hd.call("gemm_nt_update", handle.ptr, M, N, K, ptr(dA), M + pad, ptr(dB), N + pad, ptr(dC),
                M + pad)
    torch_cuda.cuda.synchronize()
    handle.check()
    got = host2d(dC, M + pad, M + pad, N)
    a, b = A[:M].astype(np.float64), B[:N].astype(np.float64)
    want = C[:M] - a @ b.T
    if lower:
        up = np.triu_indices(M, 1)
        want[up] = C[:M][up]
    # (K + 2) roundings of 2^-24 on a sum of K products
    bound = (K + 2) * 2.0 ** -24 * (np.abs(a) @ np.abs(b).T + np.abs(C[:M]))
    assert (np.abs(got[:M] - want) <= bound).all()
    assert np.isnan(got[M:]).all()
