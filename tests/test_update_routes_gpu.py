"""Updates on both sides of the lines between the small-update kernel and the larger
tiles, FP32 and FP64, whole and lower triangle: whole-number operands, so that every
kernel has to give the same exact result."""
import os

import numpy as np
import pytest

from tests.common import dev, host2d, ptr

pytestmark = pytest.mark.gpu


@pytest.fixture()
def plain(hd, torch_cuda):
    """A handle whose FP32 updates stay off the tensor cores, with and without an arena."""
    os.environ["HDBF_TC_SGEMM"] = "0"
    try:
        h = hd.Handle(torch_cuda.cuda.current_stream().cuda_stream)
    finally:
        del os.environ["HDBF_TC_SGEMM"]
    yield h
    torch_cuda.cuda.synchronize()
    h.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("reserve", [False, True])
@pytest.mark.parametrize("M,N,K", [(1500, 520, 300), (1500, 520, 40), (1537, 1530, 33), (2049, 1000, 64),
                                   (2048, 384, 2049), (769, 385, 2050), (100, 70, 1030),
                                   (4097, 190, 130), (1000, 0, 513), (1500, 0, 64), (300, 0, 2051),
                                   (2050, 0, 1025)])
def test_routes_agree(hd, plain, torch_cuda, dtype, reserve, M, N, K):
    if reserve:
        plain.reserve(hd.lib().hdbf_workspace_bytes_for(1024))
    lower, N = N == 0, N or M
    rng = np.random.default_rng(M + N + K)
    lda = M + 3
    A = np.zeros((lda, K), dtype)
    A[:M] = rng.integers(-8, 9, (M, K))
    B = A[:N] if lower else rng.integers(-8, 9, (N, K)).astype(dtype)
    C = rng.integers(-99, 100, (M, N)).astype(dtype)
    dA, dB, dC = dev(torch_cuda, A), dev(torch_cuda, B), dev(torch_cuda, C)
    tail = "" if dtype == np.float32 else "_double"
    if lower:
        hd.call("syrk_lower_update" + tail, plain.ptr, N, K, ptr(dA), lda, ptr(dC), M)
    else:
        hd.call("gemm_nt_update" + tail, plain.ptr, M, N, K, ptr(dA), lda, ptr(dB), N, ptr(dC), M)
    torch_cuda.cuda.synchronize()
    plain.check()
    want = C - (A[:M].astype(np.float64) @ B.astype(np.float64).T)  # below 2^24: exact
    if lower:
        want = np.tril(want) + np.triu(C, 1)
    np.testing.assert_array_equal(host2d(dC, M, M, N), want.astype(dtype))


@pytest.mark.parametrize("nbytes", [1, 1 << 20])
def test_small_reservation(hd, plain, torch_cuda, nbytes):
    """A reservation below the smallest arena still gives the split-K scratch its room."""
    M, N, K = 777, 640, 2100
    plain.reserve(nbytes)
    rng = np.random.default_rng(1)
    A, B, C = (rng.integers(-8, 9, s).astype(np.float32) for s in ((M, K), (N, K), (M, N)))
    free = torch_cuda.cuda.mem_get_info()[0]
    dA, dB, dC = dev(torch_cuda, A), dev(torch_cuda, B), dev(torch_cuda, C)
    hd.call("gemm_nt_update", plain.ptr, M, N, K, ptr(dA), M, ptr(dB), N, ptr(dC), M)
    torch_cuda.cuda.synchronize()
    plain.check()
    np.testing.assert_array_equal(host2d(dC, M, M, N), C - A @ B.T)
    # the arena was whole when the reservation returned: nothing grew afterwards
    assert free - torch_cuda.cuda.mem_get_info()[0] < 64 << 20
    assert plain_arena(hd, torch_cuda, nbytes) >= 256 << 20


def plain_arena(hd, torch, nbytes):
    """Device memory that a new handle takes for a reservation."""
    h = hd.Handle(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    h.reserve(nbytes)
    after = torch.cuda.mem_get_info()[0]
    h.close()
    return before - after
