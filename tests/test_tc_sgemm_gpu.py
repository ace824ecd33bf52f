"""FP32 updates on the tensor cores (three BF16 words per operand): error against
FP64 no larger than the FP32 kernel's, at the edges of its tiles and K chunks, and
the FP32 kernel's results where the split has no range."""
import os

import numpy as np
import pytest

from tests.common import dev, host2d, ptr

pytestmark = pytest.mark.gpu


@pytest.fixture()
def handles(hd, torch_cuda):
    out = {}
    for mode in (0, 2):  # never / wherever possible
        os.environ["HDBF_TC_SGEMM"] = str(mode)
        try:
            out[mode] = hd.Handle(torch_cuda.cuda.current_stream().cuda_stream)
        finally:
            del os.environ["HDBF_TC_SGEMM"]
        out[mode].reserve(hd.lib().hdbf_workspace_bytes_for(2048))
    yield out
    torch_cuda.cuda.synchronize()
    for h in out.values():
        h.close()


def product(torch, hd, h, A, B, C, lower=False):
    M, K = A.shape
    N = B.shape[0]
    dA, dB, dC = dev(torch, A), dev(torch, B), dev(torch, C)
    if lower:
        hd.call("syrk_lower_update", h.ptr, N, K, ptr(dA), M, ptr(dC), M)
    else:
        hd.call("gemm_nt_update", h.ptr, M, N, K, ptr(dA), M, ptr(dB), N, ptr(dC), M)
    torch.cuda.synchronize()
    h.check()
    assert h.device_errors() == 0
    return host2d(dC, M, M, N)


def operands(M, N, K, lower, positive=False):
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    A, B, C = (rng.uniform(0 if positive else -1, 1, s).astype(np.float32)
               for s in ((M, K), (N, K), (M, N)))
    return A, (A if lower else B), C


@pytest.mark.parametrize("M,N,K", [(1, 40, 64), (127, 33, 1), (128, 256, 64), (129, 257, 65),
                                   (300, 300, 63), (256, 512, 1000), (1000, 130, 129),
                                   (777, 640, 2100), (2048, 300, 4096)])
@pytest.mark.parametrize("lower,positive", [(False, False), (True, False), (False, True)])
def test_error_not_above_fp32(hd, torch_cuda, handles, M, N, K, lower, positive):
    if lower:
        N = M = min(M, 1000)
    A, B, C = operands(M, N, K, lower, positive)
    want = C - A.astype(np.float64) @ B.astype(np.float64).T
    got = product(torch_cuda, hd, handles[2], A, B, C, lower)
    if lower:
        up = np.triu_indices(M, 1)
        np.testing.assert_array_equal(got[up], C[up])
        want[up] = C[up]
    # the final subtraction rounds once (2^-24); the products carry at most
    # 2^-23 of |x||y| (six of nine kept), their sums a truncation of 2^-22 per
    # 64 of K and a rounding of 2^-24 per further chunk
    bound = (2.0 ** -22 + 2.0 ** -23 + 2.0 ** -24 * (K / 64 + 2)) * (
        np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64).T) + 2.0 ** -23 * np.abs(C)
    assert (np.abs(got - want) <= bound).all()
    if K >= 63 and M * N >= 1000:
        plain = product(torch_cuda, hd, handles[0], A, B, C, lower)
        if lower:
            plain[up] = C[up]
        rms = lambda x: float(np.sqrt(np.mean((x - want) ** 2)))
        assert rms(got) <= 1.05 * rms(plain)


@pytest.mark.parametrize("case", ["inf", "nan", "huge", "tiny", "zero", "graded"])
def test_range(hd, torch_cuda, handles, case):
    M, N, K = 300, 280, 200
    A, B, C = operands(M, N, K, False)
    if case == "inf":
        A[17, 5] = np.inf
    elif case == "nan":
        B[250, 199] = np.nan
    elif case == "huge":
        A[3, 3] = 3e38
        B *= np.float32(0.01)
    elif case == "tiny":
        A *= np.float32(1e-36)
        C *= np.float32(1e-36)
    elif case == "zero":
        A[:] = 0
    else:  # rows over the whole exponent range the split covers
        A *= np.float32(2.0) ** np.linspace(-60, 60, M).astype(np.int32)[:, None]
        C *= np.float32(2.0) ** np.linspace(-60, 60, M).astype(np.int32)[:, None]
    got = product(torch_cuda, hd, handles[2], A, B, C)
    plain = product(torch_cuda, hd, handles[0], A, B, C)
    if case in ("inf", "nan", "huge", "tiny", "zero"):  # the FP32 kernel's results
        np.testing.assert_array_equal(got, plain)
        return
    want = C - A.astype(np.float64) @ B.astype(np.float64).T
    scale = np.abs(C) + np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64).T
    assert (np.abs(got - want) <= 2.0 ** -20 * scale).all()
