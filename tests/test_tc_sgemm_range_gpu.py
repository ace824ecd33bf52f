"""FP32 updates on the tensor cores at the ends of the exponent range and over many
tiles and K chunks: entry by entry against FP64, and no further from it than the FP32
kernel.  Every call is checked to have taken the tensor-core kernel."""
import os

import numpy as np
import pytest

from tests.common import dev, host2d, ptr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def handles(hd, torch_cuda):
    out = {}
    for mode in (0, 2):  # never / wherever possible
        os.environ["HDBF_TC_SGEMM"] = str(mode)
        try:
            out[mode] = hd.Handle(torch_cuda.cuda.current_stream().cuda_stream)
        finally:
            del os.environ["HDBF_TC_SGEMM"]
        out[mode].reserve(hd.lib().hdbf_workspace_bytes_for(8192))
    yield out
    torch_cuda.cuda.synchronize()
    for h in out.values():
        h.close()


def product(torch, hd, h, A, B, C, lower=False, tensor=True):
    M, K = A.shape
    N = B.shape[0]
    dA, dB, dC = dev(torch, A), dev(torch, B), dev(torch, C)
    h.profile_begin()
    if lower:
        hd.call("syrk_lower_update", h.ptr, N, K, ptr(dA), M, ptr(dC), M)
    else:
        hd.call("gemm_nt_update", h.ptr, M, N, K, ptr(dA), M, ptr(dB), N, ptr(dC), M)
    ran = h.profile_end().get("tc_gemm_kernels", (0,))[0]
    torch.cuda.synchronize()
    h.check()
    assert h.device_errors() == 0
    assert (ran > 0) == tensor
    return host2d(dC, M, M, N)


def uniform(shape, seed, low=-1.0):
    return np.random.default_rng(seed).uniform(low, 1, shape).astype(np.float32)


def entry_bound(A, B, C):
    """Six of nine products, 2^-23 of |x||y| each; a truncation of 2^-22 per 64 of K, a
    rounding of 2^-24 per further chunk and one of C; and half a unit of the subnormal
    grid, which the final result has to lie on."""
    K = A.shape[1]
    size = np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64).T
    return ((2.0 ** -22 + 2.0 ** -23 + 2.0 ** -24 * (K / 64 + 2)) * size + 2.0 ** -23 * np.abs(C)
            + 2.0 ** -149)


@pytest.mark.parametrize("case", ["rows_small", "rows_subnormal", "both_small", "wide", "mixed",
                                  "columns"])
def test_every_entry(hd, torch_cuda, handles, case):
    M, N, K = 300, 280, 200
    A, B, C = uniform((M, K), 1), uniform((N, K), 2), uniform((M, N), 3)

    def rows(lo, hi, n):
        return (2.0 ** np.linspace(lo, hi, n).astype(np.int32))[:, None]

    if case == "rows_small":  # some rows at the end of the normal range, some at 1
        s = rows(-125, 0, M)
        A, C = A * s.astype(np.float32), C * s.astype(np.float32)
    elif case == "rows_subnormal":
        s = rows(-148, 0, M)  # (an operand wholly below 2^-90 has the FP32 kernel)
        A = (A * s).astype(np.float32)
        C *= 0
    elif case == "both_small":  # results among the subnormals
        A, B = A * np.float32(2.0 ** -80), B * np.float32(2.0 ** -60)
        C = (C * 2.0 ** -140).astype(np.float32)
    elif case == "wide":
        A, C = [(X * rows(-120, 60, M)).astype(np.float32) for X in (A, C)]
    elif case == "mixed":  # tiny next to ordinary entries, met by zeros of B in half the rows
        A[:, ::2] *= np.float32(2.0 ** -120)
        B[::2, 1::2] = 0
        C[:, ::2] *= np.float32(2.0 ** -120)
    else:
        B = (B * rows(-125, 10, N)).astype(np.float32)
        C = (C * rows(-125, 10, N).T).astype(np.float32)
    got = product(torch_cuda, hd, handles[2], A, B, C)
    want = C - A.astype(np.float64) @ B.astype(np.float64).T
    assert (np.abs(got - want) <= entry_bound(A, B, C)).all()


@pytest.mark.parametrize("case", ["large", "sum_overflows", "nan", "inf"])
def test_fp32_kernel_behind(hd, torch_cuda, handles, case):
    """Outside the range, at a size whose FP32 kernel is the 128 x 128 one: its results."""
    M, N, K = 2304, 1100, 600
    A, B, C = uniform((M, K), 1), uniform((N, K), 2), uniform((M, N), 3)
    if case == "large":
        A[5, 7] = 2.0 ** 115
    elif case == "sum_overflows":
        A, B = A * np.float32(2.0 ** 40), B * np.float32(2.0 ** 40)
    elif case == "nan":
        B[1000, 599] = np.nan
    else:
        A[2303, 0] = -np.inf
    got = product(torch_cuda, hd, handles[2], A, B, C)
    # the same kernel without a split of K
    want = C - A.astype(np.float64) @ B.astype(np.float64).T
    plain = product(torch_cuda, hd, handles[0], A, B, C, tensor=False)
    odd = ~np.isfinite(want)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(plain))
    np.testing.assert_array_equal(got[odd], plain[odd])
    size = (np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64).T + np.abs(C))[~odd]
    assert (np.abs(got[~odd] - want[~odd]) <= (K + 2) * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("M,N,K,lower", [(4096, 1024, 1000, False), (4096, 2048, 4100, False),
                                         (2500, 2500, 700, False), (4096, 4096, 2100, True),
                                         (3000, 3000, 520, True)])
@pytest.mark.parametrize("low", [-1.0, 0.0])
def test_long_k(hd, torch_cuda, handles, M, N, K, lower, low):
    """More than one tile per CTA, ring and accumulators round many times, more than one
    K chunk."""
    A, B, C = uniform((M, K), 4, low), uniform((N, K), 5, low), uniform((M, N), 6, low)
    if lower:
        B = A
    a, b = torch_cuda.from_numpy(A).cuda().double(), torch_cuda.from_numpy(B).cuda().double()
    want = C - (a @ b.T).cpu().numpy()
    bound = (2.0 ** -22 + 2.0 ** -23 + 2.0 ** -24 * (K / 64 + 2)) * (
        a.abs() @ b.abs().T).cpu().numpy() + 2.0 ** -23 * np.abs(C)
    got = product(torch_cuda, hd, handles[2], A, B, C, lower)
    plain = product(torch_cuda, hd, handles[0], A, B, C, lower, tensor=False)
    where = np.tril(np.ones((M, N), bool)) if lower else np.ones((M, N), bool)
    np.testing.assert_array_equal(got[~where], C[~where])
    assert (np.abs(got - want) <= bound)[where].all()
    rms = lambda x: float(np.sqrt(np.mean((x - want)[where] ** 2)))
    assert rms(got) <= 1.05 * rms(plain)


@pytest.mark.parametrize("M,N,K,lower", [(6000, 6000, 6000, True), (5000, 4000, 6200, False)])
def test_same_bits_whatever_the_arena(hd, torch_cuda, M, N, K, lower):
    """How K is cut follows from the shape, not from how far earlier calls grew the
    handle's arena."""
    A = uniform((M, K), 7)
    B = A if lower else uniform((N, K), 8)
    C = uniform((M, N), 9)
    out = []
    h = hd.Handle(torch_cuda.cuda.current_stream().cuda_stream)
    for order in (64, max(M, N) + K, 20000):
        h.reserve(hd.lib().hdbf_workspace_bytes_for(order))
        out.append(product(torch_cuda, hd, h, A, B, C, lower))
    h.close()
    np.testing.assert_array_equal(out[1], out[0])


def test_same_factor_whatever_the_handle_did_before(hd, torch_cuda):
    """An LU whose outer update of K = 6144 is cut in two, before and after the same
    handle had a larger problem."""
    n = 12288
    g = torch_cuda.Generator(device="cuda")
    g.manual_seed(1)
    A0 = torch_cuda.rand(n, n, generator=g, device="cuda") * 2 - 1
    A0[torch_cuda.arange(n), torch_cuda.randperm(n, generator=g, device="cuda")] += 200.0
    h = hd.Handle(torch_cuda.cuda.current_stream().cuda_stream)

    def factor():
        A = A0.clone()
        ipiv = torch_cuda.zeros(n, dtype=torch_cuda.int32, device="cuda")
        info = torch_cuda.zeros(1, dtype=torch_cuda.int32, device="cuda")
        hd.call("double_blocked_getrf", h.ptr, ptr(A), n, n, 6144, 512, 0, 0, ptr(ipiv), ptr(info))
        torch_cuda.cuda.synchronize()
        h.check()
        assert info.item() == 0
        return A, ipiv

    first = factor()
    h.reserve(hd.lib().hdbf_workspace_bytes_for(32768))
    again = factor()
    h.close()
    assert torch_cuda.equal(first[1], again[1])
    assert torch_cuda.equal(first[0], again[0])


@pytest.mark.parametrize("kind", ["posv", "gesv"])
def test_prec_fp32_is_simt(hd, torch_cuda, kind):
    """HDBF_PREC_FP32 is documented as FP32 SIMT updates, whatever the handle's own FP32
    factorizations use (the same orders on it do run on the tensor cores)."""
    import ctypes

    torch, n = torch_cuda, 4096
    h = hd.Handle(torch.cuda.current_stream().cuda_stream)
    A = torch.full((n, n), 0.5 / n, dtype=torch.float64, device="cuda")
    A.diagonal().fill_(1.0)
    B = torch.ones(1, n, dtype=torch.float64, device="cuda")
    X, out = torch.zeros_like(B), hd.IrInfo()
    h.profile_begin()
    st = hd.call("hdbf_d%s_mixed_auto" % kind, h.ptr, hd.PREC["fp32"], A.data_ptr(), n, n, 1,
                 B.data_ptr(), n, X.data_ptr(), n, 1e-13, 30, ctypes.byref(out))
    ran = h.profile_end()
    assert st == 0 and out.converged and out.final_precision == hd.PREC["fp32"]
    assert ran["sgemm_sub_kernel"][0] > 0
    assert ran.get("tc_gemm_kernels", (0,))[0] == 0
    A32, info = A.float(), torch.zeros(1, dtype=torch.int32, device="cuda")
    h.profile_begin()
    hd.call("double_blocked_potrf", h.ptr, ptr(A32), n, n, 2048, 256, ptr(info))
    assert h.profile_end()["tc_gemm_kernels"][0] > 0
    h.close()
