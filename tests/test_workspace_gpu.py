"""Device memory that a handle takes: the operand words of the tensor-core updates only
for the calls that run them."""
import pytest

from tests.common import ptr

pytestmark = pytest.mark.gpu


def taken(torch, call):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    call()
    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info()[0]


def spd(torch, n, dtype):
    A = torch.full((n, n), 0.5 / n, dtype=dtype, device="cuda")
    A.diagonal().fill_(1.0)
    return A


@pytest.mark.parametrize("kind", ["potrf64", "getrf64", "posv", "gesv"])
def test_no_words_for_fp64_and_mixed(hd, torch_cuda, kind):
    """FP64 calls (whose arena is that of twice the order) and mixed ones: less than the
    words of one stream at that order."""
    torch, n = torch_cuda, 6144
    h = hd.Handle(torch.cuda.current_stream().cuda_stream)
    h.set_graphs(False)  # a graph's own memory is not the handle's workspace
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    ipiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    A = spd(torch, n, torch.float64 if kind.endswith("64") else torch.float32)

    def call():
        if kind == "potrf64":
            hd.call("double_blocked_potrf_double", h.ptr, ptr(A), n, n, 2048, 256, ptr(info))
        elif kind == "getrf64":
            hd.call("double_blocked_getrf_double", h.ptr, ptr(A), n, n, 2048, 256, 0, 0, ptr(ipiv),
                    ptr(info))
        elif kind == "posv":
            assert hd.call("hdbf_spotrf_mixed", h.ptr, hd.PREC["bf16"], ptr(A), n, n, 512,
                           ptr(info)) == 0
        else:
            assert hd.call("hdbf_sgetrf_mixed", h.ptr, hd.PREC["fp16x3"], ptr(A), n, n, 512,
                           ptr(ipiv), ptr(info)) == 0

    got = taken(torch, call)
    assert info.item() == 0
    h.close()
    # the layout less the words: exchange slots, inverses, split-K halves, swap and solve
    # scratch; for mixed calls the 16-bit shadows and the backup of the matrix too
    order = 2 * n + 128 if kind.endswith("64") else n
    words = 12 * order * 2048
    assert got < 400 * 2 ** 20 + (0 if kind.endswith("64") else 4 * n * n + 16 * n * 512)
    assert kind != "potrf64" or got < words


def test_capture_without_words(hd, torch_cuda):
    """A call in a caller's capture whose words have no room runs, on the FP32 kernels."""
    torch, n = torch_cuda, 2560
    stream = torch.cuda.Stream()
    h = hd.Handle(stream.cuda_stream)
    h.reserve(hd.lib().hdbf_workspace_bytes_for(64))
    K = 1200
    B = torch.rand(K, n, device="cuda")
    C0 = torch.rand(n, n, device="cuda")
    C = C0.clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        hd.call("gemm_nt_update", h.ptr, n, n, K, ptr(B), n, ptr(B), n, ptr(C), n)
    h.check()
    g.replay()
    torch.cuda.synchronize()
    want = C0.double() - B.double().T @ B.double()
    size = B.double().T @ B.double() + C0.double()
    assert bool(((C.double() - want).abs() <= (K + 2) * 2.0 ** -24 * size).all())
    h.close()
