"""The work this library is used for, as cases that can be timed and checked.

Every case goes through a public entry point of the C ABI with the arguments a
program passes: a matrix in device memory that is factored in place (so a pass
first copies the pristine matrix over it, as a program with a new matrix would),
device pivots and info, and one handle per process.

Kinds: FP32 Cholesky and partially pivoted LU (``potrf``, ``getrf``), their FP64
twins (``potrf64``, ``getrf64``), mixed-precision solves refined to an FP64
backward error of 1e-13 (``posv``, ``gesv``) and the batched factor-and-solve of
many small systems (``batch``).
"""
import ctypes

import numpy as np
import torch

import hygondoubleblockedfactorizations_b200 as hd
from hygondoubleblockedfactorizations_b200.batch import DeviceBatch

_state = {}


def _handle(order):
    """The process's handle on the current stream, with room for `order`."""
    if "handle" not in _state:
        _state["handle"] = hd.Handle(torch.cuda.current_stream().cuda_stream)
    h = _state["handle"]
    h.reserve(hd.lib().hdbf_workspace_bytes_for(order))
    return h


# ------------------------------------------------------------------- cases
def listed():
    return [
        # A small covariance or normal-equation matrix factored on its own: the
        # call is all latency.
        {"name": "potrf-256", "kind": "potrf", "n": 256, "lda": 256, "nb": 256, "b": 64},
        # The base Cholesky configuration of the tests (outer 512, inner 64).
        {"name": "potrf-2048", "kind": "potrf", "n": 2048, "lda": 2048, "nb": 512, "b": 64},
        # An odd order inside a larger buffer: ragged tiles, a leading dimension
        # that is no multiple of four floats.
        {"name": "potrf-7777", "kind": "potrf", "n": 7777, "lda": 7779, "nb": 2048, "b": 256},
        # The headline order and blocks.
        {"name": "potrf-32768", "kind": "potrf", "n": 32768, "lda": 32768, "nb": 4096, "b": 512},
        # A small general system, odd order, interchanges applied at once.
        {"name": "getrf-1001", "kind": "getrf", "n": 1001, "lda": 1001, "nb": 512, "b": 128,
         "batched_pivots": False},
        # An ordinary LU with the sweep's smaller blocks.
        {"name": "getrf-8192", "kind": "getrf", "n": 8192, "lda": 8192, "nb": 2048, "b": 256,
         "batched_pivots": True},
        # The headline LU: headline order and blocks.
        {"name": "getrf-32768", "kind": "getrf", "n": 32768, "lda": 32768, "nb": 8192, "b": 1024,
         "batched_pivots": True},
        # FP64 accuracy from an FP16 Cholesky, several right-hand sides.
        {"name": "posv-fp16-16384", "kind": "posv", "n": 16384, "nb": 1024, "prec": "fp16",
         "nrhs": 16},
        # The same for a general matrix with the split FP16 updates.
        {"name": "gesv-fp16x3-8192", "kind": "gesv", "n": 8192, "nb": 512, "prec": "fp16x3",
         "nrhs": 16},
        # The uneven batch: 4096 SPD systems of order 16..512 and 2048 general ones of 32..768.
        {"name": "batch-6144", "kind": "batch", "spd": 4096, "gen": 2048, "lo": 16, "hi_spd": 512,
         "hi_gen": 768, "variant": 2},
        # A small batch of small systems: few blocks, short chains.
        {"name": "batch-256", "kind": "batch", "spd": 128, "gen": 128, "lo": 16, "hi_spd": 128,
         "hi_gen": 128, "variant": 0},
        # The FP64 twin of the LU, at an order where its panel and its GEMM both count.
        {"name": "getrf64-4096", "kind": "getrf64", "n": 4096, "lda": 4096, "nb": 2048, "b": 256,
         "batched_pivots": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["potrf", "potrf", "potrf", "getrf", "getrf", "getrf", "posv", "gesv",
                       "batch", "batch", "potrf64", "getrf64"])
    if kind in ("potrf", "getrf"):
        n = _log_int(rng, 200, 20000)
        if rng.random() < 0.5:
            n = max(256, n // 256 * 256)
        nb, b = rng.choice([(512, 64), (1024, 128), (2048, 256), (4096, 256), (4096, 512),
                            (8192, 1024)])
        c = {"kind": kind, "n": n, "lda": n + rng.choice([0, 0, 0, 1, 4, 64]), "nb": nb, "b": b}
    elif kind in ("potrf64", "getrf64"):
        n = _log_int(rng, 300, 6000)
        nb, b = rng.choice([(512, 64), (1024, 128), (2048, 256)])
        c = {"kind": kind, "n": n, "lda": n + rng.choice([0, 0, 1, 64]), "nb": nb, "b": b}
    elif kind in ("posv", "gesv"):
        n = _log_int(rng, 1024, 16384)
        if rng.random() < 0.5:
            n = n // 512 * 512
        prec = rng.choice(["bf16", "fp16", "bf16x3", "fp16x3"] if kind == "posv" else
                          ["bf16x3", "fp16x3", "fp32"])
        return {"kind": kind, "n": n, "nb": rng.choice([256, 512, 1024]), "prec": prec,
                "nrhs": rng.choice([1, 4, 16, 32])}
    else:
        return {"kind": "batch", "spd": rng.randint(0, 2048), "gen": rng.randint(16, 1024),
                "lo": rng.choice([16, 32]), "hi_spd": rng.randint(64, 512),
                "hi_gen": rng.randint(64, 768), "variant": rng.randint(0, 5)}
    if kind in ("getrf", "getrf64"):
        c["batched_pivots"] = rng.random() < 0.7
    return c


# ------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _spd(n, g, dtype, ridge=1.0):
    """Covariance of n variables from at most 1024 uniform factors plus a ridge."""
    r = min(n, 1024)
    G = torch.rand(n, r, generator=g, device="cuda", dtype=dtype).mul_(2).sub_(1)
    A = torch.mm(G, G.t()).div_(r)
    for i in range(0, n, 4096):  # exactly symmetric
        for j in range(0, i + 1, 4096):
            blk = A[i:i + 4096, j:j + 4096]
            if i == j:
                blk.copy_(torch.tril(blk) + torch.tril(blk, -1).t())
            else:
                A[j:j + 4096, i:i + 4096] = blk.t()
    A.diagonal().add_(ridge)
    return A


def _general(n, g, dtype):
    """Dense coupling U[-1,1) plus one strong coefficient per unknown, of either
    sign, whose rows come in no order: every column needs an interchange, and
    which one does not hang on the last bits."""
    A = torch.rand(n, n, generator=g, device="cuda", dtype=dtype).mul_(2).sub_(1)
    rows = torch.randperm(n, generator=g, device="cuda")
    sign = torch.randint(0, 2, (n,), generator=g, device="cuda").to(dtype).mul_(2).sub_(1)
    A[torch.arange(n, device="cuda"), rows] += sign * (2.0 * n ** 0.5)
    return A  # row j holds column j of the matrix (column-major storage)


def _matrix(case, seed):
    dtype = torch.float64 if case["kind"] in ("potrf64", "getrf64", "posv", "gesv") else \
        torch.float32
    g = _generator(seed)
    n = case["n"]
    if case["kind"] == "posv":
        A = _spd(n, g, dtype, 0.1)
    elif case["kind"].startswith("potrf"):
        A = _spd(n, g, dtype)
    else:
        A = _general(n, g, dtype)
    return A, g


def _batch_sizes(case):
    """Sizes are the case's, not the seed's: every seed has the same work."""
    rng = np.random.default_rng(3)
    spd = rng.integers(case["lo"], case["hi_spd"] + 1, size=case["spd"])
    gen = rng.integers(max(32, case["lo"]), case["hi_gen"] + 1, size=case["gen"])
    ops = np.concatenate([np.zeros(len(spd), np.int32), np.ones(len(gen), np.int32)])
    return ops, np.concatenate([spd, gen]).astype(np.int32)


def _batch_inputs(case, seed, batch):
    """Fills the packed batch: SPD systems are symmetric with a dominant
    diagonal, general ones as in `_general`; right-hand sides N(0,1)."""
    g = _generator(seed)
    batch.A.uniform_(-1.0, 1.0, generator=g)
    batch.b.normal_(generator=g)
    off = torch.from_numpy(batch.offsets).cuda()
    ns = torch.from_numpy(batch.ns.astype(np.int64)).cuda()
    op = torch.from_numpy(batch.ops.astype(np.int64)).cuda()
    # one (system, column) pair for every row of every system
    sysid = torch.repeat_interleave(torch.arange(batch.count, device="cuda"), ns)
    start = torch.cumsum(ns, 0) - ns
    col = torch.arange(len(sysid), device="cuda") - start[sysid]
    n = ns[sysid]
    # general: the strong entry of a column sits in a random row, each row once
    key = sysid.double() + torch.rand(len(sysid), generator=g, device="cuda",
                                      dtype=torch.float64)
    perm = torch.argsort(key) - start[sysid]
    sign = torch.randint(0, 2, (len(sysid),), generator=g, device="cuda") * 2 - 1
    row = torch.where(op[sysid] == 1, perm, col)
    for i in np.nonzero(batch.ops == 0)[0]:
        M = batch.matrix(int(i))
        M.copy_(torch.tril(M) + torch.tril(M, -1).t())
    add = torch.where(op[sysid] == 1, sign * 2.0 * n.double().sqrt(), n.double().sqrt() * 1.5 + 1)
    where = off[sysid] + col * n + row
    batch.A[where] += add.float()
    return batch


# ----------------------------------------------------------------- the work
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        h = _handle(1024)
        b = _batch_inputs(case, seed, DeviceBatch(torch, *_batch_sizes(case)))
        return {"case": case, "h": h, "batch": b, "A0": b.A.clone(), "b0": b.b.clone()}
    n = case["n"]
    A, g = _matrix(case, seed)
    if kind in ("posv", "gesv"):
        B = torch.randn(case["nrhs"], n, generator=g, device="cuda", dtype=torch.float64)
        return {"case": case, "h": _handle(n), "A": A, "B": B, "X": torch.zeros_like(B),
                "out": hd.IrInfo()}
    wide = A.dtype == torch.float64
    lda = case["lda"]
    A0 = A
    if lda != n:
        A0 = torch.zeros(n, lda, dtype=A.dtype, device="cuda")
        A0[:, :n] = A
        del A
    s = {"case": case, "h": _handle(2 * n + 128 if wide else n), "A0": A0,
         "A": torch.empty_like(A0), "info": torch.zeros(1, dtype=torch.int32, device="cuda")}
    if kind.startswith("getrf"):
        tile = 64  # columns of the caller's swap buffer
        s["ipiv"] = torch.zeros(n, dtype=torch.int32, device="cuda")
        s["moves"] = torch.zeros(2, n, dtype=torch.int32, device="cuda")
        s["swap"] = torch.zeros(tile, n, dtype=A0.dtype, device="cuda")
        s["host"] = [np.zeros(n, np.int32) for _ in range(4)]
        s["ws"] = hd.WorkspacePivot(s["moves"][0].data_ptr(), s["moves"][1].data_ptr(),
                                    s["swap"].data_ptr(), *[a.ctypes.data for a in s["host"]],
                                    n, tile)
    return s


def run(s):
    c, h = s["case"], s["h"]
    kind = c["kind"]
    if kind == "batch":
        b = s["batch"]
        b.A.copy_(s["A0"])
        b.b.copy_(s["b0"])
        if b.run(h, c["variant"]) != 0:
            raise RuntimeError("hdbf_batched_factor_solve failed")
        return {"A": b.A, "b": b.b, "ipiv": b.ipiv_buf, "info": b.info}
    n = c["n"]
    if kind in ("posv", "gesv"):
        st = hd.call("hdbf_dposv_mixed_auto" if kind == "posv" else "hdbf_dgesv_mixed_auto", h.ptr,
                     hd.PREC[c["prec"]], s["A"].data_ptr(), n, n, c["nrhs"], s["B"].data_ptr(), n,
                     s["X"].data_ptr(), n, 1e-13, 30, ctypes.byref(s["out"]))
        if st != 0 or not s["out"].converged:
            raise RuntimeError("the solve did not converge")
        return {"X": s["X"]}
    A = s["A"]
    A.copy_(s["A0"])
    tail = "_double" if kind.endswith("64") else ""
    if kind.startswith("potrf"):
        hd.call("double_blocked_potrf%s_kblocked_syrk" % tail, h.ptr, A.data_ptr(), c["lda"], n,
                c["nb"], c["b"], 0, s["info"].data_ptr())
        h.check(kind)
        return {"A": A[:, :n], "info": s["info"]}
    if c["batched_pivots"]:
        hd.call("double_blocked_getrf%s_batched_pivot" % tail, h.ptr, A.data_ptr(), c["lda"], n,
                c["nb"], c["b"], 1, 0, 0, s["ipiv"].data_ptr(), s["info"].data_ptr(),
                ctypes.byref(s["ws"]))
    else:
        hd.call("double_blocked_getrf%s" % tail, h.ptr, A.data_ptr(), c["lda"], n, c["nb"], c["b"],
                0, 0, s["ipiv"].data_ptr(), s["info"].data_ptr())
    h.check(kind)
    return {"A": A[:, :n], "ipiv": s["ipiv"], "info": s["info"]}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        ops, ns = _batch_sizes(case)
        n = ns.astype(np.float64)
        flops = np.where(ops == 0, n ** 3 / 3, 2 * n ** 3 / 3) + 2 * n * n
        move = np.where(ops == 0, 4 * n * n, 8 * n * n) + 8 * n
        return {"bytes": float(move.sum()), "flops": float(flops.sum())}
    n = float(case["n"])
    half = kind.startswith("po")  # a Cholesky reads and writes one triangle
    flops = n ** 3 / 3 if half else 2 * n ** 3 / 3
    if kind in ("posv", "gesv"):
        # A once (FP64), and B and X; one factorization and one pair of solves
        return {"bytes": 8 * n * n * (0.5 if half else 1) + 16 * n * case["nrhs"],
                "flops": flops + 2 * n * n * case["nrhs"]}
    size = 8 if kind.endswith("64") else 4
    return {"bytes": 2 * size * n * n * (0.5 if half else 1), "flops": flops}


# -------------------------------------------------------------- 64-bit answers
def _lu64(A_colmajor):
    """Packed LU of the matrix whose columns are the rows given, laid out the same."""
    LU, _ = torch.linalg.lu_factor(A_colmajor.t())
    return LU.t()


def _exact_batch(case, seed):
    b = _batch_inputs(case, seed, DeviceBatch(torch, *_batch_sizes(case)))
    A, x = torch.empty_like(b.A, dtype=torch.float64), torch.empty_like(b.b, dtype=torch.float64)
    for op in (0, 1):
        ids = np.nonzero(b.ops == op)[0]
        ids = ids[np.argsort(b.ns[ids], kind="stable")]
        for at in range(0, len(ids), 128):
            part = ids[at:at + 128]
            top = int(b.ns[part].max())
            # a system of lower order sits in the corner of an identity
            M = torch.eye(top, dtype=torch.float64, device="cuda").repeat(len(part), 1, 1)
            r = torch.zeros(len(part), top, 1, dtype=torch.float64, device="cuda")
            for k, i in enumerate(part):
                n = int(b.ns[i])
                M[k, :n, :n] = b.matrix(int(i))
                r[k, :n, 0] = b.rhs(int(i))
            if op == 0:
                F = torch.linalg.cholesky(M)
                r = torch.cholesky_solve(r, F)
                F = F + torch.triu(M, 1)
            else:
                F, p = torch.linalg.lu_factor(M)
                r = torch.linalg.lu_solve(F, p, r)
            for k, i in enumerate(part):
                n, o, q = int(b.ns[i]), int(b.offsets[i]), int(b.roffsets[i])
                A[o:o + n * n].view(n, n).copy_(F[k, :n, :n].t())
                x[q:q + n] = r[k, :n, 0]
    return {"A": A, "b": x, "ipiv": None, "info": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, seed)
    A, g = _matrix(case, seed)
    if kind in ("posv", "gesv"):
        B = torch.randn(case["nrhs"], case["n"], generator=g, device="cuda", dtype=torch.float64)
        if kind == "posv":
            return {"X": torch.cholesky_solve(B.t(), torch.linalg.cholesky(A)).t().contiguous()}
        return {"X": torch.linalg.solve(A.t(), B.t()).t().contiguous()}
    if kind.startswith("potrf"):
        A = A.double()
        L = torch.linalg.cholesky(A)
        F = L.t()  # row j holds column j
        n = case["n"]
        for i in range(0, n, 4096):  # the other triangle keeps the input
            blk = F[i:i + 4096]
            keep = torch.arange(n, device="cuda")[None, :] < torch.arange(
                i, min(n, i + 4096), device="cuda")[:, None]
            blk[keep] = A[i:i + 4096][keep]
        return {"A": F, "info": None}
    return {"A": _lu64(A.double()), "ipiv": None, "info": None}
