"""The calls whose speed counts: one dict per case, and how it is prepared, run and checked.

Every case is one call (or one in-place solve, with its right-hand side put
back first) of the Python front-end, on the sizes of this repository's own
workloads: the small calls of its smoke test and unit tests, the n = 4096 and
n = 16384 SYRK / TRSM, the wide-exponent SYR2K / TRMM / SYMM, the FP64 DSYRK
and the batch of uneven instances.

Matrices named *_cm hold column-major data: a (cols, rows) torch tensor is
the rows x cols column-major matrix.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "tensor-blas_b200", "python"))
import TensorBLAS as T  # noqa: E402

_L, _P = ctypes.c_long, ctypes.c_void_p
T.lib.tb_dsyrk_ozaki.argtypes = [ctypes.c_char, ctypes.c_char, _L, _L, ctypes.c_double, _P, _L, ctypes.c_double, _P,
                                 _L, ctypes.c_int]
T.lib.tb_dsyrk_ozaki.restype = ctypes.c_int

PREC = {"plain": T.PLAIN, "split": T.SPLIT, "fp8": T.FP8}


def listed():
    return [
        # the smallest calls: the reference's two Python functions on a few
        # hundred rows (synchronous: latency and launches are all there is)
        {"name": "tc_syrk_384", "op": "tc_syrk", "n": 384, "k": 200, "nb": 256},
        {"name": "tc_trsm_320", "op": "tc_trsm", "m": 96, "n": 320, "nb": 128},
        # a solve with few right-hand sides: the recursion's serial chain
        {"name": "trsm_left_4096x256", "op": "strsm", "side": "L", "m": 4096, "n": 256, "nb": 256, "prec": "plain"},
        # an ordinary covariance-sized SYRK
        {"name": "syrk_4096", "op": "ssyrk", "n": 4096, "k": 4096, "trans": "N", "beta": 0.0, "prec": "plain"},
        # the headline pair
        {"name": "syrk_16384", "op": "ssyrk", "n": 16384, "k": 16384, "trans": "N", "beta": 0.0, "prec": "plain"},
        {"name": "trsm_left_16384", "op": "strsm", "side": "L", "m": 16384, "n": 16384, "nb": 512, "prec": "plain"},
        # the reference's own side (X A^T = B) at FP32 accuracy, with ragged sizes
        {"name": "trsm_right_split_ragged", "op": "strsm", "side": "R", "m": 6003, "n": 4100, "nb": 512,
         "prec": "split"},
        # wide-exponent operands at FP32 accuracy, from row-major torch matrices
        {"name": "syr2k_split_16384x4096", "op": "syr2k", "n": 16384, "k": 4096, "layout": "row", "prec": "split"},
        # the same data class through the plain form (column-major operands)
        {"name": "trmm_upper_16384", "op": "trmm", "m": 16384, "n": 16384, "uplo": "U", "layout": "col",
         "prec": "plain"},
        # and through the block-scaled e4m3 form
        {"name": "symm_fp8_16384", "op": "symm", "m": 16384, "n": 16384, "uplo": "L", "beta": 0.0, "layout": "col",
         "prec": "fp8"},
        # FP64 on the INT8 tensor cores, slice count chosen by the library
        {"name": "dsyrk_ozaki_8192", "op": "dsyrk", "n": 8192, "k": 8192, "phi": 0.5},
        # many small uneven SYRK / TRSM instances, replayed as one CUDA graph
        {"name": "batch_512_split", "op": "batch", "count": 512, "lo": 64, "hi": 2048, "mix": 2025, "prec": "split"},
    ]


def _log(rng, lo, hi):
    """A size between lo and hi, spread over its logarithm; one in three a multiple of 64."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, v if rng.random() < 0.67 else (v + 32) // 64 * 64))


def _cost(case):
    """Tensor-core products of a case, in the order of its time."""
    return work(case)["flops"] * {"plain": 1.0, "split": 3.0, "fp8": 1.0}.get(case.get("prec"), 1.0)


def draw(rng):
    while True:
        op = rng.choice(["tc_syrk", "tc_trsm", "ssyrk", "ssyrk", "strsm", "strsm", "strsm", "syr2k", "trmm", "symm",
                         "dsyrk", "batch"])
        prec = rng.choice(["plain", "split"])
        prec8 = rng.choice(["plain", "split", "fp8"])
        layout = rng.choice(["row", "col"])
        if op == "tc_syrk":
            c = {"op": op, "n": _log(rng, 64, 2048), "k": _log(rng, 64, 2048), "nb": 256}
        elif op == "tc_trsm":
            c = {"op": op, "m": _log(rng, 64, 2048), "n": _log(rng, 64, 2048), "nb": rng.choice([128, 256])}
        elif op == "ssyrk":
            c = {"op": op, "n": _log(rng, 512, 16384), "k": _log(rng, 256, 16384), "trans": rng.choice(["N", "T"]),
                 "beta": rng.choice([0.0, 0.0, 0.5]), "prec": prec}
        elif op == "strsm":
            c = {"op": op, "side": rng.choice(["L", "R"]), "m": _log(rng, 256, 16384), "n": _log(rng, 256, 16384),
                 "nb": rng.choice([256, 512]), "prec": prec}
        elif op == "syr2k":
            c = {"op": op, "n": _log(rng, 512, 16384), "k": _log(rng, 256, 4096), "layout": layout, "prec": prec8}
        elif op == "trmm":
            c = {"op": op, "m": _log(rng, 512, 16384), "n": _log(rng, 512, 16384), "uplo": rng.choice(["L", "U"]),
                 "layout": layout, "prec": prec8}
        elif op == "symm":
            c = {"op": op, "m": _log(rng, 512, 16384), "n": _log(rng, 512, 16384), "uplo": rng.choice(["L", "U"]),
                 "beta": rng.choice([0.0, 0.5]), "layout": layout, "prec": prec8}
        elif op == "dsyrk":
            c = {"op": op, "n": _log(rng, 512, 8192), "k": _log(rng, 512, 8192), "phi": rng.choice([0.5, 2.0])}
        else:
            c = {"op": op, "count": _log(rng, 16, 512), "lo": 64, "hi": _log(rng, 256, 2048),
                 "mix": rng.randrange(1 << 30), "prec": prec}
        if _cost(c) <= 8.8e12:
            return c


# ------------------------------------------------------------------ inputs
class _Gen:
    """Seeded matrices on the GPU, logical rows x cols; every call draws the next ones."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))

    def uniform(self, *shape):
        return torch.rand(*shape, device="cuda", generator=self.g) * 2 - 1

    def wide(self, *shape):
        """N(0, 1) * 2^U(-8, 8): entries of widely different exponents."""
        x = torch.randn(*shape, device="cuda", generator=self.g)
        return x * torch.exp2(torch.rand(*shape, device="cuda", generator=self.g) * 16 - 8)

    def lower(self, n):
        """A well-conditioned lower-triangular matrix (n x n, logical)."""
        d = torch.rand(n, device="cuda", generator=self.g) + 1
        return torch.tril(self.uniform(n, n), -1) / n ** 0.5 + torch.diag(d)


def _col(x):
    """The same logical matrix in column-major storage (a transposed view)."""
    return x.t().contiguous().t()


def _batch_sizes(case):
    r = np.random.RandomState(case["mix"] % (1 << 31))
    return [int(v) for v in np.round(np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), case["count"])))]


def _batch_offsets(ns):
    """Where each n x n instance starts in one flat buffer (512-byte aligned), and the buffer's length."""
    offs, at = [], 0
    for n in ns:
        offs.append(at)
        at += (n * n + 127) // 128 * 128
    return offs, at


def prepare(case, seed):
    g, op = _Gen(seed), case["op"]
    s = {"case": case}
    if op == "tc_syrk":
        s["A"] = g.uniform(case["n"], case["k"])
    elif op == "tc_trsm":
        s["A"] = g.lower(case["n"])
        s["B"] = g.uniform(case["m"], case["n"])
    elif op == "ssyrk":
        n, k = case["n"], case["k"]
        s["A"] = g.uniform(k, n) if case["trans"] == "N" else g.uniform(n, k)
        if case["beta"]:
            s["C0"] = g.uniform(n, n)
        s["C"] = torch.zeros(n, n, device="cuda")
    elif op == "strsm":
        s["A"] = g.lower(case["m"] if case["side"] == "L" else case["n"]).t().contiguous()
        s["B0"] = g.uniform(case["n"], case["m"])
        s["B"] = torch.empty_like(s["B0"])
    elif op in ("syr2k", "trmm", "symm"):
        rows = case["n"] if op == "syr2k" else case["m"]
        lay = _col if case["layout"] == "col" else (lambda x: x)
        s["A"] = lay(g.wide(rows, case["k"] if op == "syr2k" else rows))
        s["B"] = lay(g.wide(rows, case["k"] if op == "syr2k" else case["n"]))
        if case.get("beta"):
            s["C"] = lay(g.wide(rows, case["n"]))
    elif op == "dsyrk":
        n, k = case["n"], case["k"]
        x = torch.randn(k, n, device="cuda", dtype=torch.float64, generator=g.g)
        s["A"] = x * torch.exp(case["phi"] * torch.randn(k, n, device="cuda", dtype=torch.float64, generator=g.g))
        s["C"] = torch.zeros(n, n, device="cuda", dtype=torch.float64)
    else:
        ns = _batch_sizes(case)
        offs, total = _batch_offsets(ns)
        s["A"] = g.uniform(total)
        s["BC0"] = g.uniform(total)
        a_list, bc_list = [], []
        s["BC"] = torch.empty(total, device="cuda")
        for i, (n, o) in enumerate(zip(ns, offs)):
            a = s["A"][o:o + n * n]
            if i % 2:
                a.copy_(g.lower(n).t().contiguous().view(-1))
            else:
                s["BC0"][o:o + n * n] = 0
            a_list.append(a)
            bc_list.append(s["BC"][o:o + n * n])
        s["batch"] = T.Batch([i % 2 for i in range(len(ns))], a_list, bc_list, precision=PREC[case["prec"]])
        s["BC"].copy_(s["BC0"])
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            s["batch"].run()
        torch.cuda.current_stream().wait_stream(side)
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            s["batch"].run()
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "tc_syrk":
        return T.tc_syrk(s["A"], nb=case["nb"])
    if op == "tc_trsm":
        return T.tc_trsm(s["A"], s["B"], nb=case["nb"])
    if op == "ssyrk":
        n, k = case["n"], case["k"]
        if case["beta"]:
            s["C"].copy_(s["C0"])
        T._bind_stream(s["A"])
        T.ssyrk(s["A"], s["C"], n, k, n if case["trans"] == "N" else k, n, 1.0, case["beta"], case["trans"], 256,
                PREC[case["prec"]])
        return s["C"]
    if op == "strsm":
        s["B"].copy_(s["B0"])
        T._bind_stream(s["A"])
        T.strsm(case["side"], s["A"], s["B"], case["m"], case["n"], s["A"].shape[0], case["m"], case["nb"],
                PREC[case["prec"]])
        return s["B"]
    if op == "syr2k":
        return T.syr2k(s["A"], s["B"], precision=PREC[case["prec"]])
    if op == "trmm":
        return T.trmm(s["A"], s["B"], uplo=case["uplo"], precision=PREC[case["prec"]])
    if op == "symm":
        if not case["beta"]:
            return T.symm(s["A"], s["B"], uplo=case["uplo"], precision=PREC[case["prec"]])
        # C is the caller's (a column-major C is updated in place): a copy keeps it for the next call
        return T.symm(s["A"], s["B"], beta=case["beta"], C=s["C"].clone(), uplo=case["uplo"],
                      precision=PREC[case["prec"]])
    if op == "dsyrk":
        n, k = case["n"], case["k"]
        T._bind_stream(s["A"])
        T._check(T.lib.tb_dsyrk_ozaki(b"L", b"N", n, k, 1.0, s["A"].data_ptr(), n, 0.0, s["C"].data_ptr(), n, 0))
        return s["C"]
    s["BC"].copy_(s["BC0"])
    s["graph"].replay()
    return s["BC"]


def work(case):
    """Operands read once, results written once (triangles where only those are used), nominal BLAS3 flops."""
    op = case["op"]
    tri = lambda v: v * (v + 1) / 2.0  # noqa: E731
    if op in ("tc_syrk", "ssyrk", "dsyrk"):
        n, k, e = case["n"], case["k"], 8 if op == "dsyrk" else 4
        out = n * n if op == "tc_syrk" else tri(n) * (2 if case.get("beta") else 1)
        return {"bytes": e * (n * k + out), "flops": 2.0 * tri(n) * k}
    if op in ("tc_trsm", "strsm"):
        m, n = case["m"], case["n"]
        nt = m if case.get("side") == "L" else n
        return {"bytes": 4.0 * (tri(nt) + 2 * m * n), "flops": float(nt) * m * n}
    if op == "syr2k":
        n, k = case["n"], case["k"]
        return {"bytes": 4.0 * (2 * n * k + tri(n)), "flops": 4.0 * tri(n) * k}
    if op == "trmm":
        m, n = case["m"], case["n"]
        return {"bytes": 4.0 * (tri(m) + 2 * m * n), "flops": float(m) * m * n}
    if op == "symm":
        m, n = case["m"], case["n"]
        return {"bytes": 4.0 * (tri(m) + (3 if case["beta"] else 2) * m * n), "flops": 2.0 * m * m * n}
    ns = _batch_sizes(case)
    return {"bytes": 4.0 * sum(n * n + tri(n) if i % 2 == 0 else tri(n) + 2 * n * n for i, n in enumerate(ns)),
            "flops": float(sum(n ** 3 for n in ns))}


def exact(case, seed):
    op = case["op"]
    s = prepare(case, seed)
    if op == "tc_syrk":
        a = s["A"].double()
        return a @ a.t()
    if op == "tc_trsm":
        return torch.linalg.solve_triangular(s["A"].double(), s["B"].double().t(), upper=False).t()
    if op == "ssyrk":
        a = s["A"].double()
        c = a.t() @ a if case["trans"] == "N" else a @ a.t()
        if not case["beta"]:
            return torch.triu(c)  # the storage of a column-major lower triangle; the rest stays zero
        c0 = s["C0"].double()
        return torch.triu(c + case["beta"] * c0) + torch.tril(c0, -1)
    if op == "strsm":
        a, b = s["A"].double(), s["B0"].double()  # storage: A^T (upper), B^T
        if case["side"] == "L":
            return torch.linalg.solve_triangular(a.t(), b.t(), upper=False).t()
        return torch.linalg.solve_triangular(a.t(), b, upper=False)
    if op == "syr2k":
        p = s["A"].double() @ s["B"].double().t()
        return torch.tril(p + p.t())
    if op == "trmm":
        a = s["A"].double()
        return (torch.tril(a) if case["uplo"] == "L" else torch.triu(a)) @ s["B"].double()
    if op == "symm":
        a = s["A"].double()
        a = torch.tril(a) + torch.tril(a, -1).t() if case["uplo"] == "L" else torch.triu(a) + torch.triu(a, 1).t()
        r = a @ s["B"].double()
        return r + case["beta"] * s["C"].double() if case["beta"] else r
    if op == "dsyrk":
        return torch.triu(s["A"].t() @ s["A"])
    ns = _batch_sizes(case)
    out = s["BC0"].double()
    for i, (n, o) in enumerate(zip(ns, _batch_offsets(ns)[0])):
        a = s["A"][o:o + n * n].view(n, n).double()  # storage: A^T
        if i % 2 == 0:
            out[o:o + n * n] = torch.triu(a.t() @ a).reshape(-1)
        else:
            b = out[o:o + n * n].view(n, n)  # storage: B^T; X A^T = B, so A X^T = B^T
            out[o:o + n * n] = torch.linalg.solve_triangular(a.t(), b, upper=False).reshape(-1)
    return out
