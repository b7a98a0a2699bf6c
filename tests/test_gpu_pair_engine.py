"""256 x 256 CTA-pair tiles of the split and FP8 forms against the single-CTA
128 x 128 tiles (TB_GEMM_PAIR=0, for split also TB_GEMM_PAIR_SPLIT=0), at sizes
that the dispatch sends to pairs: the library's launch counters show which
kernel ran, the results must be bit-identical (but for the split upper TRMM,
whose pair tiles fold at other K blocks) and agree with FP64. A launch takes pairs when its waves of pair
tiles, 1.45 single-tile times each, are fewer than those of single tiles; on
either side of that line the counters must show it. The engine is read once
per process, so each setting runs in its own subprocess."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SPLIT, FP8 = 1, 2
BOUND = {SPLIT: 2e-6, FP8: 8e-2}

SCRIPT = r"""
import ctypes, hashlib, sys, numpy as np, torch
sys.path.insert(0, sys.argv[1])
import TensorBLAS as TB
g = torch.Generator(device="cuda")
g.manual_seed(23)
f = lambda r, c: torch.rand(r, c, device="cuda", generator=g) * 2 - 1

def pair_launches(call):
    TB.lib.tb_profile_begin()
    out = call()
    TB.synchronize()
    ms, flops, n = ctypes.c_double(), ctypes.c_double(), ctypes.c_long()
    TB._check(TB.lib.tb_profile_end(ctypes.byref(ms), ctypes.byref(flops), ctypes.byref(n)))
    TB._check(TB.lib.tb_profile_kernel(1, None, None, None, ctypes.byref(n)))
    return out, n.value

def run(op, m, n, k, prec, beta):
    if op == "syrk":
        A, C = f(n, k), f(n, n)
        X, pairs = pair_launches(lambda: TB.syrk(A, beta=beta, C=C, precision=prec))
        ref = torch.tril(A.double() @ A.double().T + beta * C.double()) + torch.triu(C.double(), 1)
    elif op == "syrkT":  # C = A^T A of a column-major k x n A, the column-major lower triangle
        A = f(n, k)
        X = torch.zeros(n, n, device="cuda")
        TB._bind_stream(A)
        _, pairs = pair_launches(lambda: TB.ssyrk(A, X, n, k, k, n, 1.0, 0.0, "T", 256, prec))
        ref = torch.triu(A.double() @ A.double().T)
    elif op == "syr2k":
        A, B = f(n, k), f(n, k)
        X, pairs = pair_launches(lambda: TB.syr2k(A, B, precision=prec))
        P = A.double() @ B.double().T
        ref = torch.tril(P + P.T)
    elif op == "symm":
        A, B, C = f(m, m), f(m, n), f(m, n)
        X, pairs = pair_launches(lambda: TB.symm(A, B, beta=beta, C=C, precision=prec))
        S = torch.tril(A.double())
        ref = (S + torch.tril(S, -1).T) @ B.double() + beta * C.double()
    elif op in ("trmm", "trmm_u"):
        A, B = f(m, m), f(m, n)
        X, pairs = pair_launches(lambda: TB.trmm(A, B, uplo="U" if op == "trmm_u" else "L", precision=prec))
        ref = (torch.triu(A) if op == "trmm_u" else torch.tril(A)).double() @ B.double()
    else:  # gemmNN, gemmTN, gemmNT, gemmTT: column-major storage of the operands
        ta, tb = op[4], op[5]
        A, B = f(k, m) if ta == "N" else f(m, k), f(n, k) if tb == "N" else f(k, n)
        X = f(n, m)
        ref = beta * X.double() + ((B if tb == "N" else B.T).double() @ (A if ta == "N" else A.T).double())
        TB._bind_stream(A)
        _, pairs = pair_launches(lambda: TB.sgemm(ta, tb, m, n, k, 1.0, A, m if ta == "N" else k, B,
                                                  k if tb == "N" else n, beta, X, m, prec))
    err = ((X.double() - ref).norm() / ref.norm()).item()
    return hashlib.sha1(X.contiguous().cpu().numpy().tobytes()).hexdigest(), pairs, err

for case in eval(sys.argv[2]):
    print(*run(*case))
"""


def _run(pair, cases, switch="TB_GEMM_PAIR"):
    out = subprocess.run([sys.executable, "-c", SCRIPT, os.path.join(ROOT, "tensor-blas_b200", "python"), repr(cases)],
                         env=dict(os.environ, **{switch: pair}), capture_output=True, text=True, timeout=900)
    assert out.returncode == 0, out.stderr[-2000:]
    return [(d, int(p), float(e)) for d, p, e in (line.split() for line in out.stdout.splitlines())]


def _check_pairs(cases, switch="TB_GEMM_PAIR"):
    for case, pair, single in zip(cases, _run("1", cases, switch), _run("0", cases, switch)):
        print(case, pair, single)
        assert pair[1] == 1 and single[1] == 0, case  # the two engines ran
        assert pair[2] <= BOUND[case[4]] and single[2] <= BOUND[case[4]], case
        yield case, pair[0] == single[0]


def test_fp8_pair_tiles_match_single_cta_tiles():
    # ragged rows, columns and K; a pair whose second CTA has no rows; tiles across the triangle
    cases = [("syrk", 0, 2432, 300, FP8, 0.0), ("syrk", 0, 2563, 1037, FP8, 0.5), ("syr2k", 0, 2500, 260, FP8, 0.0),
             ("symm", 2100, 1700, 0, FP8, 0.5), ("trmm", 2050, 1930, 0, FP8, 0.0), ("trmm_u", 1999, 2301, 0, FP8, 0.0),
             ("gemmTN", 2000, 2100, 129, FP8, 0.5)]
    assert all(same for _, same in _check_pairs(cases))


@pytest.mark.parametrize("switch", ["TB_GEMM_PAIR", "TB_GEMM_PAIR_SPLIT"])
def test_split_pair_tiles_match_single_cta_tiles(switch):
    cases = [("syrk", 0, 2304, 2048, SPLIT, 0.0), ("syrk", 0, 2500, 1100, SPLIT, 0.5),
             ("syrkT", 0, 2432, 1536, SPLIT, 0.0), ("syr2k", 0, 2304, 1025, SPLIT, 0.0),
             ("trmm", 2048, 2048, 0, SPLIT, 0.0), ("trmm_u", 2048, 1990, 0, SPLIT, 0.0),
             ("symm", 2048, 2048, 0, SPLIT, 0.5), ("gemmNN", 2048, 2048, 1536, SPLIT, 0.0),
             ("gemmTN", 1990, 2048, 1100, SPLIT, 0.5), ("gemmNT", 2048, 1801, 1537, SPLIT, 0.0),
             ("gemmTT", 2002, 2001, 1100, SPLIT, 0.5)]
    differ = [case for case, same in _check_pairs(cases, switch) if not same]
    assert [case[0] for case in differ] in ([], ["trmm_u"]), differ


def test_fp8_engine_follows_the_waves():
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    up = lambda a, b: -(-a // b)  # noqa: E731
    sizes = [(512, 512), (1024, 1024), (1536, 1536), (1792, 1792), (2048, 2048), (2304, 2304), (1100, 8192),
             (640, 16384), (4096, 4096)]
    cases = [("gemmNN", m, n, 200, FP8, 0.0) for m, n in sizes]
    for (m, n), (_, pairs, err) in zip(sizes, _run("1", cases)):
        singles = up(up(m, 128) * up(n, 128), sms)
        fewer = up(up(m, 256) * up(n, 256), sms // 2) * 1.45 <= singles
        assert (pairs == 1) == fewer, (m, n, pairs)
        assert err <= BOUND[FP8], (m, n)
