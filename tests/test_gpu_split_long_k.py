"""Split products of long K: the correction (hi lo + lo hi) is summed in a
truncating tensor-core accumulator for at most 32 folds of the main sum
(K = 8192), so its error does not grow with K.

The operands leave the correction alone: A's entries are FP16 values, equal in
pairs of rows, B's are +1 and -1 in turn plus a positive part below half an
FP16 ulp. The main products cancel exactly, every correction product has the
same sign, and the result is the correction. Its accumulator truncates at most
twice per 16-deep step, each time by less than 2^-23 of the running sum, so a
stretch of 512 steps is off by at most 2^-22 * 512 / 2 = 6.2e-5 of its sum; the
lo parts' own rounding (2^-12 at random signs) averages out below 1e-5. Summed
over all of K the loss is 2e-4 at K = 32768."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TOL = 2.0 ** -22 * 512 / 2 + 1e-5


@pytest.mark.parametrize("m,n,k", [(100, 130, 40000),      # 64-column tiles, ragged
                                   (640, 2500, 33000),     # single CTAs, 128 x 128
                                   (2304, 2304, 32768),    # CTA pairs, whole stretches
                                   (2304, 2310, 33100)])   # CTA pairs, a short last stretch
def test_correction_error_is_bounded(tblas, m, n, k):
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    a = torch.randint(0, 1024, (k, m), device="cuda", generator=g).float() / 2048 + 0.5  # column-major m x k
    a[1::2] = a[0::2]
    b = torch.rand(n, k, device="cuda", generator=g) * (0.99 * 2.0 ** -12)  # column-major k x n
    b[:, 0::2] += 1
    b[:, 1::2] -= 1
    c = torch.empty(n, m, device="cuda")
    tblas._bind_stream(a)
    tblas.sgemm("N", "N", m, n, k, 1.0, a, m, b, k, 0.0, c, m, tblas.SPLIT)
    tblas.synchronize()
    ref = b.double() @ a.double()
    err = ((c.double() - ref).norm() / ref.norm()).item()
    print(f"{m} x {n} x {k}: correction error {err:.3e}")
    assert err <= TOL


SCRIPT = r"""
import hashlib, sys, torch
sys.path.insert(0, sys.argv[1])
import TensorBLAS as TB
nt, other = 17408, 96
g = torch.Generator(device="cuda")
g.manual_seed(5)
A = torch.triu(torch.rand(nt, nt, device="cuda", generator=g) * 2 - 1) / nt ** 0.5  # column-major lower triangle
A.diagonal().copy_(torch.rand(nt, device="cuda", generator=g) + 1)
for side, m, n in (("L", nt, other), ("R", other, nt)):
    B = torch.rand(n, m, device="cuda", generator=g)
    TB._bind_stream(A)
    TB.strsm(side, A, B, m, n, nt, m, 512, TB.SPLIT)
    TB.synchronize()
    assert torch.isfinite(B).all()
    print(hashlib.sha1(B.cpu().numpy().tobytes()).hexdigest())
"""


def test_persistent_solve_folds_like_the_launches():
    """The first update of an order of 17408 has K = 8704, one stretch and a half fold more."""
    def run(dag):
        out = subprocess.run([sys.executable, "-c", SCRIPT, os.path.join(ROOT, "tensor-blas_b200", "python")],
                             env=dict(os.environ, TB_TRSM_DAG=dag), capture_output=True, text=True, timeout=600)
        assert out.returncode == 0, out.stderr[-2000:]
        return out.stdout.split()
    digests = run("1")
    assert len(digests) == 2 and digests == run("0")
