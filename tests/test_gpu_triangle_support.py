"""An infinity in B reaches the 128 rows (left side) or columns (right side) of
C = op(A) B / B op(A) that its block of the triangle touches and those beyond,
but none of the blocks that the triangle does not connect it with: those equal,
bit for bit, the product of the same B with a finite value in that place. FP8
on CTA-pair tiles, whose K range spans four 128 x 128 parts."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

FP8 = 2


@pytest.mark.parametrize("na,other", [(2050, 1930), (1920, 2048)])
@pytest.mark.parametrize("side", ["L", "R"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("trans", ["N", "T"])
def test_infinity_stays_in_its_blocks(tblas, na, other, side, uplo, trans):
    g = torch.Generator(device="cuda")
    g.manual_seed(31)
    m, n = (na, other) if side == "L" else (other, na)
    A = torch.rand(na, na, device="cuda", generator=g) * 2 - 1
    B = torch.rand(n, m, device="cuda", generator=g) * 2 - 1  # column-major m x n
    op_lower = (uplo == "L") == (trans == "N")
    # the index of B that meets A's order: rows >= p of C see it when op(A) is
    # lower (left), columns <= p (right); p in the half of a 256 block that the
    # other half must not see
    sees_above = (side == "L") == op_lower
    p = 700 if sees_above else 600
    if side == "L":
        B[5, p] = 0.5
    else:
        B[p, 5] = 0.5

    def trmm():
        C = torch.empty(n, m, device="cuda")
        f, v = ctypes.c_char, ctypes.c_long
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        tblas._bind_stream(A)
        tblas._check(tblas.lib.tb_strmm_ex(f(side.encode()), f(uplo.encode()), f(trans.encode()), f(b"N"), v(m), v(n),
                                           ctypes.c_float(1.0), ptr(A), v(na), ptr(B), v(m), ptr(C), v(m), FP8))
        tblas.synchronize()
        return C if side == "R" else C.t()  # along A's order first

    want = trmm()
    if side == "L":
        B[5, p] = float("inf")
    else:
        B[p, 5] = float("inf")
    got = trmm()
    keep = slice(0, 640) if sees_above else slice(640, na)
    # the infinity changes its block's scale: that block's columns (rows) are finite, not equal
    assert torch.equal(got[keep, 128:], want[keep, 128:])
    assert torch.isfinite(got[keep]).all()
    assert not torch.isfinite(got[p]).all()
