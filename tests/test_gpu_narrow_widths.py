"""Launches of few tiles run on tiles of 64 columns; the same columns of a
product with so many columns that its tiles of 128 (256) exceed half of the
SMs must be equal bit for bit, and both agree with FP64. One row, one row
block, ragged tiles, a second half without columns, short and long K, a
leading dimension that TMA cannot address."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,bound", [(0, 2e-3), (1, 2e-6)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (100, 63, 40), (128, 64, 1024), (97, 190, 1100), (200, 129, 513)])
@pytest.mark.parametrize("ta,tb,beta,odd", [("N", "N", 0.0, 0), ("N", "T", 0.5, 0), ("T", "N", 0.5, 1),
                                            ("T", "T", 0.0, 1)])
def test_narrow_tiles_match_wider_ones(tblas, prec, bound, m, n, k, ta, tb, beta, odd):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    row_blocks = -(-m // 128)
    wide = 256 * (sms // (2 * row_blocks) + 1)  # columns: over half of the SMs have a tile of 256
    assert -(-n // 128) * row_blocks * 2 <= sms < -(-wide // 256) * row_blocks * 2
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    f = lambda r, c: torch.rand(r, c, device="cuda", generator=g) * 2 - 1  # noqa: E731
    A = f(k, m) if ta == "N" else f(m, k)        # storage of the column-major operand
    B = f(wide, k) if tb == "N" else f(k, wide)
    ldc = (m + 3) // 4 * 4 + odd
    C0 = f(wide, ldc)
    Cw, Cn = C0.clone(), C0[:n].clone()
    lda, ldb = (m if ta == "N" else k), (k if tb == "N" else wide)
    tblas._bind_stream(A)
    tblas.sgemm(ta, tb, m, wide, k, -0.75, A, lda, B, ldb, beta, Cw, ldc, prec)
    tblas.sgemm(ta, tb, m, n, k, -0.75, A, lda, B, ldb, beta, Cn, ldc, prec)
    tblas.synchronize()
    assert torch.equal(Cn[:, :m], Cw[:n, :m])
    assert torch.equal(Cn[:, m:], C0[:n, m:])    # the padding between columns is not written
    ref = beta * C0[:, :m].double() - 0.75 * ((B if tb == "N" else B.T).double() @ (A if ta == "N" else A.T).double())
    err = ((Cw[:, :m].double() - ref).norm() / ref.norm()).item()
    assert err <= bound
