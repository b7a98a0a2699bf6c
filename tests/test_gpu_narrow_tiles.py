"""Launches that leave more than half of the SMs idle run on tiles of 64
columns. Every element's products, accumulation order and folds are those of
the wider tiles, so the columns of a small product must equal, bit for bit,
the same columns of a product wide enough for 128- and 256-column tiles. The
sizes leave ragged tiles, a second half without columns, short and long K (one
and several fold rounds) and a leading dimension TMA cannot address."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (100, 63, 40), (130, 65, 300), (256, 129, 513), (257, 200, 1100),
                                   (512, 64, 2100)])
@pytest.mark.parametrize("ta,tb,beta,odd", [("N", "N", 0.0, 0), ("N", "T", 0.5, 0), ("T", "N", 0.5, 1),
                                            ("T", "T", 0.0, 1)])
def test_narrow_tiles_match_wide_ones(tblas, prec, m, n, k, ta, tb, beta, odd):
    wide = 6144
    g = np.random.Generator(np.random.PCG64(5))
    f = lambda r, c: torch.from_numpy(g.uniform(-1, 1, (r, c)).astype(np.float32)).cuda()  # noqa: E731
    A = f(k, m) if ta == "N" else f(m, k)              # storage of the column-major operand
    B = f(wide, k) if tb == "N" else f(k, wide)        # column-major k x wide / wide x k
    ldc = (m + 3) // 4 * 4 + odd
    C0 = f(wide, ldc)
    Cw, Cn = C0.clone(), C0[:n].clone()
    lda, ldb = (m if ta == "N" else k), (k if tb == "N" else wide)
    tblas._bind_stream(A)
    tblas.sgemm(ta, tb, m, wide, k, -0.75, A, lda, B, ldb, beta, Cw, ldc, prec)
    tblas.sgemm(ta, tb, m, n, k, -0.75, A, lda, B, ldb, beta, Cn, ldc, prec)
    tblas.synchronize()
    assert torch.equal(Cn[:, :m], Cw[:n, :m])
    assert torch.equal(Cn[:, m:], C0[:n, m:])          # the padding between columns is not written
