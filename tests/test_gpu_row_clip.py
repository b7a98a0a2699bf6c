"""Rows of C past M belong to the caller (padding, or the matrix that C is a
block of): TMA stores clip at 16 bytes, so a C whose M is no multiple of 4
must not let the store of its last row tile reach them. Every engine: short
and long K, single CTAs and CTA pairs, per-element and staged tiles, FP8."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("m,n,k,ldc", [(1, 1, 1, 4), (130, 65, 300, 132), (1001, 700, 300, 1004),
                                       (1001, 700, 2000, 1012), (1002, 4096, 1500, 1004), (515, 516, 1100, 516)])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_rows_past_m_are_not_written(tblas, prec, m, n, k, ldc, beta):
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    A = torch.rand(k, m, device="cuda", generator=g)
    B = torch.rand(n, k, device="cuda", generator=g)
    C0 = torch.rand(n, ldc, device="cuda", generator=g)
    C = C0.clone()
    tblas._bind_stream(A)
    tblas.sgemm("N", "N", m, n, k, 1.0, A, m, B, k, beta, C, ldc, prec)
    tblas.synchronize()
    assert torch.equal(C[:, m:], C0[:, m:])
    ref = (B.double() @ A.double()) + beta * C0[:, :m].double()
    err = ((C[:, :m].double() - ref).norm() / ref.norm()).item()
    assert err <= (8e-2 if prec == 2 else 2e-3), err
