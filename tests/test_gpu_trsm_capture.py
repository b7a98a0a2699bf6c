"""A solve captured in a CUDA graph (plain launches) against the same call
outside a capture (dependent launches, set-up of a launch overlapping the one
before): the same bits, from right-hand sides put back between the replays."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,m,n,nb,prec", [("L", 1100, 130, 128, 1), ("R", 257, 2304, 256, 0), ("L", 2560, 96, 512, 0)])
def test_captured_solve_matches(tblas, side, m, n, nb, prec):
    nt = m if side == "L" else n
    g = torch.Generator(device="cuda")
    g.manual_seed(nt)
    A = torch.triu(torch.rand(nt, nt, device="cuda", generator=g) * 2 - 1, 1) / nt ** 0.5  # column-major lower triangle
    A.diagonal().copy_(torch.rand(nt, device="cuda", generator=g) + 1)
    B0 = torch.rand(n, m, device="cuda", generator=g) * 2 - 1
    B, want = B0.clone(), B0.clone()
    tblas._bind_stream(A)
    tblas.strsm(side, A, want, m, n, nt, m, nb, prec)
    tblas.synchronize()
    side_stream = torch.cuda.Stream()
    side_stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side_stream):
        tblas._bind_stream(A)
        tblas.strsm(side, A, B, m, n, nt, m, nb, prec)  # warm on this stream
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side_stream):
        tblas._bind_stream(A)
        tblas.strsm(side, A, B, m, n, nt, m, nb, prec)
    for _ in range(2):
        B.copy_(B0)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(B, want)
    tblas._bind_stream(A)
    tblas.synchronize()
