"""tb_synchronize from more threads than there are page-locked words for the
error codes (64): the others copy the codes the blocking way, and none reports
a fault."""
import ctypes
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_synchronize_from_many_threads(tblas):
    n, k, threads, rounds = 200, 96, 100, 20
    dev = torch.cuda.current_device()
    A = [torch.rand(k, n, device="cuda") for _ in range(threads)]  # column-major n x k
    C = [torch.zeros(n, n, device="cuda") for _ in range(threads)]
    streams = [torch.cuda.Stream() for _ in range(4)]  # shared, so that calls wait together
    torch.cuda.synchronize()
    start, faults = threading.Barrier(threads), []

    def work(i):
        torch.cuda.set_device(dev)
        tblas.lib.tb_set_stream(ctypes.c_void_p(streams[i % 4].cuda_stream))
        start.wait()
        for _ in range(rounds):
            st = tblas.lib.tb_synchronize()
            if st != 0:
                faults.append((i, st))

    tblas.lib.tb_set_stream(ctypes.c_void_p(streams[0].cuda_stream))
    for a, c in zip(A, C):
        tblas.ssyrk(a, c, n, k, n, n, precision=tblas.SPLIT)
    pool = [threading.Thread(target=work, args=(i,)) for i in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join(120)
    assert not any(t.is_alive() for t in pool) and not faults
    tblas.lib.tb_set_stream(ctypes.c_void_p(streams[0].cuda_stream))
    tblas.synchronize()
    for a, c in zip(A, C):
        ref = torch.triu(a.double().T @ a.double())  # the column-major lower triangle
        assert ((c.double() - ref).norm() / ref.norm()).item() < 2e-6
    tblas._bind_stream(A[0])
