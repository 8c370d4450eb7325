"""Two host threads whose kernels both give up on a wait (no operand loads, as in
the single-threaded test): each thread's call reports it, and the calls after
them are clean.
"""
import threading

import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu

MWBLAS_ERR_TIMEOUT = -4


def test_both_threads_report(gpu, oracle, rng):
    import torch
    m, n, k = 256, 512, 1024
    A, B, C0 = mwb.dd_matrix(rng, m, k), mwb.dd_matrix(rng, k, n), mwb.dd_matrix(rng, m, n)
    al, be = mwb.random_dd(rng, ()), mwb.random_dd(rng, ())
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    dC = [torch.from_numpy(C0).cuda() for _ in range(2)]

    def together():
        codes, gate = [None, None], threading.Barrier(2)

        def body(i):
            gate.wait()
            gpu.mgemm("N", "N", m, n, k, al, dA.data_ptr(), m, dB.data_ptr(), k, be, dC[i].data_ptr(), m,
                      engine="ozaki")
            codes[i] = gpu.last_error()[0]

        threads = [threading.Thread(target=body, args=(i,)) for i in range(2)]
        [t.start() for t in threads]
        [t.join() for t in threads]
        return codes

    gpu.lib.mwblas_set_wait_limit_ns(20_000_000)   # 20 ms
    try:
        for _ in range(3):
            gpu.lib.mwblas_debug_lose_operand_loads(2)
            assert together() == [MWBLAS_ERR_TIMEOUT] * 2
    finally:
        gpu.lib.mwblas_debug_lose_operand_loads(0)
        gpu.lib.mwblas_set_wait_limit_ns(0)
    for c in dC:
        c.copy_(torch.from_numpy(C0))
    torch.cuda.synchronize()
    assert together() == [0, 0]
    want = oracle.qgemm("N", "N", m, n, k, al, A, m, B, k, be, C0.copy(), m)
    op = orc.dd_abs(al) * k * orc.dd_absmax(A) * orc.dd_absmax(B) + orc.dd_abs(be) * orc.dd_absmax(C0)
    for c in dC:
        assert orc.normwise_error(c.cpu().numpy(), want, op) <= max(10, 4 * k) * orc.EPS_DD
