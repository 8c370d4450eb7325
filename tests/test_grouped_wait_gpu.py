"""The bounded-wait failure path of the grouped limb tiles, on the GPU: a launch
that issues no operand copies (the library's injection hook; nothing is in
flight) gives up at its wait limit, every warp leaves, split tiles included,
and the call reports MWBLAS_ERR_TIMEOUT. The same batch is then correct.
"""
import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu

MWBLAS_ERR_TIMEOUT = -4


@pytest.mark.parametrize("shapes", [[(8, 16, 64)], [(16, 16, 4096)], [(9, 17, 5000), (40, 40, 70), (5, 6, 9000)]])
def test_lost_copies_report_timeout(gpu, oracle, rng, shapes):
    import torch
    al, be = mwb.random_dd(rng, ()), mwb.random_dd(rng, ())
    inst = [(m, n, k, mwb.dd_matrix(rng, m, k), mwb.dd_matrix(rng, k, n), mwb.dd_matrix(rng, m, n))
            for m, n, k in shapes]
    dev = [[torch.from_numpy(x).cuda() for x in t[3:]] for t in inst]
    col = lambda i: [t[i] for t in inst]
    count = len(inst)

    def call():
        return gpu.mgemm_grouped(["N"] * count, ["N"] * count, col(0), col(1), col(2), [al] * count,
                                 [d[0].data_ptr() for d in dev], col(0), [d[1].data_ptr() for d in dev], col(2),
                                 [be] * count, [d[2].data_ptr() for d in dev], col(0))

    prev = gpu.lib.mwblas_set_grouped_tile(16)
    try:
        gpu.lib.mwblas_set_wait_limit_ns(20_000_000)   # 20 ms
        gpu.lib.mwblas_debug_lose_operand_loads(1)
        assert call() == MWBLAS_ERR_TIMEOUT, gpu.last_error()
        assert "gave up" in gpu.last_error()[1]
        gpu.lib.mwblas_debug_lose_operand_loads(0)
        gpu.lib.mwblas_set_wait_limit_ns(0)
        for d, t in zip(dev, inst):
            d[2].copy_(torch.from_numpy(t[5]))
        torch.cuda.synchronize()
        for _ in range(2):   # a new graph, then its replay
            for d, t in zip(dev, inst):
                d[2].copy_(torch.from_numpy(t[5]))
            torch.cuda.synchronize()
            assert call() == 0, gpu.last_error()
    finally:
        gpu.lib.mwblas_debug_lose_operand_loads(0)
        gpu.lib.mwblas_set_wait_limit_ns(0)
        gpu.lib.mwblas_set_grouped_tile(prev)
    for (m, n, k, A, B, C0), d in zip(inst, dev):
        want = oracle.qgemm("N", "N", m, n, k, al, A, m, B, k, be, C0.copy(), m)
        op = orc.dd_abs(al) * k * orc.dd_absmax(A) * orc.dd_absmax(B) + orc.dd_abs(be) * orc.dd_absmax(C0)
        err = orc.normwise_error(d[2].cpu().numpy(), want, op)
        assert err <= 16 * orc.EPS_DD
