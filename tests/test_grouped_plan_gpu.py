"""The grouped GEMM's kept plan after a call that failed half way (an injected
allocation failure): the layout before it is prepared anew, not taken for the
one whose buffers are gone or rewritten. Each case runs on a thread of its own,
whose plan starts empty.
"""
import threading

import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu

MWBLAS_ERR_ALLOC = -2


class Batch:
    def __init__(self, rng, shapes):
        import torch
        self.inst = [(m, n, k, mwb.dd_matrix(rng, m, k), mwb.dd_matrix(rng, k, n), mwb.dd_matrix(rng, m, n))
                     for m, n, k in shapes]
        self.dev = [[torch.from_numpy(x).cuda() for x in t[3:]] for t in self.inst]
        self.al, self.be = mwb.random_dd(rng, ()), mwb.random_dd(rng, ())

    def call(self, gpu):
        import torch
        for d, t in zip(self.dev, self.inst):
            d[2].copy_(torch.from_numpy(t[5]))
        torch.cuda.synchronize()
        col = lambda i: [t[i] for t in self.inst]
        ptr = lambda i: [d[i].data_ptr() for d in self.dev]
        count = len(self.inst)
        return gpu.mgemm_grouped(["N"] * count, ["N"] * count, col(0), col(1), col(2), [self.al] * count, ptr(0),
                                 col(0), ptr(1), col(2), [self.be] * count, ptr(2), col(0))

    def check(self, oracle):
        for (m, n, k, A, B, C0), d in zip(self.inst, self.dev):
            want = oracle.qgemm("N", "N", m, n, k, self.al, A, m, B, k, self.be, C0.copy(), m)
            op = orc.dd_abs(self.al) * k * orc.dd_absmax(A) * orc.dd_absmax(B)
            op += orc.dd_abs(self.be) * orc.dd_absmax(C0)
            assert orc.normwise_error(d[2].cpu().numpy(), want, op) <= 16 * orc.EPS_DD


SMALL = [(20, 30, 40), (9, 17, 70)]
LARGE = [(60, 50, 300), (33, 90, 64), (100, 100, 90)]
TENSOR = [(130, 140, 64)]


@pytest.mark.parametrize("first,second,allowed", [(SMALL, LARGE, 0), (SMALL + TENSOR, LARGE + TENSOR * 3, 0),
                                                  (SMALL + TENSOR, LARGE + TENSOR * 3, 1)])
def test_layout_before_a_failed_call(gpu, oracle, rng, first, second, allowed):
    x, y, failures = Batch(rng, first), Batch(rng, second), []

    def body():
        try:
            assert x.call(gpu) == 0, gpu.last_error()
            x.check(oracle)
            gpu.lib.mwblas_debug_fail_alloc_after(allowed)
            assert y.call(gpu) == MWBLAS_ERR_ALLOC, gpu.last_error()
            gpu.lib.mwblas_debug_fail_alloc_after(-1)
            for b in (x, x, y, x):
                assert b.call(gpu) == 0, gpu.last_error()
                b.check(oracle)
        except BaseException as e:
            failures.append(e)
        finally:
            gpu.lib.mwblas_debug_fail_alloc_after(-1)

    t = threading.Thread(target=body)
    t.start()
    t.join()
    if failures:
        raise failures[0]
