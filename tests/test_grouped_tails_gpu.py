"""Grouped products whose k ends before their class's (64, 128, 256, 512, ..): the
columns between are zeroed, whatever an earlier batch of another layout left in
the residue planes. Against the binary128 oracle within 4k 2^-104 |A| |B|."""
import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu


def run(gpu, inst):
    import torch
    dev = [[torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in t[3:]] for t in inst]
    col = lambda i: [t[i] for t in inst]
    one, zero = [np.array([1.0, 0.0])] * len(inst), [np.zeros(2)] * len(inst)
    rc = gpu.mgemm_grouped(["N"] * len(inst), ["N"] * len(inst), col(0), col(1), col(2), one,
                           [d[0].data_ptr() for d in dev], col(0), [d[1].data_ptr() for d in dev], col(2), zero,
                           [d[2].data_ptr() for d in dev], col(0))
    assert rc == 0, gpu.last_error()
    return [d[2].cpu().numpy() for d in dev]


@pytest.mark.parametrize("ks", [(65, 96, 97, 128), (129, 160, 255, 256), (300, 480, 513, 1000)])
def test_tails(gpu, oracle, rng, ks):
    prev = gpu.lib.mwblas_set_grouped_tensor_min(64)
    try:
        make = lambda m, n, k: (m, n, k, mwb.dd_matrix(rng, m, k), mwb.dd_matrix(rng, k, n), np.zeros((n, m, 2)))
        run(gpu, [make(300, 290, 1024)] + [make(260, 130, k) for k in (511, 512, 128)])   # leaves its residues behind
        inst = [make(130 + i, 65 + i, k) for i, k in enumerate(ks)]
        for (m, n, k, A, B, C), got in zip(inst, run(gpu, inst)):
            want = oracle.qgemm("N", "N", m, n, k, np.array([1.0, 0.0]), A, m, B, k, np.zeros(2), C.copy(), m)
            err = orc.normwise_error(got, want, k * orc.dd_absmax(A) * orc.dd_absmax(B))
            assert err <= 4 * k * orc.EPS_DD, (m, n, k, err)
    finally:
        gpu.lib.mwblas_set_grouped_tensor_min(prev)
