"""Grouped products whose operands' magnitudes change along k: every K split of the
limb tiles scales its lines by its own largest entries, as the square tiles do, so
entries that are small against their line but not against their split keep their
bits. Against the binary128 oracle, to 16 units of 2^-104 of k times the sum over
the splits (512 deep here) of the splits' own maxima.
"""
import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu

SPLIT = 512


@pytest.mark.parametrize("tile", [16, 32])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "T")])
@pytest.mark.parametrize("m,n", [(8, 16), (33, 20), (64, 64), (128, 17)])
def test_graded_along_k(gpu, oracle, rng, m, n, ta, tb, tile):
    import torch
    k = 2 * SPLIT
    A, B, C0 = mwb.random_dd(rng, (k, m)), mwb.random_dd(rng, (n, k)), np.zeros((n, m, 2))
    A[SPLIT:] *= 2.0 ** -80                     # large against small, then small against large
    B[:, :SPLIT] *= 2.0 ** -80
    absmax = lambda v: np.abs(v[..., 0]).max()
    scale = sum(absmax(A[q:q + SPLIT]) * absmax(B[:, q:q + SPLIT]) for q in (0, SPLIT))
    if ta == "T":
        A = np.ascontiguousarray(A.transpose(1, 0, 2))
    if tb == "T":
        B = np.ascontiguousarray(B.transpose(1, 0, 2))
    one, zero = np.array([1.0, 0.0]), np.zeros(2)
    want = oracle.qgemm(ta, tb, m, n, k, one, A, A.shape[1], B, B.shape[1], zero, C0.copy(), m)
    d = [torch.from_numpy(v).cuda() for v in (A, B, C0)]
    prev = gpu.lib.mwblas_set_grouped_tile(tile)
    try:
        assert gpu.mgemm_grouped([ta], [tb], [m], [n], [k], [one], [d[0].data_ptr()], [A.shape[1]], [d[1].data_ptr()],
                                 [B.shape[1]], [zero], [d[2].data_ptr()], [m]) == 0, gpu.last_error()
    finally:
        gpu.lib.mwblas_set_grouped_tile(prev)
    got = d[2].cpu().numpy()
    err = np.abs((got[..., 0] - want[..., 0]) + (got[..., 1] - want[..., 1])).max()
    assert err <= 16 * orc.EPS_DD * k * scale, err / (orc.EPS_DD * k * scale)
