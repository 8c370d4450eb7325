"""Products at every width that mwblas_set_ozaki_bits takes near its upper end, on
both residue paths, up to the most moduli there are (32), against the binary128
oracle: 8 units of 2^-104 of |alpha| k |A| |B| + |beta C|.
"""
import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tc", [1, 0])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("bits", [106, 116, 117, 118, 119, 120])
def test_bits(gpu, oracle, rng, bits, cplx, tc):
    m, n, k = 130, 70, 200
    A, B, C0 = (mwb.dd_matrix(rng, *s, cplx_=cplx) for s in ((m, k), (k, n), (m, n)))
    one = lambda: mwb.random_dd(rng, ()) + np.array([1.25, 0.0])
    al, be = (np.stack([one(), one()]), np.stack([one(), one()])) if cplx else (one(), one())
    want, got = C0.copy(), C0.copy()
    prev, pb = gpu.lib.mwblas_set_gemm_engine(2), gpu.lib.mwblas_set_ozaki_bits(bits)
    pt = gpu.lib.mwblas_set_residue_tc(tc)
    try:
        (oracle.qwgemm if cplx else oracle.qgemm)("N", "N", m, n, k, al, A, m, B, k, be, want, m)
        (gpu.wgemm if cplx else gpu.mgemm)("N", "N", m, n, k, al, A, m, B, k, be, got, m)
        assert gpu.last_error()[0] == 0, gpu.last_error()
    finally:
        gpu.lib.mwblas_set_gemm_engine(prev)
        gpu.lib.mwblas_set_ozaki_bits(pb)
        gpu.lib.mwblas_set_residue_tc(pt)
    op = np.abs(al).sum() * k * orc.dd_absmax(A) * orc.dd_absmax(B) + np.abs(be).sum() * orc.dd_absmax(C0)
    err = np.abs((got[..., 0] - want[..., 0]) + (got[..., 1] - want[..., 1])).max()
    assert err <= 8 * orc.EPS_DD * op, err / op / orc.EPS_DD


def test_most_moduli(gpu, oracle, rng):
    """120 bits and a long k need 32 moduli; the sums cover two steps of 16 whole."""
    m, n, k = 40, 33, 40000
    A, B, C0 = (mwb.dd_matrix(rng, *s) for s in ((m, k), (k, n), (m, n)))
    one = np.array([1.0, 0.0])
    want = oracle.qgemm("N", "N", m, n, k, one, A, m, B, k, one, C0.copy(), m)
    got = C0.copy()
    prev = gpu.lib.mwblas_set_ozaki_bits(120)
    try:
        gpu.mgemm("N", "N", m, n, k, one, A, m, B, k, one, got, m, engine="ozaki")
        assert gpu.last_error()[0] == 0 and gpu.lib.mwblas_last_ozaki_moduli() == 32
    finally:
        gpu.lib.mwblas_set_ozaki_bits(prev)
    op = k * orc.dd_absmax(A) * orc.dd_absmax(B) + orc.dd_absmax(C0)
    assert orc.normwise_error(got, want, op) <= 8 * orc.EPS_DD
