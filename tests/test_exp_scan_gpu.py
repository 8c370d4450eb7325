"""The exponent scan of both operands: one entry 2^60 above the others at the
places where a thread's batches, remainders and column pieces meet. A bound that
missed it would leave the product without any right digit; the oracle's result
is met within max(10, 4k) 2^-104 |A| |B|."""
import numpy as np
import pytest

from conftest import mwb, orc
from test_ozaki_gpu import op_norm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T")])
@pytest.mark.parametrize("k,at", [(1, 0), (7, 6), (9, 8), (16, 15), (255, 254), (257, 256), (300, 287)])
def test_scan_finds_the_largest(gpu, oracle, rng, ta, tb, k, at):
    m, n = 257, 35
    A = mwb.dd_matrix(rng, m if ta == "N" else k, k if ta == "N" else m)
    B = mwb.dd_matrix(rng, k if tb == "N" else n, n if tb == "N" else k)
    a, b = (A if ta == "T" else A.transpose(1, 0, 2)), (B if tb == "N" else B.transpose(1, 0, 2))
    a[m - 1, at] *= 2.0 ** 60          # [row of op(A), depth] and [column of op(B), depth]
    b[n - 1, at] *= 2.0 ** 60
    al, be = np.array([1.0, 0.0]), np.zeros(2)
    lda, ldb = (m if ta == "N" else k), (k if tb == "N" else n)
    want = oracle.qgemm(ta, tb, m, n, k, al, A, lda, B, ldb, be, np.zeros((n, m, 2)), m)
    got = np.zeros((n, m, 2))
    gpu.mgemm(ta, tb, m, n, k, al, A, lda, B, ldb, be, got, m, engine="ozaki")
    assert gpu.last_error()[0] == 0, gpu.last_error()
    err = orc.normwise_error(got, want, op_norm(al, k, A, B, be, got * 0))
    assert err <= max(10, 4 * k) * orc.EPS_DD, err
    # without the spike's row and column nothing is above the plain sizes
    err = orc.normwise_error(got[:n - 1, :m - 1], want[:n - 1, :m - 1], k)
    assert err <= max(10, 4 * k) * orc.EPS_DD, err
