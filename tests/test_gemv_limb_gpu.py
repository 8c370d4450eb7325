"""mgemv_ around the edges of its tensor-core kernel, against the binary128
oracle: 32 outputs per warp, groups of 4, windows of 32 reduction indices,
chunks of whole windows, and the operands that leave its straight-line path.

Every product is exact in 2^-110 of its output's largest one and the update of
y rounds once, so each output is good to a few units of 2^-104 of
|alpha| sum |A x| + |beta y| (16 allowed, as the oracle's sum of the same
length and the double-double alpha and beta products add theirs).
"""
import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu


def operands(rng, m, n, lx, kind):
    A, x = mwb.dd_matrix(rng, m, n), mwb.random_dd(rng, (lx,))
    if kind == "zeros":                        # sparse operands, whole zero groups among them
        A[rng.random(A.shape[:2]) < 0.7] = 0.0
        x[rng.random(lx) < 0.3] = 0.0
        x[: lx // 2] = 0.0
    elif kind == "fp64":                       # lo = 0, both signs of zero
        A[..., 1] = 0.0 * np.sign(A[..., 0])
        x[:, 1] = 0.0
    elif kind == "spread":                     # growing blocks, long alignments
        A *= 2.0 ** rng.integers(-90, 90, A.shape[:2])[..., None]
        x *= 2.0 ** np.sort(rng.integers(-60, 60, lx))[:, None]
    elif kind == "far_lo":                     # lo far below hi, and subnormal
        A[..., 1] *= 2.0 ** -rng.integers(0, 60, A.shape[:2]).astype(float)
        A *= 2.0 ** 900                        # products and sums stay in the normal range
        x *= 2.0 ** -990
        x[:, 1] = np.where(rng.random(lx) < 0.5, 5e-324, 0.0)
    elif kind == "loose":                      # not normalised: lo up to hi's size
        A[..., 1] = A[..., 0] * rng.uniform(-0.4, 0.4, A.shape[:2])
    return A, x


@pytest.mark.parametrize("kind", ["plain", "zeros", "fp64", "spread", "far_lo", "loose"])
@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("outs,red", [(1, 1), (1, 5000), (31, 3), (32, 4), (33, 65), (257, 31), (300, 33), (5, 2113),
                                      (1030, 97)])
def test_gemv_edges(gpu, oracle, rng, outs, red, trans, kind):
    m, n = (outs, red) if trans == "N" else (red, outs)
    A, x = operands(rng, m, n, red, kind)
    y0 = mwb.random_dd(rng, (outs,))
    al, be = mwb.random_dd(rng, ()) + np.array([1.5, 0.0]), mwb.random_dd(rng, ())
    want, got = y0.copy(), y0.copy()
    oracle.qgemv(trans, m, n, al, A, m, x, 1, be, want, 1)
    gpu.mgemv(trans, m, n, al, A, m, x, 1, be, got, 1)
    assert gpu.last_error()[0] == 0, gpu.last_error()
    absA = np.abs(A[..., 0]) + np.abs(A[..., 1])
    absx = np.abs(x[:, 0]) + np.abs(x[:, 1])
    total = (absA.T @ absx) if trans == "N" else (absA @ absx)
    bound = orc.dd_abs(al) * total + orc.dd_abs(be) * np.abs(y0[:, 0])
    err = np.abs((got[:, 0] - want[:, 0]) + (got[:, 1] - want[:, 1]))
    assert np.all(err <= 16 * orc.EPS_DD * bound), np.max(err / bound) / orc.EPS_DD


@pytest.mark.parametrize("trans", ["N", "T"])
def test_gemv_nonfinite(gpu, rng, trans):
    """A non-finite entry of A makes its own output NaN, one of x every output."""
    outs, red = 70, 130
    m, n = (outs, red) if trans == "N" else (red, outs)
    A, x = mwb.dd_matrix(rng, m, n), mwb.random_dd(rng, (red,))
    one, zero = np.array([1.0, 0.0]), np.zeros(2)
    for bad in (np.inf, np.nan):
        B = A.copy()
        B[(77, 41) if trans == "N" else (41, 77)] = (bad, 0.0)
        y = np.zeros((outs, 2))
        gpu.mgemv(trans, m, n, one, B, m, x, 1, zero, y, 1)
        assert np.array_equal(np.isnan(y[:, 0]), np.arange(outs) == 41)
        xb = x.copy()
        xb[129] = (bad, 0.0)
        y = np.zeros((outs, 2))
        gpu.mgemv(trans, m, n, one, A, m, xb, 1, zero, y, 1)
        assert np.all(np.isnan(y[:, 0]))
