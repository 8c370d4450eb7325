"""mgemv_ with a short reduction (up to 32: a thread per output) around its lengths
and groups of four, against the binary128 oracle: 16 units of 2^-104 of
|alpha| sum |A x| + |beta y|, as for the long reductions.
"""
import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["plain", "zeros", "spread", "far_lo", "subnormal"])
@pytest.mark.parametrize("beta", ["zero", "one", "general"])
@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("outs,red", [(1, 1), (257, 3), (1000, 4), (255, 5), (700, 31), (600, 32), (600, 33),
                                      (700000, 7)])
def test_short(gpu, oracle, rng, outs, red, trans, beta, kind):
    m, n = (outs, red) if trans == "N" else (red, outs)
    A, x = mwb.dd_matrix(rng, m, n, m + 1, fill=7.0), mwb.random_dd(rng, (red,))
    if kind == "zeros":
        A[rng.random(A.shape[:2]) < 0.5] = 0.0
        x[rng.random(red) < 0.4] = 0.0
    elif kind == "spread":
        A *= 2.0 ** rng.integers(-90, 90, A.shape[:2])[..., None]
        x *= 2.0 ** rng.integers(-60, 60, red)[:, None]
    elif kind == "far_lo":
        A[..., 1] *= 2.0 ** -rng.integers(0, 60, A.shape[:2]).astype(float)
    elif kind == "subnormal":
        A[:, ::3] *= 2.0 ** -1000
        x *= 2.0 ** 300
    y0 = mwb.random_dd(rng, (outs,))
    al = mwb.random_dd(rng, ()) + np.array([1.5, 0.0])
    be = {"zero": np.zeros(2), "one": np.array([1.0, 0.0]), "general": mwb.random_dd(rng, ())}[beta]
    if beta == "zero":
        y0[::2] = np.nan                            # y is written, never read
    want, got = np.nan_to_num(y0), y0.copy()
    oracle.qgemv(trans, m, n, al, A, m + 1, x, 1, be, want, 1)
    gpu.mgemv(trans, m, n, al, A, m + 1, x, 1, be, got, 1)
    assert gpu.last_error()[0] == 0, gpu.last_error()
    absA, absx = np.abs(A[:, :m, 0]), np.abs(x[:, 0])
    total = (absA.T @ absx) if trans == "N" else (absA @ absx)
    bound = orc.dd_abs(al) * total + orc.dd_abs(be) * np.abs(np.nan_to_num(y0[:, 0]))
    err = np.abs((got[:, 0] - want[:, 0]) + (got[:, 1] - want[:, 1]))
    assert np.all(err <= 16 * orc.EPS_DD * bound + 5e-324), np.max(err / bound) / orc.EPS_DD


@pytest.mark.parametrize("incx,incy", [(2, 1), (-1, -3)])
def test_increments(gpu, oracle, rng, incx, incy):
    m, n = 300, 9
    A = mwb.dd_matrix(rng, m, n)
    x, y0 = mwb.random_dd(rng, (1 + (n - 1) * abs(incx),)), mwb.random_dd(rng, (1 + (m - 1) * abs(incy),))
    one, be = np.array([1.0, 0.0]), mwb.random_dd(rng, ())
    want, got = y0.copy(), y0.copy()
    oracle.qgemv("N", m, n, one, A, m, x, incx, be, want, incy)
    gpu.mgemv("N", m, n, one, A, m, x, incx, be, got, incy)
    assert np.abs((got[:, 0] - want[:, 0]) + (got[:, 1] - want[:, 1])).max() <= 16 * orc.EPS_DD * (n + 1)


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_nonfinite(gpu, rng, bad):
    m, n = 70, 6
    one, zero = np.array([1.0, 0.0]), np.zeros(2)
    A, x, y = mwb.dd_matrix(rng, m, n), mwb.random_dd(rng, (n,)), np.zeros((m, 2))
    A[4, 41] = (bad, 0.0)
    gpu.mgemv("N", m, n, one, A, m, x, 1, zero, y, 1)
    assert np.array_equal(np.isnan(y[:, 0]), np.arange(m) == 41)
    A[4, 41] = 0.0
    x[4] = (bad, 0.0)
    gpu.mgemv("N", m, n, one, A, m, x, 1, zero, y, 1)
    assert np.all(np.isnan(y[:, 0]))
