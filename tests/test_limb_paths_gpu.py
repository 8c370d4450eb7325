"""The groups of mgemv_ and mdot_ that leave the kernels' short path for the loop of
any shift, and come back: zeros in all places, whole groups of them, exponents
that rise past their block by a few bits or many, falling ones, and non-finite
entries beside zeros, against the binary128 oracle.

Bounds as in the tests of the kernels' edges: 16 (mgemv_) and 8 (mdot_) units of
2^-104 of the sum of magnitudes.
"""
import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu

KINDS = ["rise", "rise_fast", "fall", "one_zero", "runs", "ends", "negative_zero"]


def shape_values(rng, v, kind):
    """v: [..., index, limb], changed along the index."""
    n = v.shape[-2]
    i = np.arange(n)
    if kind == "rise":                       # a bit every 5 indices: past the block by a few bits at a time
        v *= (2.0 ** (i // 5 % 200))[:, None]
    elif kind == "rise_fast":                # 4 bits per index: by more than the spare bits
        v *= (2.0 ** (4 * (i % 60)))[:, None]
    elif kind == "fall":                     # shifts from none to past every bit
        v *= (2.0 ** -(i % 150).astype(float))[:, None]
    elif kind == "one_zero":
        v[..., i % 37 == 11, :] = 0.0
    elif kind == "runs":                     # groups and windows of zeros between dense ones
        v[..., (i // 40) % 3 == 1, :] = 0.0
    elif kind == "ends":
        v[..., : n // 3, :] = 0.0
        v[..., n - n // 4:, :] = 0.0
    elif kind == "negative_zero":
        v[..., i % 3 == 1, :] = -0.0
        v[..., i % 7 == 2, 1] = -0.0
    return v


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("where", ["A", "x"])
@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("outs,red", [(33, 700), (300, 131)])
def test_gemv(gpu, oracle, rng, outs, red, trans, where, kind):
    m, n = (outs, red) if trans == "N" else (red, outs)
    A, x = mwb.random_dd(rng, (outs, red)), mwb.random_dd(rng, (red,))
    if where == "A":
        shape_values(rng, A[::2], kind)      # every second output, its neighbours stay dense
    else:
        shape_values(rng, x, kind)
    if trans == "N":
        A = np.ascontiguousarray(A.transpose(1, 0, 2))
    y0 = mwb.random_dd(rng, (outs,))
    al, be = mwb.random_dd(rng, ()) + np.array([1.5, 0.0]), mwb.random_dd(rng, ())
    want, got = y0.copy(), y0.copy()
    oracle.qgemv(trans, m, n, al, A, m, x, 1, be, want, 1)
    gpu.mgemv(trans, m, n, al, A, m, x, 1, be, got, 1)
    assert gpu.last_error()[0] == 0, gpu.last_error()
    absA, absx = np.abs(A[..., 0]), np.abs(x[:, 0])
    total = (absA.T @ absx) if trans == "N" else (absA @ absx)
    bound = orc.dd_abs(al) * total + orc.dd_abs(be) * np.abs(y0[:, 0])
    err = np.abs((got[:, 0] - want[:, 0]) + (got[:, 1] - want[:, 1]))
    assert np.all(err <= 16 * orc.EPS_DD * bound), np.max(err / bound) / orc.EPS_DD


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("where", ["x", "y", "both"])
@pytest.mark.parametrize("n", [700, 400000])
def test_dot(gpu, oracle, rng, n, where, kind):
    x, y = mwb.random_dd(rng, (n,)), mwb.random_dd(rng, (n,))
    if where != "y":
        shape_values(rng, x, kind)
    if where != "x":
        shape_values(rng, y, kind)
    got = np.array(gpu.mdot(n, x, 1, y, 1))
    assert gpu.last_error()[0] == 0, gpu.last_error()
    want = oracle.qdot(n, x, 1, y, 1)
    total = np.sum(np.abs(x[:, 0]) * np.abs(y[:, 0]))
    err = abs((got[0] - want[0]) + (got[1] - want[1]))
    assert err <= 8 * orc.EPS_DD * total, err / total / orc.EPS_DD


@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("zeros", ["matrix", "vector"])
def test_nonfinite_beside_zeros(gpu, rng, bad, zeros):
    """0 * inf is not a number, also where everything around it is zero."""
    outs, red = 70, 200
    A, x = mwb.dd_matrix(rng, outs, red), mwb.random_dd(rng, (red,))
    if zeros == "matrix":
        A[:, :, :] = 0.0
        x[77] = (bad, 0.0)
        want = np.ones(outs, bool)
    else:
        x[:, :] = 0.0
        A[77, 41] = (bad, 0.0)
        want = np.arange(outs) == 41
    y = np.zeros((outs, 2))
    gpu.mgemv("N", outs, red, np.array([1.0, 0.0]), A, outs, x, 1, np.zeros(2), y, 1)
    assert np.array_equal(np.isnan(y[:, 0]), want)
    u, v = np.zeros((red, 2)), np.zeros((red, 2))
    (u if zeros == "matrix" else v)[133] = (bad, 0.0)
    assert np.isnan(gpu.mdot(red, u, 1, v, 1)[0])
