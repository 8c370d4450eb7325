"""mdot_ around the edges of its tensor-core kernel, against the binary128
oracle: groups of 32 pairs, turns of 64 per warp, moves of the sums every four
turns, and the operands that leave its straight-line path.

Every product is exact in 2^-110 of its warp's largest one and the result is
rounded once, so it is good to a few units of 2^-104 of sum |x y| (8 allowed).
"""
import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["plain", "zeros", "fp64", "spread", "loose", "positive"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 64, 65, 511, 512, 513, 200001, 1300000])
def test_dot_edges(gpu, oracle, rng, n, kind):
    x, y = mwb.random_dd(rng, (n,)), mwb.random_dd(rng, (n,))
    if kind == "zeros":
        x[rng.random(n) < 0.5] = 0.0
        y[: n // 2] = 0.0
    elif kind == "fp64":
        x[:, 1] = 0.0
        y[:, 1] = -0.0
    elif kind == "spread":                     # growing blocks, long alignments
        x *= 2.0 ** rng.integers(-90, 90, n)[:, None]
        y *= 2.0 ** np.sort(rng.integers(-60, 60, n))[:, None]
    elif kind == "loose":                      # not normalised: lo up to hi's size
        x[:, 1] = x[:, 0] * rng.uniform(-0.4, 0.4, n)
    elif kind == "positive":                   # limb sums at their largest
        x, y = np.abs(x[:, :1]) * [1.0, 2.0 ** -54], np.abs(y[:, :1]) * [1.0, 2.0 ** -54]
    got = np.array(gpu.mdot(n, x, 1, y, 1))
    assert gpu.last_error()[0] == 0, gpu.last_error()
    want = oracle.qdot(n, x, 1, y, 1)
    total = np.sum(np.abs(x).sum(axis=1) * np.abs(y).sum(axis=1))
    err = abs((got[0] - want[0]) + (got[1] - want[1]))
    assert err <= 8 * orc.EPS_DD * total, err / total / orc.EPS_DD


@pytest.mark.parametrize("incx,incy", [(3, 1), (-1, 2), (-2, -5)])
def test_dot_increments(gpu, oracle, rng, incx, incy):
    n = 3333
    x, y = (mwb.random_dd(rng, (1 + (n - 1) * abs(i),)) for i in (incx, incy))
    got, want = np.array(gpu.mdot(n, x, incx, y, incy)), oracle.qdot(n, x, incx, y, incy)
    err = abs((got[0] - want[0]) + (got[1] - want[1]))
    assert err <= 8 * orc.EPS_DD * n
