"""MTRSM's alpha: in the products that first read B where it is near one, in B
itself where it is not (2^64 and beyond on either side), against the binary128
oracle within the substitution's max(20, 8 n^2) 2^-104 |alpha| |B|."""
import numpy as np
import pytest

from conftest import mwb, orc
from test_level3_gpu import dominant_triangle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,uplo,ta", [("L", "L", "N"), ("L", "L", "T"), ("R", "U", "N"), ("R", "U", "T")])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** 62, 2.0 ** 66, 2.0 ** -66])
def test_alpha(gpu, oracle, rng, side, uplo, ta, scale):
    na, nr = 201, 130
    m, n = (na, nr) if side == "L" else (nr, na)
    A = dominant_triangle(rng, na, na)
    B0 = mwb.dd_matrix(rng, m, n, m)
    al = (mwb.random_dd(rng, ()) + np.array([1.5, 0.0])) * scale
    want, got = B0.copy(), B0.copy()
    oracle.qtrsm(side, uplo, ta, "N", m, n, al, A, na, want, m)
    gpu.mtrsm(side, uplo, ta, "N", m, n, al, A, na, got, m)
    assert gpu.last_error()[0] == 0, gpu.last_error()
    err = orc.normwise_error(got, want, orc.dd_abs(al) * orc.dd_absmax(B0))
    assert err <= max(20, 8 * na * na) * orc.EPS_DD, err


@pytest.mark.parametrize("side,uplo,diag", [("L", "L", "N"), ("L", "U", "U"), ("R", "U", "N"), ("R", "L", "U")])
@pytest.mark.parametrize("na", [129, 144, 145, 159])
def test_last_inverted_block(gpu, oracle, rng, side, uplo, diag, na):
    """The last diagonal block of 1, 16, 17 and 31 rows: one half alone, and two."""
    nr = 5
    m, n = (na, nr) if side == "L" else (nr, na)
    A = dominant_triangle(rng, na, na)
    B0 = mwb.dd_matrix(rng, m, n, m)
    al = mwb.random_dd(rng, ())
    want, got = B0.copy(), B0.copy()
    oracle.qtrsm(side, uplo, "N", diag, m, n, al, A, na, want, m)
    gpu.mtrsm(side, uplo, "N", diag, m, n, al, A, na, got, m)
    assert gpu.last_error()[0] == 0, gpu.last_error()
    err = orc.normwise_error(got, want, orc.dd_abs(al) * orc.dd_absmax(B0))
    assert err <= max(20, 8 * na * na) * orc.EPS_DD, err
