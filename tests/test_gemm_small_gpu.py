"""The fixed-point engine's small tiles (8 x 8 and 16 x 16 outputs, K in chunks
of 64) against the binary128 oracle: edges of tiles and chunks, every transpose
pair, padding, triangles, scaled rows and non-finite entries.

Operands are rounded to 116 bits of their row or column maximum and the rest is
exact up to one rounding: normwise max(10, 4k) 2^-104 as for every engine, and
for these k a few units, 16 2^-104 k |A| |B|, are allowed.
"""
import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu


def check(gpu, oracle, rng, ta, tb, m, n, k, pad=3, beta=None, A=None, B=None):
    A = mwb.dd_matrix(rng, m if ta == "N" else k, k if ta == "N" else m,
                      (m if ta == "N" else k) + pad, fill=np.nan) if A is None else A
    B = mwb.dd_matrix(rng, k if tb == "N" else n, n if tb == "N" else k,
                      (k if tb == "N" else n) + pad, fill=np.nan) if B is None else B
    C0 = mwb.dd_matrix(rng, m, n, m + pad, fill=7.0)
    al = mwb.random_dd(rng, ()) + np.array([1.5, 0.0])
    be = mwb.random_dd(rng, ()) if beta is None else np.array(beta)
    want, got = C0.copy(), C0.copy()
    oracle.qgemm(ta, tb, m, n, k, al, A, A.shape[1], B, B.shape[1], be, want, m + pad)
    gpu.mgemm(ta, tb, m, n, k, al, A, A.shape[1], B, B.shape[1], be, got, m + pad, engine="fixed")
    assert gpu.last_error()[0] == 0, gpu.last_error()
    assert np.array_equal(got[:, m:], C0[:, m:])
    a = A[:, : m if ta == "N" else k]
    b = B[:, : k if tb == "N" else n]
    op = orc.dd_abs(al) * k * orc.dd_absmax(a) * orc.dd_absmax(b) + orc.dd_abs(be) * orc.dd_absmax(C0[:, :m])
    assert orc.normwise_error(got[:, :m], want[:, :m], op) <= 16 * orc.EPS_DD


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T")])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (8, 8, 64), (9, 7, 65), (16, 17, 63), (15, 33, 129), (200, 200, 70),
                                   (161, 150, 64), (16, 16, 3000), (3, 900, 31), (900, 3, 5)])
def test_small_tiles(gpu, oracle, rng, m, n, k, ta, tb):
    check(gpu, oracle, rng, ta, tb, m, n, k)


@pytest.mark.parametrize("beta", [[0.0, 0.0], [1.0, 0.0]])
@pytest.mark.parametrize("k", [40, 100])
def test_small_tiles_beta(gpu, oracle, rng, beta, k):
    check(gpu, oracle, rng, "N", "T", 37, 21, k, beta=beta)


@pytest.mark.parametrize("k", [30, 150])
def test_small_tiles_scaled_rows_and_nonfinite(gpu, oracle, rng, k):
    """Rows of A and columns of B over 2^+-200: each output is good to its own
    row and column; a non-finite entry makes its row of C NaN, a zero row gives beta C."""
    m, n = 20, 25
    A, B = mwb.dd_matrix(rng, m, k), mwb.dd_matrix(rng, k, n)
    A *= (2.0 ** rng.integers(-200, 200, m))[None, :, None]
    B *= (2.0 ** rng.integers(-200, 200, n))[:, None, None]
    A[:, 4] = 0.0
    one, zero = np.array([1.0, 0.0]), np.zeros(2)
    want, got = np.zeros((n, m, 2)), np.zeros((n, m, 2))
    oracle.qgemm("N", "N", m, n, k, one, A, m, B, k, zero, want, m)
    gpu.mgemm("N", "N", m, n, k, one, A, m, B, k, zero, got, m, engine="fixed")
    bound = np.abs(B[..., 0]).max(axis=1)[:, None] * np.abs(A[..., 0]).max(axis=0)[None, :] * k
    err = np.abs((got[..., 0] - want[..., 0]) + (got[..., 1] - want[..., 1]))
    assert np.all(err <= 16 * orc.EPS_DD * bound)
    A[k // 2, 9] = (np.inf, 0.0)
    gpu.mgemm("N", "N", m, n, k, one, A, m, B, k, zero, got, m, engine="fixed")
    assert np.array_equal(np.isnan(got[..., 0]), np.broadcast_to(np.arange(m) == 9, (n, m)))


@pytest.mark.parametrize("uplo", ["U", "L"])
def test_small_tiles_triangle(gpu, oracle, rng, uplo):
    n, k = 45, 70
    A, C0 = mwb.dd_matrix(rng, n, k), mwb.dd_matrix(rng, n, n)
    al, be = mwb.random_dd(rng, ()), mwb.random_dd(rng, ())
    want, got = C0.copy(), C0.copy()
    oracle.qsyrk(uplo, "N", n, k, al, A, n, be, want, n)
    gpu.msyrk(uplo, "N", n, k, al, A, n, be, got, n)
    op = orc.dd_abs(al) * k * orc.dd_absmax(A) ** 2 + orc.dd_abs(be) * orc.dd_absmax(C0)
    assert orc.normwise_error(got, want, op) <= 16 * orc.EPS_DD
    keep = np.triu(np.ones((n, n), bool)) if uplo == "U" else np.tril(np.ones((n, n), bool))   # [row, column]
    assert np.array_equal(got[~keep.T], C0[~keep.T])
