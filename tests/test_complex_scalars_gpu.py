"""Complex products on the tensor-core engine with scalars of which one part is
zero, against the binary128 oracle, entry by entry: good to 2^-104
(4k |A||B| |alpha| + 4 |beta C|) in each part, twice that for complex products.
"""
import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu

PARTS = ["re", "im", "both"]


def scalar(rng, parts):
    one = lambda: mwb.random_dd(rng, ()) + np.array([1.25, 0.0])
    zero = np.zeros(2)
    return np.stack([zero if parts == "im" else one(), zero if parts == "re" else one()])


def check(got, want, C0, A, B, al, be, k):
    f = (lambda v: np.abs(v).reshape(*v.shape[:2], -1).sum(axis=2))
    bound = 4 * k * np.abs(al).sum() * orc.dd_absmax(A) * orc.dd_absmax(B) + 4 * np.abs(be).sum() * f(C0)
    err = np.abs((got[..., 0] - want[..., 0]) + (got[..., 1] - want[..., 1])).reshape(*bound.shape, -1).max(axis=2)
    assert np.all(err <= 2 * orc.EPS_DD * bound), np.max(err / bound) / orc.EPS_DD


@pytest.mark.parametrize("beta", PARTS)
@pytest.mark.parametrize("alpha", PARTS)
@pytest.mark.parametrize("data", ["complex", "real"])
def test_wgemm(gpu, oracle, rng, data, alpha, beta):
    m, n, k = 129, 70, 200
    A, B, C0 = (mwb.dd_matrix(rng, *s, cplx_=True) for s in ((m, k), (k, n), (m, n)))
    if data == "real":          # products whose imaginary part is exactly zero
        A[..., 1, :] = B[..., 1, :] = 0.0
    al, be = scalar(rng, alpha), scalar(rng, beta)
    want, got = C0.copy(), C0.copy()
    prev = gpu.lib.mwblas_set_gemm_engine(2)
    try:
        oracle.qwgemm("N", "N", m, n, k, al, A, m, B, k, be, want, m)
        gpu.wgemm("N", "N", m, n, k, al, A, m, B, k, be, got, m)
        assert gpu.last_error()[0] == 0, gpu.last_error()
    finally:
        gpu.lib.mwblas_set_gemm_engine(prev)
    check(got, want, C0, A, B, al, be, k)


@pytest.mark.parametrize("what", ["alpha", "beta"])
def test_real_scalar_without_high_limb(gpu, oracle, rng, what):
    """A real scalar with hi = 0 and lo != 0 is a zero of the fixed-point update:
    the other term keeps its bits."""
    m, n, k = 129, 70, 200
    A, B, C0 = (mwb.dd_matrix(rng, *s) for s in ((m, k), (k, n), (m, n)))
    tiny, al, be = np.array([0.0, 2.0 ** -300]), np.array([1.25, 0.0]), np.array([0.75, 0.0])
    if what == "alpha":
        al = tiny
    else:
        be = tiny
    want, got = C0.copy(), C0.copy()
    prev = gpu.lib.mwblas_set_gemm_engine(2)
    try:
        oracle.qgemm("N", "N", m, n, k, al, A, m, B, k, be, want, m)
        gpu.mgemm("N", "N", m, n, k, al, A, m, B, k, be, got, m)
        assert gpu.last_error()[0] == 0, gpu.last_error()
    finally:
        gpu.lib.mwblas_set_gemm_engine(prev)
    f = (lambda v: np.abs(v).sum(axis=2))
    bound = 4 * k * np.abs(al).sum() * orc.dd_absmax(A) * orc.dd_absmax(B) + 4 * np.abs(be).sum() * f(C0)
    err = np.abs((got[..., 0] - want[..., 0]) + (got[..., 1] - want[..., 1]))
    assert np.all(err <= orc.EPS_DD * bound), np.max(err / bound) / orc.EPS_DD
