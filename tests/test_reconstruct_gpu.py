"""The tensor-core engine's reconstruction at the operands that choose its
paths, against the binary128 oracle: C far above and far below the product, C
with zero, subnormal and non-finite entries, unnormalised C, more than 32
moduli, zero rows, both triangles, real and complex.

An output is good to 2^-104 (4k |A||B| |alpha| + 4 |beta C|), entry by entry
where C is scaled.
"""
import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu

SIZES = [(70, 65, 64), (129, 63, 200), (260, 33, 33)]


def scalars(rng, cplx):
    one = lambda: mwb.random_dd(rng, ()) + np.array([1.25, 0.0])
    return (np.stack([one(), one()]), np.stack([one(), one()])) if cplx else (one(), one())


def c_entries(C, rng, kind):
    shape = C.shape[:2]
    if kind == "wide":
        C *= (2.0 ** rng.integers(-140, 140, shape)).reshape(*shape, *([1] * (C.ndim - 2)))
    elif kind == "special":
        u = rng.random(shape)
        C[u < 0.2] = 0.0
        C[(u >= 0.2) & (u < 0.4)] *= 2.0 ** -1010
        C[(u >= 0.4) & (u < 0.6), ..., 1] = C[(u >= 0.4) & (u < 0.6), ..., 0] * 0.3     # not normalised
    return C


@pytest.mark.parametrize("kind", ["plain", "wide", "special"])
@pytest.mark.parametrize("beta", ["zero", "one", "general"])
@pytest.mark.parametrize("m,n,k", SIZES)
@pytest.mark.parametrize("cplx", [False, True])
def test_reconstruction_paths(gpu, oracle, rng, cplx, m, n, k, beta, kind):
    A, B = mwb.dd_matrix(rng, m, k, cplx_=cplx), mwb.dd_matrix(rng, k, n, cplx_=cplx)
    C0 = c_entries(mwb.dd_matrix(rng, m, n, m + 2, cplx_=cplx, fill=3.0), rng, kind)
    A[:, 5] = 0.0                                   # a row without a nonzero entry
    al, be = scalars(rng, cplx)
    if beta != "general":
        be = np.zeros_like(be)
        if beta == "one":
            be[..., 0].flat[0] = 1.0
    want, got = C0.copy(), C0.copy()
    prev = gpu.lib.mwblas_set_gemm_engine(2)
    try:
        if cplx:
            oracle.qwgemm("N", "N", m, n, k, al, A, m, B, k, be, want, m + 2)
            gpu.wgemm("N", "N", m, n, k, al, A, m, B, k, be, got, m + 2)
        else:
            oracle.qgemm("N", "N", m, n, k, al, A, m, B, k, be, want, m + 2)
            gpu.mgemm("N", "N", m, n, k, al, A, m, B, k, be, got, m + 2)
        assert gpu.last_error()[0] == 0, gpu.last_error()
    finally:
        gpu.lib.mwblas_set_gemm_engine(prev)
    assert np.array_equal(got[:, m:], C0[:, m:])
    f = (lambda v: np.abs(v).reshape(*v.shape[:2], -1).sum(axis=2))
    bound = 4 * k * np.abs(al).sum() * orc.dd_absmax(A) * orc.dd_absmax(B) + 4 * np.abs(be).sum() * f(C0[:, :m])
    if cplx:
        bound *= 2
    err = np.abs((got[:, :m, ..., 0] - want[:, :m, ..., 0]) + (got[:, :m, ..., 1] - want[:, :m, ..., 1]))
    err = err.reshape(n, m, -1).max(axis=2)
    assert np.all(err <= orc.EPS_DD * bound), np.max(err / bound) / orc.EPS_DD


@pytest.mark.parametrize("cplx", [False, True])
def test_reconstruction_of_30_moduli(gpu, oracle, rng, cplx):
    m, n, k = 130, 70, 96
    A, B, C0 = (mwb.dd_matrix(rng, *s, cplx_=cplx) for s in ((m, k), (k, n), (m, n)))
    al, be = scalars(rng, cplx)
    want, got = C0.copy(), C0.copy()
    prev, bits = gpu.lib.mwblas_set_gemm_engine(2), gpu.lib.mwblas_set_ozaki_bits(116)
    try:
        (oracle.qwgemm if cplx else oracle.qgemm)("N", "N", m, n, k, al, A, m, B, k, be, want, m)
        (gpu.wgemm if cplx else gpu.mgemm)("N", "N", m, n, k, al, A, m, B, k, be, got, m)
        assert gpu.last_error()[0] == 0 and gpu.lib.mwblas_last_ozaki_moduli() > 28
    finally:
        gpu.lib.mwblas_set_gemm_engine(prev)
        gpu.lib.mwblas_set_ozaki_bits(bits)
    op = np.abs(al).sum() * k * orc.dd_absmax(A) * orc.dd_absmax(B) + np.abs(be).sum() * orc.dd_absmax(C0)
    err = np.abs((got[..., 0] - want[..., 0]) + (got[..., 1] - want[..., 1])).max()
    assert err <= 8 * orc.EPS_DD * op


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_reconstruction_nonfinite_c(gpu, rng, bad):
    m, n, k = 100, 70, 64
    A, B, C = mwb.dd_matrix(rng, m, k), mwb.dd_matrix(rng, k, n), mwb.dd_matrix(rng, m, n)
    C[13, 41] = (bad, 0.0)
    one = np.array([1.0, 0.0])
    gpu.mgemm("N", "N", m, n, k, one, A, m, B, k, one, C, m, engine="ozaki")
    off = ~np.isfinite(C[..., 0])
    assert off[13, 41] and off.sum() == 1


@pytest.mark.parametrize("uplo", ["U", "L"])
@pytest.mark.parametrize("n", [63, 64, 65, 200, 600])
def test_reconstruction_triangles(gpu, oracle, rng, uplo, n):
    k = 64
    A, C0 = mwb.dd_matrix(rng, n, k), mwb.dd_matrix(rng, n, n)
    al, be = scalars(rng, False)
    want, got = C0.copy(), C0.copy()
    prev = gpu.lib.mwblas_set_gemm_engine(2)
    try:
        oracle.qsyrk(uplo, "N", n, k, al, A, n, be, want, n)
        gpu.msyrk(uplo, "N", n, k, al, A, n, be, got, n)
    finally:
        gpu.lib.mwblas_set_gemm_engine(prev)
    op = orc.dd_abs(al) * k * orc.dd_absmax(A) ** 2 + orc.dd_abs(be) * orc.dd_absmax(C0)
    assert orc.normwise_error(got, want, op) <= 8 * orc.EPS_DD
    keep = np.triu(np.ones((n, n), bool)) if uplo == "U" else np.tril(np.ones((n, n), bool))   # [row, column]
    assert np.array_equal(got[~keep.T], C0[~keep.T])
