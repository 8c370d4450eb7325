"""A complex alpha whose parts differ by many binades, on real data in complex
arrays: the product's parts are alpha's times one real number, and each is good
to its own 2^-104 (rounded once, from 128 bits), against exact rationals.
"""
from fractions import Fraction as F

import numpy as np
import pytest

from conftest import mwb

pytestmark = pytest.mark.gpu

M, N, K = 70, 33, 64


@pytest.mark.parametrize("small", ["re", "im"])
@pytest.mark.parametrize("binades", [20, 60, 100, 127, 200])
def test_parts(gpu, rng, binades, small):
    a, b = rng.integers(-4096, 4096, (K, M)), rng.integers(-4096, 4096, (N, K))     # [column, row]
    p = b @ a

    def cplx(v):
        out = np.zeros((*v.shape, 2, 2))
        out[..., 0, 0] = v
        return out

    parts = [mwb.random_dd(rng, ()) + np.array([1.25, 0.0]) for _ in range(2)]
    parts[0 if small == "re" else 1] *= 2.0 ** -binades
    C = np.full((N, M, 2, 2), 7.0)
    prev = gpu.lib.mwblas_set_gemm_engine(2)
    try:
        gpu.wgemm("N", "N", M, N, K, np.stack(parts), cplx(a), M, cplx(b), K, np.zeros((2, 2)), C, M)
        assert gpu.last_error()[0] == 0, gpu.last_error()
    finally:
        gpu.lib.mwblas_set_gemm_engine(prev)
    for w in range(2):
        scale = F(float(parts[w][0])) + F(float(parts[w][1]))
        for j in range(N):
            for i in range(M):
                want, got = scale * int(p[j, i]), F(float(C[j, i, w, 0])) + F(float(C[j, i, w, 1]))
                assert abs(got - want) <= abs(want) * F(2) ** -104, (w, j, i, float(abs(got - want) / abs(want)))
