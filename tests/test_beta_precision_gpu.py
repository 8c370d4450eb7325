"""C + alpha A B where the product lies far below C, or C's low limb far below its
high one: the update of the tensor-core engine and of the grouped limb tiles
keeps 2^-122 of C (extended floats of 128 bits did), against exact rationals.

A and B are small integers times 2^-75, so the product is exact, near 2^-120, and
C's limbs are such that the result's low limb holds 2^-123 of it.
"""
from fractions import Fraction as F

import numpy as np
import pytest

from conftest import mwb

pytestmark = pytest.mark.gpu

M, N, K = 70, 33, 64


def operands(rng, kind):
    a, b = rng.integers(-4096, 4096, (K, M)), rng.integers(-4096, 4096, (N, K))     # [column, row]
    p = b @ a                                                                       # in units of 2^-150
    A, B = (np.stack([v * 2.0 ** -75, np.zeros(v.shape)], axis=-1) for v in (a, b))
    C = np.zeros((N, M, 2))
    C[..., 0] = 1.0 + rng.integers(0, 1 << 20, (N, M)) * 2.0 ** -20
    if kind == "far_lo":
        C[..., 1] = rng.integers(-(1 << 50), 1 << 50, (N, M)) * 2.0 ** -122         # 70 bits and more below hi
    return A, B, C, p


def worst(got, C, p, beta):
    """The largest error in units of 2^-122 |C|."""
    exact = lambda v: F(float(v[0])) + F(float(v[1]))
    return max(float(abs(exact(got[j, i]) - beta * exact(C[j, i]) - F(int(p[j, i]), 1 << 150)) / F(float(C[j, i, 0])))
               for j in range(N) for i in range(M)) * 2.0 ** 122


@pytest.mark.parametrize("kind", ["high_limb", "far_lo"])
@pytest.mark.parametrize("beta", [1.0, 0.75])
@pytest.mark.parametrize("path", ["real", "complex", "grouped"])
def test_far_below_c(gpu, rng, path, beta, kind):
    import torch
    A, B, C, p = operands(rng, kind)
    be, one = np.array([beta, 0.0]), np.array([1.0, 0.0])
    if path == "grouped":
        d = [torch.from_numpy(v).cuda() for v in (A, B, C)]
        prev = gpu.lib.mwblas_set_grouped_tile(16)
        try:
            assert gpu.mgemm_grouped(["N"], ["N"], [M], [N], [K], [one], [d[0].data_ptr()], [M], [d[1].data_ptr()],
                                     [K], [be], [d[2].data_ptr()], [M]) == 0, gpu.last_error()
        finally:
            gpu.lib.mwblas_set_grouped_tile(prev)
        got = d[2].cpu().numpy()
    else:
        prev = gpu.lib.mwblas_set_gemm_engine(2)
        try:
            if path == "real":
                got = C.copy()
                gpu.mgemm("N", "N", M, N, K, one, A, M, B, K, be, got, M)
            else:
                zero = np.zeros(2)
                cplx = lambda v: np.stack([v, np.zeros(v.shape)], axis=-2)
                full = cplx(C)
                gpu.wgemm("N", "N", M, N, K, np.stack([one, zero]), cplx(A), M, cplx(B), K, np.stack([be, zero]), full,
                          M)
                got = full[..., 0, :]
                assert np.all(full[..., 1, :] == 0.0)
            assert gpu.last_error()[0] == 0, gpu.last_error()
        finally:
            gpu.lib.mwblas_set_gemm_engine(prev)
    assert worst(got, C, p, F(beta)) <= 1.0
