"""The CTA-pair residue GEMM's epilogue against the CUDA-core residue kernel, bit
for bit: column pairs cut by an odd edge, rows and columns past a tile, both sides
of the K at which the accumulator hand-back changes (3072), and triangles, whose
tiles are walked alone."""
import numpy as np
import pytest

from conftest import mwb
from test_ozaki_gpu import OZAKI, engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(255, 129), (513, 257)])
@pytest.mark.parametrize("k", [3072, 3073])
def test_epilogue_bits(gpu, rng, m, n, k):
    A, B = mwb.dd_matrix(rng, m, k), mwb.dd_matrix(rng, k, n)
    outs = []
    for kind in (1, 3):   # CUDA cores, CTA pairs
        prev = gpu.lib.mwblas_set_ozaki_mma(kind)
        try:
            c = np.zeros((n, m, 2))
            gpu.mgemm("N", "N", m, n, k, 1.0, A, m, B, k, 0.0, c, m, engine="ozaki")
            assert gpu.last_error()[0] == 0, gpu.last_error()
            outs.append(c)
        finally:
            gpu.lib.mwblas_set_ozaki_mma(prev)
    np.testing.assert_array_equal(outs[0], outs[1])


@pytest.mark.parametrize("uplo", ["U", "L"])
@pytest.mark.parametrize("n", [256, 257, 769])
def test_triangle_bits(gpu, rng, uplo, n):
    k = 70
    A, C = mwb.dd_matrix(rng, n, k), mwb.dd_matrix(rng, n, n)
    outs = []
    for kind in (1, 3):
        prev = gpu.lib.mwblas_set_ozaki_mma(kind)
        try:
            c = C.copy()
            with engine(gpu, OZAKI):
                gpu.msyrk(uplo, "N", n, k, 1.0, A, n, 0.5, c, n)
            assert gpu.last_error()[0] == 0, gpu.last_error()
            outs.append(c)
        finally:
            gpu.lib.mwblas_set_ozaki_mma(prev)
    np.testing.assert_array_equal(outs[0], outs[1])
    other = np.tril_indices(n, -1) if uplo == "L" else np.triu_indices(n, 1)   # [column, row] storage
    np.testing.assert_array_equal(outs[1][other], C[other])
