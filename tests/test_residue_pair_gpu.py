"""Both operands' residues in one launch against the FP32 path, bit for bit: every
pair of layouts, row tiles of 16 cut short on either side, and k past a tile."""
import numpy as np
import pytest

from conftest import mwb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T")])
@pytest.mark.parametrize("m,n,k", [(1, 300, 33), (257, 15, 64), (130, 131, 97)])
def test_pair(gpu, rng, ta, tb, m, n, k):
    A = mwb.dd_matrix(rng, m if ta == "N" else k, k if ta == "N" else m)
    B = mwb.dd_matrix(rng, k if tb == "N" else n, n if tb == "N" else k)
    outs = []
    for tc in (0, 1):
        prev = gpu.lib.mwblas_set_residue_tc(tc)
        try:
            c = np.zeros((n, m, 2))
            import torch
            a, b, d = (torch.from_numpy(x).cuda() for x in (A, B, c))
            gpu.mgemm(ta, tb, m, n, k, 1.0, a.data_ptr(), A.shape[1], b.data_ptr(), B.shape[1], 0.0, d.data_ptr(), m,
                      engine="ozaki")
            assert gpu.last_error()[0] == 0, gpu.last_error()
            outs.append(d.cpu().numpy())
        finally:
            gpu.lib.mwblas_set_residue_tc(prev)
    np.testing.assert_array_equal(outs[0], outs[1])
