"""The grouped GEMM's tensor-core tiles (8 x 16 outputs, two columns at a time, k in
steps of 16, copies of 64, accumulators of 256, splits from 4096) at their edges,
against the binary128 oracle, in batches that mix every shape.

Operands are rounded to 116 bits of their row or column maximum and the rest is
exact up to one rounding (16 2^-104 k |A| |B| allowed, as for the small tiles of
the single product).
"""
import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (2, 3, 15), (15, 16, 16), (16, 17, 17), (17, 5, 63), (33, 1, 64), (1, 33, 65), (16, 16, 128),
          (31, 20, 129), (48, 47, 1), (8, 16, 256), (9, 17, 257), (7, 15, 513), (5, 6, 4096), (3, 18, 4100), (9, 4, 9000), (20, 20, 0), (127, 40, 50)]


def batch(gpu, oracle, rng, kind, ta, tb):
    import torch
    al, be = mwb.random_dd(rng, ()) + np.array([1.5, 0.0]), mwb.random_dd(rng, ())
    betas = [be, np.zeros(2), np.array([1.0, 0.0])]
    inst = []
    for q, (m, n, k) in enumerate(SHAPES):
        A = mwb.dd_matrix(rng, m if ta == "N" else k, k if ta == "N" else m, (m if ta == "N" else k) + 1, fill=0.5)
        B = mwb.dd_matrix(rng, k if tb == "N" else n, n if tb == "N" else k, (k if tb == "N" else n) + 2, fill=0.5)
        C = mwb.dd_matrix(rng, m, n, m + 1, fill=9.0)
        if kind == "spread":
            A *= 2.0 ** rng.integers(-60, 60, A.shape[:2])[..., None]
            B *= 2.0 ** rng.integers(-60, 60, B.shape[:2])[..., None]
        elif kind == "zeros":
            A[rng.random(A.shape[:2]) < 0.6] = 0.0
            B[rng.random(B.shape[:2]) < 0.6] = 0.0
            C[rng.random(C.shape[:2]) < 0.5] = 0.0
        elif kind == "signs":                      # limb sums at their largest, both signs
            A[..., 0], A[..., 1] = -np.abs(A[..., 0]), np.abs(A[..., 1])
            B[..., 0] = np.abs(B[..., 0])
        inst.append((m, n, k, A, B, C, al if q % 3 else np.array([1.0, 0.0]), betas[q % 3]))
    dev = [[torch.from_numpy(np.ascontiguousarray(x) if x.size else np.zeros((1, 1, 2))).cuda() for x in t[3:6]]
           for t in inst]
    col = lambda i: [t[i] for t in inst]
    prev = gpu.lib.mwblas_set_grouped_tile(16)
    try:
        rc = gpu.mgemm_grouped([ta] * len(inst), [tb] * len(inst), col(0), col(1), col(2), col(6),
                               [d[0].data_ptr() for d in dev], [t[3].shape[1] for t in inst],
                               [d[1].data_ptr() for d in dev], [t[4].shape[1] for t in inst], col(7),
                               [d[2].data_ptr() for d in dev], [t[5].shape[1] for t in inst])
    finally:
        gpu.lib.mwblas_set_grouped_tile(prev)
    assert rc == 0, gpu.last_error()
    return inst, [d[2].cpu().numpy() for d in dev]


@pytest.mark.parametrize("kind", ["plain", "spread", "zeros", "signs"])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T")])
def test_limb_tiles(gpu, oracle, rng, ta, tb, kind):
    inst, got = batch(gpu, oracle, rng, kind, ta, tb)
    for (m, n, k, A, B, C, al, be), out in zip(inst, got):
        want = C.copy()
        oracle.qgemm(ta, tb, m, n, k, al, A, A.shape[1], B, B.shape[1], be, want, C.shape[1])
        assert np.array_equal(out[:, m:], C[:, m:])
        a, b = A[:, : m if ta == "N" else k], B[:, : k if tb == "N" else n]
        prod = k * orc.dd_absmax(a) * orc.dd_absmax(b) if k else 0.0
        op = orc.dd_abs(al) * prod + orc.dd_abs(be) * orc.dd_absmax(C[:, :m])
        err = np.abs((out[:, :m, 0] - want[:, :m, 0]) + (out[:, :m, 1] - want[:, :m, 1])).max()
        assert err <= 16 * orc.EPS_DD * op, (m, n, k, err / op / orc.EPS_DD)


def test_limb_tiles_nonfinite(gpu, rng):
    import torch
    m, n, k = 35, 20, 70
    A, B, C = mwb.dd_matrix(rng, m, k), mwb.dd_matrix(rng, k, n), mwb.dd_matrix(rng, m, n)
    A[40, 17] = (np.inf, 0.0)
    C[3, 2] = (np.nan, 0.0)
    d = [torch.from_numpy(x).cuda() for x in (A, B, C)]
    one = np.array([1.0, 0.0])
    assert gpu.mgemm_grouped(["N"], ["N"], [m], [n], [k], [one], [d[0].data_ptr()], [m], [d[1].data_ptr()], [k], [one],
                             [d[2].data_ptr()], [m]) == 0
    off = np.isnan(d[2].cpu().numpy()[..., 0])   # [column, row]
    want = np.zeros((n, m), bool)
    want[:, 17] = True
    want[3, 2] = True
    assert np.array_equal(off, want)
