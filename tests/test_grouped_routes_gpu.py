"""Grouped products at the lines between the limb tiles, their waves and pieces, and
the square tiles: short k, instances of more lines than a wave holds (rows,
columns, both), and a k so long that a wave holds few lines. Against the binary128
oracle (16 units of 2^-104 k |A| |B|, as for the tiles alone); the scratch that a
call keeps stays below a wave (1 GiB) and what the square tiles' partials take.
"""
import threading

import numpy as np
import pytest

from conftest import mwb, orc

pytestmark = pytest.mark.gpu

WAVE = 1 << 19          # lines of up to 64 k


def on_thread(body):
    """On a thread of its own, whose plan starts empty."""
    failures = []

    def run():
        try:
            body()
        except BaseException as e:
            failures.append(e)

    t = threading.Thread(target=run)
    t.start()
    t.join()
    if failures:
        raise failures[0]


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "T")])
def test_short_k(gpu, oracle, rng, ta, tb):
    import torch
    shapes = [(m, n, k) for m, n in ((1, 1), (8, 16), (40, 48), (64, 64), (127, 130), (300, 40))
              for k in (0, 1, 7, 8, 9, 16, 17, 24, 25, 32)]
    al, be = mwb.random_dd(rng, ()) + np.array([1.5, 0.0]), mwb.random_dd(rng, ())
    inst = [(m, n, k, mwb.dd_matrix(rng, *((m, k) if ta == "N" else (k, m))),
             mwb.dd_matrix(rng, *((k, n) if tb == "N" else (n, k))), mwb.dd_matrix(rng, m, n)) for m, n, k in shapes]
    dev = [[torch.from_numpy(np.ascontiguousarray(x) if x.size else np.zeros((1, 1, 2))).cuda() for x in t[3:]]
           for t in inst]
    col, ptr, count = (lambda i: [t[i] for t in inst]), (lambda i: [d[i].data_ptr() for d in dev]), len(inst)
    lda = [max(1, m if ta == "N" else k) for m, n, k in shapes]
    ldb = [max(1, k if tb == "N" else n) for m, n, k in shapes]
    assert gpu.mgemm_grouped([ta] * count, [tb] * count, col(0), col(1), col(2), [al] * count, ptr(0), lda, ptr(1), ldb,
                             [be] * count, ptr(2), col(0)) == 0, gpu.last_error()
    for (m, n, k, A, B, C0), d, la, lb in zip(inst, dev, lda, ldb):
        want = oracle.qgemm(ta, tb, m, n, k, al, A, la, B, lb, be, C0.copy(), m)
        op = orc.dd_abs(al) * (k * orc.dd_absmax(A) * orc.dd_absmax(B) if k else 0.0)
        op += orc.dd_abs(be) * orc.dd_absmax(C0)
        assert orc.normwise_error(d[2].cpu().numpy(), want, op) <= 16 * orc.EPS_DD, (m, n, k)


@pytest.mark.parametrize("m,n,k", [(20, WAVE + 100000, 32), (WAVE + 3, 8, 40), (24, 140000, 300), (60, 1000000, 1),
                                   (9, 17, 70000), (600, 8, 70000)])
def test_more_lines_than_a_wave(gpu, oracle, rng, m, n, k):
    import torch

    def values(cols, rows):
        hi = torch.rand((cols, rows), dtype=torch.float64, device="cuda") * 2 - 1
        lo = hi * (torch.rand((cols, rows), dtype=torch.float64, device="cuda") * 2 - 1) * 2.0 ** -54
        s = hi + lo
        return torch.stack([s, lo - (s - hi)], dim=-1)

    torch.manual_seed(int(rng.integers(1 << 30)))
    A, B, C = values(k, m), values(n, k), values(n, m)
    C0 = C.clone()
    al, be = mwb.random_dd(rng, ()) + np.array([1.5, 0.0]), mwb.random_dd(rng, ())
    torch.cuda.synchronize()
    free = []

    def body():
        free.append(torch.cuda.mem_get_info()[0])
        rc = gpu.mgemm_grouped(["N"], ["N"], [m], [n], [k], [al], [A.data_ptr()], [m], [B.data_ptr()], [k], [be],
                               [C.data_ptr()], [m])
        assert rc == 0, gpu.last_error()
        free.append(torch.cuda.mem_get_info()[0])

    on_thread(body)
    assert free[0] - free[1] <= (1 << 30) + (64 << 20)
    # every row and column of the output, in samples that cross the cuts
    rows = np.unique(np.concatenate([np.arange(min(m, 8)), rng.integers(0, m, 12), [m - 1]]))
    cols = np.unique(np.concatenate([np.arange(min(n, 8)), rng.integers(0, n, 12), [n - 1]]))
    rows, cols = (np.unique(np.concatenate([v, w[w < s]])) for v, s, w in
                  ((rows, m, WAVE // 2 + np.arange(-2, 2)), (cols, n, WAVE // 2 + np.arange(-2, 2))))
    a, b = A[:, rows].cpu().numpy(), B[cols].cpu().numpy()
    want = C0[cols][:, rows].cpu().numpy()
    oracle.qgemm("N", "N", len(rows), len(cols), k, al, np.ascontiguousarray(a), len(rows), np.ascontiguousarray(b), k,
                 be, want, len(rows))
    got = C[cols][:, rows].cpu().numpy()
    err = np.abs((got[..., 0] - want[..., 0]) + (got[..., 1] - want[..., 1])).max()
    assert err <= 16 * orc.EPS_DD * (orc.dd_abs(al) * k + orc.dd_abs(be))
    # and the whole of it in 64 bits
    for j in range(0, n, 1 << 17):
        ref = al[0] * (B[j:j + (1 << 17), :, 0] @ A[..., 0]) + be[0] * C0[j:j + (1 << 17), :, 0]
        assert torch.max(torch.abs(C[j:j + (1 << 17), :, 0] - ref)).item() <= 1e-13 * k
