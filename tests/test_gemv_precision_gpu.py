"""mgemv_ on long sums of equal sign beside one dominating product, against exact
integers.

An element of A is rounded to a unit of 2^-113 of its output's and chunk's largest
product, and a chunk is at most 2048 products: 2^-103 of the largest one if all
erred alike. Here they err at random, six standard deviations are
6 sqrt(2048 / 12) 2^-113 < 2^-106; what operands have below 2^-117 of their high
limb is less, the final rounding below 2^-106. Allowed: half a unit of
2^-104 sum |a x|.
"""
from fractions import Fraction as F

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Y = np.array([0.7312345, 0.7312345 * 2.0 ** -54 * 0.7])


def vector(rng, n, ones):
    """Double-doubles near 2^-40 with ones at the given places, and their exact sum."""
    a, b = rng.integers(1 << 52, 1 << 53, n), rng.integers(-(1 << 51), 1 << 51, n)
    hi, lo = a * 2.0 ** -92, b * 2.0 ** -146
    a[ones] = 0
    b[ones] = 0
    hi[ones], lo[ones] = 1.0, 0.0
    low = (1 << 26) - 1
    total = F((int((a >> 26).sum()) << 26) + int((a & low).sum())) / F(2) ** 92
    total += F((int((b >> 26).sum()) << 26) + int((b & low).sum())) / F(2) ** 146
    return np.stack([hi, lo], axis=-1), total + len(ones)


def units(got, want):
    return float(abs(F(float(got[0])) + F(float(got[1])) - want) / want * F(2) ** 104)


@pytest.mark.parametrize("place", [0, 37, 1999])
@pytest.mark.parametrize("trans,rows,length", [("N", 16384, 2000), ("N", 40, 16384), ("T", 40, 16384), ("T", 5003, 7001)])
def test_gemv(gpu, rng, trans, rows, length, place):
    import torch
    distinct = [vector(rng, length, np.array([place])) for _ in range(20)]
    A = torch.from_numpy(np.stack([d[0] for d in distinct])).cuda()[torch.arange(rows) % 20]   # [output, index]
    dA = A.transpose(0, 1).contiguous() if trans == "N" else A                                 # column-major
    m, n = (rows, length) if trans == "N" else (length, rows)
    dx = torch.from_numpy(Y).cuda().expand(length, 2).contiguous()
    dy = torch.zeros((rows, 2), dtype=torch.float64, device="cuda")
    one, zero = np.array([1.0, 0.0]), np.zeros(2)
    torch.cuda.synchronize()
    gpu.mgemv(trans, m, n, one, dA.data_ptr(), m, dx.data_ptr(), 1, zero, dy.data_ptr(), 1)
    assert gpu.last_error()[0] == 0, gpu.last_error()
    y = dy.cpu().numpy()
    want = [d[1] * (F(Y[0]) + F(Y[1])) for d in distinct]
    worst = max(units(y[r], want[r % 20]) for r in range(rows))
    assert worst <= 0.5, worst
