"""mdot_ on long sums of equal sign beside one dominating product, against exact
integers.

One factor of a product is rounded to a unit of 2^-115 of its warp's block's
largest product, and a block is at most 4096 products: 2^-104 of the largest one
if all erred alike. Here they err at random, six standard deviations are
6 sqrt(4096 / 12) 2^-115 < 2^-108; what operands have below 2^-117 of their high
limb is less, the final rounding below 2^-106. Allowed: half a unit of
2^-104 sum |x y|.
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


@pytest.mark.parametrize("every", [None, 640, 1000003])
@pytest.mark.parametrize("n", [4099, 1000000, 10000000])
def test_dot(gpu, rng, n, every):
    import torch
    ones = np.array([0]) if every is None else np.arange(0, n, every)
    x, total = vector(rng, n, ones)
    dx, dy = torch.from_numpy(x).cuda(), torch.from_numpy(Y).cuda().expand(n, 2).contiguous()
    torch.cuda.synchronize()
    got = gpu.mdot(n, dx.data_ptr(), 1, dy.data_ptr(), 1)
    assert gpu.last_error()[0] == 0, gpu.last_error()
    assert units(got, total * (F(Y[0]) + F(Y[1]))) <= 0.5
