"""CPU check of the reconstruction's sums with zero terms (csrc/fixround.cuh,
compiled for the host): a zero term in a coarser frame leaves the value alone."""
import ctypes as C
import os
import random
import subprocess
import tempfile
from fractions import Fraction

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
U = C.c_uint32


@pytest.fixture(scope="module")
def fr():
    so = os.path.join(tempfile.mkdtemp(), "libft.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "fixterm_harness.cpp"), "-o",
                    so], check=True)
    return C.CDLL(so)


def words(v, n):
    return (U * n)(*[(v >> (32 * t)) & 0xFFFFFFFF for t in range(n)])


@pytest.mark.parametrize("zero_term", [True, False])
def test_terms(fr, zero_term):
    rng = random.Random(4)
    for _ in range(2000):
        a, ea = rng.getrandbits(rng.randrange(1, 161)), rng.randrange(-200, 200)
        eq = ea + rng.choice([0, 1, -1, 31, 108, 160, 300, -40, -300])
        q, na, nq = 0 if zero_term else rng.getrandbits(155) | 1, rng.randrange(2), rng.randrange(2)
        w, e, neg = words(a, 6), C.c_int(ea), U(na)
        fr.fr_add_term(w, C.byref(e), C.byref(neg), words(q, 5), eq, U(nq))
        value = sum(int(x) << (32 * t) for t, x in enumerate(w))
        got = Fraction(-value if neg.value else value) * Fraction(2) ** e.value
        want = Fraction(-a if na else a) * Fraction(2) ** ea + Fraction(-q if nq else q) * Fraction(2) ** eq
        if zero_term or a == 0:
            assert got == want
        else:
            assert abs(got - want) < Fraction(2) ** max(ea, eq)
