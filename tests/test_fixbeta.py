"""CPU check of beta C in the reconstruction's fixed-point update
(csrc/fixbeta.cuh, compiled for the host) against exact rationals: C keeps 2^-127
of itself whatever the gap between its limbs, and a sum with it its other term to
2^-158 of C (beta = 1) or 2^-122 (a general beta, from the product)."""
import ctypes as C
import math
import os
import random
import subprocess
import tempfile
from fractions import Fraction as F

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
U, D = C.c_uint32, C.c_double


@pytest.fixture(scope="module")
def fb():
    so = os.path.join(tempfile.mkdtemp(), "libfb.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "fixbeta_harness.cpp"), "-o",
                    so], check=True)
    return C.CDLL(so)


def add(fb, a, ea, na, c, b, one):
    w, e, neg = (U * 6)(*[(a >> (32 * t)) & 0xFFFFFFFF for t in range(6)]), C.c_int(ea), U(na)
    ok = fb.fb_add(w, C.byref(e), C.byref(neg), D(c[0]), D(c[1]), D(b[0]), D(b[1]), one)
    value = sum(int(x) << (32 * t) for t, x in enumerate(w))
    return ok, F(-value if neg.value else value) * F(2) ** e.value


def double_double(rng, gap):
    hi = rng.uniform(1.0, 2.0) * 2.0 ** rng.randrange(-300, 300) * rng.choice([-1, 1])
    lo = math.ldexp(rng.uniform(0.5, 1.0) * rng.choice([-1, 1]), math.frexp(hi)[1] - gap) if gap else 0.0
    return (hi, lo) if hi + lo == hi else (hi, lo / 2)


@pytest.mark.parametrize("one", [0, 1])
def test_beta_c(fb, one):
    rng = random.Random(6)
    for _ in range(6000):
        c = double_double(rng, rng.choice([0, 53, 54, 55, 60, 64, 65, 70, 74, 80, 84, 85, 96, 107, 117, 126, 127, 200]))
        b = (1.0, 0.0) if one else double_double(rng, rng.choice([0, 54, 60, 74]))
        bc = (F(b[0]) + F(b[1])) * (F(c[0]) + F(c[1]))
        # the other term: up to 160 bits at or below C, down to its 2^-150
        a, na = rng.getrandbits(rng.choice([1, 53, 107, 160])), rng.randrange(2)
        ea = math.frexp(float(abs(bc)))[1] - a.bit_length() - rng.choice([0, 5, 60, 100, 118, 150])
        ok, got = add(fb, a, ea, na, c, b, one)
        assert ok == 1
        want = F(-a if na else a) * F(2) ** ea + bc
        cut = F(2) ** -126 + (F(2) ** -158 if one else F(2) ** -122)     # of C itself, and in the sum
        if one and (c[1] == 0.0 or abs(F(c[1])) >= F(2) ** -73 * abs(F(c[0]))):
            cut = F(2) ** -156                                           # every bit of C is held
        assert abs(got - want) <= cut * abs(bc) + F(2) ** ea             # and a unit of the other term


def test_what_the_general_path_takes(fb):
    for c in ((0.0, float("inf")), (float("inf"), 0.0), (1.0, 0.25), (1.0, float("nan")), (2.0 ** -1000, 0.0)):
        assert add(fb, 5, 0, 0, c, (1.0, 0.0), 1) == (0, 5)
    assert add(fb, 5, 0, 0, (0.0, 0.0), (1.0, 0.0), 1) == (1, 5)
    assert add(fb, 5, 0, 0, (-0.0, 0.0), (3.0, 0.0), 0) == (1, 5)
    assert add(fb, 5, 0, 0, (1.5, 0.0), (0.0, 0.0), 0) == (1, 5)          # beta zero
