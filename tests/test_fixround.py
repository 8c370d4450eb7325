"""CPU check of the CRT reconstruction's fixed-point update and rounding
(csrc/fixround.cuh, compiled for the host) against exact integers."""
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
    so = os.path.join(tempfile.mkdtemp(), "libfr.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "fixround_harness.cpp"), "-o",
                    so], check=True)
    return C.CDLL(so)


def words(v, n):
    return (U * n)(*[(v >> (32 * t)) & 0xFFFFFFFF for t in range(n)])


def value(w):
    return sum(int(x) << (32 * t) for t, x in enumerate(w))


def some(rng, bits):
    """An integer below 2^bits: random, sparse, or with long runs of ones and zeros."""
    kind = rng.randrange(4)
    if kind == 0:
        return rng.getrandbits(bits)
    if kind == 1:
        return rng.getrandbits(bits) >> rng.randrange(bits)
    if kind == 2:
        return (1 << rng.randrange(bits)) - rng.randrange(2)
    return ((1 << bits) - 1) ^ ((1 << rng.randrange(bits)) - 1)


def test_products(fr):
    rng = random.Random(1)
    for _ in range(4000):
        t, a, b = some(rng, 160), some(rng, 128), some(rng, 128)
        p = (U * 5)()
        fr.fr_mul54(words(t, 5), words(a, 4), p)
        assert 0 <= (t * a >> 128) - value(p) <= 4          # three products below 2^128 dropped, and their carry
        fr.fr_mul44(words(a, 4), words(b, 4), p)
        assert 0 <= (a * b >> 96) - value(p) < 1 << 34       # the same, in units of 2^96


def test_sums(fr):
    rng = random.Random(2)
    for _ in range(6000):
        a, q = some(rng, 161), some(rng, 155)
        ea, eq = rng.randrange(-300, 300), 0
        eq = ea + rng.choice([0, 1, -1, 31, 32, 33, -64, 100, -100, 159, -161, 200, -250, rng.randrange(-170, 170)])
        na, nq = rng.randrange(2), rng.randrange(2)
        w, e, neg = words(a, 6), C.c_int(ea), U(na)
        fr.fr_add(w, C.byref(e), C.byref(neg), words(q, 5), eq, U(nq))
        got = Fraction(value(w) * (-1 if neg.value else 1)) * Fraction(2) ** e.value
        want = Fraction(-a if na else a) * Fraction(2) ** ea + Fraction(-q if nq else q) * Fraction(2) ** eq
        if a == 0:
            assert got == want
        else:
            assert e.value == max(ea, eq) and abs(got - want) < Fraction(2) ** e.value


def test_rounding(fr):
    rng = random.Random(3)
    for _ in range(8000):
        a, e, neg = some(rng, rng.choice([60, 100, 128, 160, 163])), rng.randrange(-500, 500), rng.randrange(2)
        hi, lo = C.c_double(), C.c_double()
        fr.fr_to_dd(words(a, 6), e, U(neg), C.byref(hi), C.byref(lo))
        hi, lo = hi.value, lo.value
        want = Fraction(-a if neg else a) * Fraction(2) ** e
        if a == 0:
            assert hi == lo == 0.0
            continue
        assert abs(Fraction(lo)) <= Fraction(2) ** (a.bit_length() + e - 54)   # half a unit of hi
        got = Fraction(hi) + Fraction(lo)
        # half a unit of lo, and what lies below the 128 bits taken
        ulp_lo = Fraction(2) ** (a.bit_length() + e - 54 - 53)
        assert abs(got - want) <= ulp_lo / 2 + Fraction(2) ** (a.bit_length() + e - 128)
