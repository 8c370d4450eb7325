"""CPU check of how host threads learn of a device wait that gave up
(csrc/statusmirror.h, compiled for the host): two threads over one mirror."""
import ctypes as C
import os
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


class Watch:
    def __init__(self, lib):
        self.lib, self.p = lib, C.c_void_p(lib.watch_new())

    def begin(self, now):
        self.lib.watch_begin(self.p, C.c_uint64(now))

    def check(self, now):
        return self.lib.watch_check(self.p, C.c_uint64(now))


@pytest.fixture(scope="module")
def lib():
    so = os.path.join(tempfile.mkdtemp(), "libsm.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "statusmirror_harness.cpp"),
                    "-o", so], check=True)
    so = C.CDLL(so)
    so.watch_new.restype = C.c_void_p
    return so


def stamp(ns, code):
    return ns << 8 | code


def test_both_threads_of_a_failure_report_it(lib):
    a, b = Watch(lib), Watch(lib)
    a.begin(0)
    b.begin(0)
    now = stamp(1000, 3)              # a's kernel gives up, b's follows the device word
    assert a.check(now) == 3
    assert b.check(now) == 3          # although a has read it


def test_a_kernel_that_follows_an_old_word(lib):
    a, b = Watch(lib), Watch(lib)
    a.begin(0)
    b.begin(0)
    first = stamp(1000, 3)
    assert b.check(first) == 3
    b.begin(first)                    # the device word is not cleared yet: b's next kernel gives up and stamps
    assert a.check(first) == 3
    assert b.check(stamp(2000, 3)) == 3


def test_a_call_after_a_failure_is_clean(lib):
    a, b = Watch(lib), Watch(lib)
    a.begin(0)
    now = stamp(1000, 2)
    assert a.check(now) == 2
    for w in (a, b):
        w.begin(now)
        assert w.check(now) == 0


def test_unsynchronised_calls_keep_the_failure(lib):
    a = Watch(lib)
    a.begin(0)                        # queued, not waited for; its kernel gives up
    now = stamp(1000, 5)
    a.begin(now)                      # the next call
    assert a.check(now) == 5
    assert a.check(now) == 0
