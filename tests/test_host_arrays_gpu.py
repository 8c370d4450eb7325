"""Host arrays: matrices at 16-byte boundaries are read by a kernel, others copied;
both give the same bits, and a call that fails after such a read was queued leaves
the next one right."""
import numpy as np
import pytest

from conftest import mwb

pytestmark = pytest.mark.gpu


def shifted(x):
    """A copy of x at an address of 8 past a 16-byte boundary."""
    buf = np.zeros(x.size + 4)
    off = 1 if buf.ctypes.data % 16 == 0 else 2
    out = buf[off:off + x.size].reshape(x.shape)
    out[...] = x
    assert out.ctypes.data % 16 == 8
    return out


@pytest.mark.parametrize("m,n,k,pad", [(1, 1, 1, 0), (3, 5, 7, 1), (65, 33, 129, 3), (513, 300, 257, 0)])
def test_aligned_and_shifted(gpu, rng, m, n, k, pad):
    A, B = mwb.dd_matrix(rng, m, k, m + pad, fill=5.0), mwb.dd_matrix(rng, k, n, k + pad, fill=7.0)
    C = mwb.dd_matrix(rng, m, n, m + pad, fill=9.0)
    al, be = mwb.random_dd(rng, ()), mwb.random_dd(rng, ())
    outs = []
    for a, b, c in ((A, B, C.copy()), (shifted(A), shifted(B), shifted(C))):
        gpu.mgemm("N", "N", m, n, k, al, a, m + pad, b, k + pad, be, c, m + pad)
        assert gpu.last_error()[0] == 0, gpu.last_error()
        outs.append(c)
    np.testing.assert_array_equal(outs[0], outs[1])
    assert np.all(outs[0][:, m:] == 9.0)


@pytest.mark.parametrize("allowed", [1, 2, 3])
def test_failure_after_a_queued_read(gpu, rng, allowed):
    n = 200
    A, B = mwb.dd_matrix(rng, n, n), mwb.dd_matrix(rng, n, n)
    want = np.zeros((n, n, 2))
    gpu.mgemm("N", "N", n, n, n, 1.0, A, n, B, n, 0.0, want, n)
    a, c = A.copy(), np.zeros((n, n, 2))
    gpu.lib.mwblas_debug_fail_alloc_after(allowed)
    try:
        gpu.mgemm("N", "N", n, n, n, 1.0, a, n, B, n, 0.0, c, n)
        assert gpu.last_error()[0] != 0
    finally:
        gpu.lib.mwblas_debug_fail_alloc_after(-1)
    del a                                  # nothing may still be reading it
    gpu.mgemm("N", "N", n, n, n, 1.0, A, n, B, n, 0.0, c, n)
    assert gpu.last_error()[0] == 0, gpu.last_error()
    np.testing.assert_array_equal(c, want)
