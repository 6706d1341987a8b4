"""The word kernels of the wire format against the oracle at their edges: one
tile of less than 1024 values, exactly one, several; 17- to 60-bit values; more
polynomials than the grid has rows."""
import numpy as np
import pytest

from conftest import Q45, Q50, Q60

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,qs,count", [(6, [65537], 5000), (9, [65537, Q50[0]], 3),
                                            (10, Q45[:3], 40), (11, [65537], 700),
                                            (12, [Q60], 2), (15, Q50[:2], 1)])
def test_wire_words(sg, oracle, log_n, qs, count):
    lib, n, L = sg.lib(), 1 << log_n, len(qs)
    x = oracle.uniform_limbs(40 + log_n, qs, n, count)
    x[0, :, 0] = np.array(qs, np.uint64) - np.uint64(1)
    primes = [oracle.Prime(q, log_n) for q in qs]
    want = np.concatenate([primes[l].serialize(x[c, l]) for c in range(count) for l in range(L)])
    ctx = sg.Context(log_n, qs)
    d, buf, back = (sg.DeviceBuffer.from_array(x), sg.DeviceBuffer(want.size + 16),
                    sg.DeviceBuffer(x.nbytes))
    sg.check(lib.shg_poly_serialize(ctx.h, buf.ptr, d.ptr, count, L, None))
    got = np.empty(want.size, np.uint8)
    sg.check(lib.shg_memcpy_d2h(got.ctypes.data, buf.ptr, got.nbytes, None))
    sg.synchronize()
    assert np.array_equal(got, want)
    sg.check(lib.shg_poly_deserialize(ctx.h, back.ptr, buf.ptr, count, L, None))
    assert np.array_equal(back.download(x.shape), x)
