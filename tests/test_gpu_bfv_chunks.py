"""BFV products through the chunked lanes and the fused combine: around the
smallest batch that takes two chunks, one to three lanes, 45-bit primes, wider ones
and one kind beside the other, on the four-step kernels and below them."""
import numpy as np
import pytest

from conftest import Q45, Q50

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,qs,ps,count,lanes", [
    (12, Q45[:2], Q45[2:5], 7, 2), (12, Q45[:2], Q45[2:5], 9, 2), (12, Q45[:2], Q45[2:5], 8, 1),
    (13, Q50[:3], Q50[3:7], 9, 2), (10, Q50[:2], Q50[2:5], 8, 2), (14, Q45[:3], Q50[:4], 8, 3)])
def test_bfv_mul_chunks(sg, oracle, log_n, qs, ps, count, lanes):
    lib, n, L = sg.lib(), 1 << log_n, len(qs)
    t = 65537
    rns, ctx = oracle.Rns(log_n, qs + ps), sg.Context(log_n, qs, t, ps=ps)
    aux = list(range(L, L + len(ps)))
    sg.check(lib.shg_context_set_ks_lanes(ctx.h, lanes))
    a = oracle.uniform_limbs(21, qs, n, 2 * count).reshape(count, 2, L, n)
    b = oracle.uniform_limbs(22, qs, n, 2 * count).reshape(count, 2, L, n)
    da, db = sg.DeviceBuffer.from_array(a), sg.DeviceBuffer.from_array(b)
    out = sg.DeviceBuffer(count * 3 * L * n * 8)
    for _ in range(2):  # the second call on streams and scratch of the first
        sg.check(lib.shg_bfv_mul(ctx.h, out.ptr, da.ptr, db.ptr, count, L, None))
    sg.check(lib.shg_device_synchronize())
    got = out.download((count, 3, L, n))
    for i in range(count):
        assert np.array_equal(got[i], rns.bfv_mul(L, aux, t, a[i], b[i])), i
