"""Kernels launched behind one another without a drain between them: a chain of calls
in which every call reads what the one before it wrote, and overwrites what that one
read, run at once and from a captured graph.  Exact arithmetic: equality."""
import ctypes

import numpy as np
import pytest

from conftest import Q45, Q50

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,qs,count", [
    (11, Q45[:2], 2), (12, Q45[:2], 3), (14, Q45, 1), (14, Q45[:4], 2), (13, Q50[:5], 35)])
def test_chained_calls(sg, oracle, log_n, qs, count):
    lib, n, L, log_bs = sg.lib(), 1 << log_n, len(qs), [20] * len(qs)
    rns, ctx = oracle.Rns(log_n, qs), sg.Context(log_n, qs)
    k = rns.gadget_dim(log_bs)
    kb, ka = (oracle.uniform_limbs(s, qs, n, k) for s in (3, 4))
    key = sg.Key(ctx, log_bs, 1, kb, ka)
    a = oracle.uniform_limbs(1, qs, n, 2 * count).reshape(count, 2, L, n)
    b = oracle.uniform_limbs(2, qs, n, 2 * count).reshape(count, 2, L, n)
    x, db, y = (sg.DeviceBuffer.from_array(v) for v in (a, b, np.zeros_like(a)))

    def chain(s):  # x -> y -> x, NTT round trips in place between
        for src, dst in ((x, y), (y, x)):
            sg.check(lib.shg_bgv_mul_relin(ctx.h, key.h, dst.ptr, src.ptr, db.ptr, count, s))
            sg.check(lib.shg_ntt_inverse(ctx.h, dst.ptr, 2 * count, L, s))
            sg.check(lib.shg_ntt_forward(ctx.h, dst.ptr, 2 * count, L, s))

    want = a
    for _ in range(2):
        want = rns.mul_relin_batch(want, b, kb, ka, log_bs, threads=8)
    chain(None)
    assert np.array_equal(x.download(a.shape), want)

    s, g = ctypes.c_void_p(), ctypes.c_void_p()
    sg.check(lib.shg_stream_create(ctypes.byref(s)))
    sg.check(lib.shg_graph_capture_begin(s))
    chain(s)
    sg.check(lib.shg_graph_capture_end(s, ctypes.byref(g)))
    for _ in range(2):  # each replay goes on from the last one's result
        sg.check(lib.shg_graph_launch(g, s))
        for _ in range(2):
            want = rns.mul_relin_batch(want, b, kb, ka, log_bs, threads=8)
    sg.check(lib.shg_stream_synchronize(s))
    assert np.array_equal(x.download(a.shape), want)
    sg.check(lib.shg_graph_destroy(g))
