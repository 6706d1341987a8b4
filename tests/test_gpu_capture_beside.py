"""Calls on a context while another call of it is being captured: the capture holds
the side streams of its lanes until it ends, the calls beside it go without them."""
import ctypes

import numpy as np
import pytest

from conftest import Q50

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes,between", [(2, "rotate"), (4, "mul_relin"), (3, "rotate")])
def test_call_beside_a_capture(sg, oracle, lanes, between):
    lib, log_n, qs, count = sg.lib(), 12, Q50[:2], 80
    n, L, log_bs = 1 << log_n, len(qs), [20, 20]
    power = pow(5, 3, 2 * n)
    rns, ctx = oracle.Rns(log_n, qs), sg.Context(log_n, qs)
    rows = [oracle.uniform_limbs(s, qs, n, rns.gadget_dim(log_bs)) for s in (3, 4)]
    key, relin = sg.Key(ctx, log_bs, power, *rows), sg.Key(ctx, log_bs, 1, *rows)
    a = oracle.uniform_limbs(1, qs, n, 2 * count).reshape(count, 2, L, n)
    da = sg.DeviceBuffer.from_array(a)
    outs = [sg.DeviceBuffer.from_array(np.zeros_like(a)) for _ in range(2)]
    sg.check(lib.shg_context_set_ks_lanes(ctx.h, lanes))
    sg.check(lib.shg_context_set_chunk(ctx.h, 16))

    def call(kind, out, s):
        if kind == "mul_relin":
            sg.check(lib.shg_bgv_mul_relin(ctx.h, relin.h, out.ptr, da.ptr, da.ptr, count, s))
        else:
            sg.check(lib.shg_bgv_rotate(ctx.h, key.h, out.ptr, da.ptr, count, s))

    call("mul_relin", outs[0], None)  # scratch for either, and the side streams
    products = outs[0].download(a.shape)
    call("rotate", outs[0], None)
    rotations = outs[0].download(a.shape)
    for i in (0, count - 1):
        sub = np.stack([rns.substitute(a[i, c], power) for c in (0, 1)])
        assert np.array_equal(rotations[i], rns.galois(sub, *rows, log_bs))
    for o in outs:
        o.upload(np.zeros_like(a))

    s, other, g = (ctypes.c_void_p() for _ in range(3))
    sg.check(lib.shg_stream_create(ctypes.byref(s)))
    sg.check(lib.shg_stream_create(ctypes.byref(other)))
    sg.check(lib.shg_graph_capture_begin(s))
    call("rotate", outs[0], s)
    call(between, outs[1], other)
    sg.check(lib.shg_graph_capture_end(s, ctypes.byref(g)))
    want = products if between == "mul_relin" else rotations
    assert np.array_equal(outs[1].download(a.shape, other), want)
    sg.check(lib.shg_graph_launch(g, s))
    sg.check(lib.shg_stream_synchronize(s))
    assert np.array_equal(outs[0].download(a.shape), rotations)
    call("rotate", outs[1], other)  # on all lanes again
    assert np.array_equal(outs[1].download(a.shape, other), rotations)
    sg.check(lib.shg_graph_destroy(g))
