"""Device memory of a key's 32-bit form: taken by the first batch with one key that
gains from it, not by the key's creation or by batches with a key per member, and
given back when an allocation fails, but not under a graph that holds it."""
import ctypes

import numpy as np
import pytest

from conftest import Q50

pytestmark = pytest.mark.gpu

SLACK = 48 << 20  # granularity of the driver's allocations


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _refused(sg):
    """An allocation that no device can hold."""
    p = ctypes.c_void_p()
    assert sg.lib().shg_device_alloc(1 << 50, ctypes.byref(p)) != 0


def test_form_is_made_by_its_first_batch_and_given_back(sg, oracle):
    lib, log_n, qs, count = sg.lib(), 15, Q50, 2
    n, L, log_bs, k = 1 << log_n, len(qs), [20] * len(qs), 36
    ctx = sg.Context(log_n, qs)
    sg.check(lib.shg_context_reserve(ctx.h, 1 << 30))
    rows = 16 * k * L * n
    comps = [oracle.uniform_limbs(40 + i, qs, n, k) for i in range(3)]
    a = oracle.uniform_limbs(1, qs, n, 2 * count).reshape(count, 2, L, n)
    b = oracle.uniform_limbs(2, qs, n, 2 * count).reshape(count, 2, L, n)
    da, db, out = (sg.DeviceBuffer.from_array(x) for x in (a, b, np.zeros_like(a)))
    start = _free()
    keys = [sg.Key(ctx, log_bs, 1, comps[i], comps[i + 1]) for i in (0, 1)]
    assert start - _free() < 2 * rows + SLACK

    want = []  # per key, through the entry point that takes one per member
    for key in keys:
        both = (ctypes.c_void_p * 2)(key.h, key.h)
        sg.check(lib.shg_bgv_mul_relin_multikey(ctx.h, both, out.ptr, da.ptr, db.ptr, count,
                                                None))
        want.append(out.download(a.shape))
    mixed = (ctypes.c_void_p * 2)(keys[0].h, keys[1].h)
    sg.check(lib.shg_bgv_mul_relin_multikey(ctx.h, mixed, out.ptr, da.ptr, db.ptr, count, None))
    assert np.array_equal(out.download(a.shape), np.stack([want[0][0], want[1][1]]))
    without = _free()
    assert start - without < 2 * rows + SLACK

    def product(i, s=None):
        sg.check(lib.shg_bgv_mul_relin(ctx.h, keys[i].h, out.ptr, da.ptr, db.ptr, count, s))

    for _ in range(2):  # made, given back, made again
        for i in (0, 1):
            product(i)
            assert np.array_equal(out.download(a.shape), want[i])
        assert without - _free() >= 3 * rows  # 1.5 times the rows of each key
        _refused(sg)
        assert without - _free() < SLACK

    # an oversized workspace gives both forms back too, and the next batch's takes its place
    product(0)
    with pytest.raises(sg.ShgError):
        sg.check(lib.shg_context_reserve(ctx.h, 1 << 50))
    assert without - _free() < SLACK
    product(1)
    assert np.array_equal(out.download(a.shape), want[1])

    # a graph keeps the form of its key; the other key's goes
    product(0)
    s, g = ctypes.c_void_p(), ctypes.c_void_p()
    sg.check(lib.shg_stream_create(ctypes.byref(s)))
    sg.check(lib.shg_graph_capture_begin(s))
    product(0, s)
    sg.check(lib.shg_graph_capture_end(s, ctypes.byref(g)))
    both = _free()
    _refused(sg)
    assert 1.4 * rows < _free() - both < 1.6 * rows
    out.upload(np.zeros_like(a))
    sg.check(lib.shg_graph_launch(g, s))
    sg.check(lib.shg_stream_synchronize(s))
    assert np.array_equal(out.download(a.shape), want[0])
    sg.check(lib.shg_graph_destroy(g))
    keys[0].close()
    keys[1].close()
    assert _free() >= start - SLACK


def test_a_capture_does_not_make_the_form(sg, oracle):
    """A key whose first call is captured runs on its rows; another context's key
    gets its form meanwhile, in the same thread, and the capture stays whole."""
    lib, log_n, qs, count = sg.lib(), 12, Q50, 5
    n, L, log_bs = 1 << log_n, len(qs), [20] * len(qs)
    rns = oracle.Rns(log_n, qs)
    kb, ka = (oracle.uniform_limbs(s, qs, n, rns.gadget_dim(log_bs)) for s in (3, 4))
    a = oracle.uniform_limbs(1, qs, n, 2 * count).reshape(count, 2, L, n)
    want = rns.mul_relin_batch(a, a, kb, ka, log_bs, threads=8)
    da = sg.DeviceBuffer.from_array(a)
    outs = [sg.DeviceBuffer(a.nbytes) for _ in range(2)]
    ctxs = [sg.Context(log_n, qs) for _ in range(2)]
    warm, keys = ([sg.Key(c, log_bs, 1, kb, ka) for c in ctxs] for _ in range(2))

    def product(i, key, s=None):
        sg.check(lib.shg_bgv_mul_relin(ctxs[i].h, key.h, outs[i].ptr, da.ptr, da.ptr, count, s))

    for i in (0, 1):
        product(i, warm[i])
        assert np.array_equal(outs[i].download(a.shape), want)
        outs[i].upload(np.zeros_like(a))
    s, g, other = (ctypes.c_void_p() for _ in range(3))
    sg.check(lib.shg_stream_create(ctypes.byref(s)))
    sg.check(lib.shg_stream_create(ctypes.byref(other)))
    sg.check(lib.shg_graph_capture_begin(s))
    product(0, keys[0], s)
    product(1, keys[1], other)
    product(0, keys[0], s)
    sg.check(lib.shg_graph_capture_end(s, ctypes.byref(g)))
    assert np.array_equal(outs[1].download(a.shape, other), want)
    sg.check(lib.shg_graph_launch(g, s))
    sg.check(lib.shg_stream_synchronize(s))
    assert np.array_equal(outs[0].download(a.shape), want)
    sg.check(lib.shg_graph_destroy(g))
