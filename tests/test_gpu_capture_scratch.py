"""Captured calls of batched operations in scratch that holds one lane of plain
chunks but not what the call would take outside a capture (more lanes, larger
chunks, the sampler's records): the capture goes through with what is there, and
its graph gives the result of the call made outside one."""
import ctypes

import numpy as np
import pytest

from conftest import Q45, Q50

pytestmark = pytest.mark.gpu


def _captured(sg, call, out, shape):
    """The result of call(stream) as a graph, with `out` cleared before its launch."""
    lib, s, g = sg.lib(), ctypes.c_void_p(), ctypes.c_void_p()
    out.upload(np.zeros(shape, np.uint64))
    sg.check(lib.shg_stream_create(ctypes.byref(s)))
    sg.check(lib.shg_graph_capture_begin(s))
    try:
        call(s)
    finally:
        end = lib.shg_graph_capture_end(s, ctypes.byref(g))
    sg.check(end)
    sg.check(lib.shg_graph_launch(g, s))
    sg.check(lib.shg_stream_synchronize(s))
    got = out.download(shape)
    sg.check(lib.shg_graph_destroy(g))
    return got


def _batch(sg, oracle, qs, n, shape, seed):
    x = oracle.uniform_limbs(seed, qs, n, int(np.prod(shape[:-2]))).reshape(shape)
    return sg.DeviceBuffer.from_array(x)


@pytest.mark.parametrize("qs,chunk,warm,count", [
    (Q50[:2], 0, 16, 64),   # sixteen a chunk on one lane; 32 on two outside a capture
    (Q50[:2], 4, 4, 13), (Q50[:5], 3, 3, 8)])
def test_rotations(sg, oracle, qs, chunk, warm, count):
    lib, log_n, L = sg.lib(), 12, len(qs)
    n, log_bs = 1 << log_n, [20] * L
    power, k = pow(5, 2, 2 * n), 3 * L
    rows = [oracle.uniform_limbs(s, qs, n, k) for s in (3, 4)]
    shape = (count, 2, L, n)
    ct, out = _batch(sg, oracle, qs, n, shape, 1), sg.DeviceBuffer(count * 2 * L * n * 8)
    free = sg.Context(log_n, qs)
    key = sg.Key(free, log_bs, power, *rows)
    sg.check(lib.shg_bgv_rotate(free.h, key.h, out.ptr, ct.ptr, count, None))
    want = out.download(shape)

    ctx = sg.Context(log_n, qs)
    key, relin = sg.Key(ctx, log_bs, power, *rows), sg.Key(ctx, log_bs, 1, *rows)
    if chunk:  # opens the side streams in no more scratch than the warm-up's
        sg.check(lib.shg_context_set_chunk(ctx.h, 1))
        sg.check(lib.shg_bgv_mul_relin(ctx.h, relin.h, out.ptr, ct.ptr, ct.ptr, 2, None))
    sg.check(lib.shg_context_set_chunk(ctx.h, chunk))
    sg.check(lib.shg_bgv_rotate(ctx.h, key.h, out.ptr, ct.ptr, warm, None))
    got = _captured(sg, lambda s: sg.check(
        lib.shg_bgv_rotate(ctx.h, key.h, out.ptr, ct.ptr, count, s)), out, shape)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("qs,count", [(Q50[:2], 64), (Q45[:6], 50)])
def test_products(sg, oracle, qs, count):
    lib, log_n, L = sg.lib(), 12, len(qs)
    n, log_bs, k = 1 << log_n, [20] * L, 3 * L
    rows = [oracle.uniform_limbs(s, qs, n, k) for s in (3, 4)]
    shape = (count, 2, L, n)
    a, b = (_batch(sg, oracle, qs, n, shape, s) for s in (1, 2))
    out = sg.DeviceBuffer(count * 2 * L * n * 8)

    def product(ctx, key, m, s=None):
        sg.check(lib.shg_bgv_mul_relin(ctx.h, key.h, out.ptr, a.ptr, b.ptr, m, s))

    free = sg.Context(log_n, qs)
    product(free, sg.Key(free, log_bs, 1, *rows), count)
    want = out.download(shape)
    ctx = sg.Context(log_n, qs)
    key = sg.Key(ctx, log_bs, 1, *rows)
    # two lanes of sixteen ciphertexts' digit transforms and the batch's components
    sg.check(lib.shg_context_reserve(ctx.h, (32 * k + count) * L * n * 8))
    product(ctx, key, 17)
    got = _captured(sg, lambda s: product(ctx, key, count, s), out, shape)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("pir", [False, True])
def test_expansion(sg, oracle, pir):
    lib, log_n, levels, log_b, count, q = sg.lib(), 10, 4, 15, 3, 1152921504606830593
    n, dim, items = 1 << log_n, 4, 11
    rows = [[oracle.uniform_limbs(7 + 2 * j + c, [q], n, dim) for c in (0, 1)]
            for j in range(levels)]
    ct = _batch(sg, oracle, [q], n, (count, 2, 1, n), 1)
    db = _batch(sg, oracle, [q], n, (items, 1, n), 2)
    shape = (count, 2, n) if pir else (count, 1 << levels, 2, n)
    out = sg.DeviceBuffer(int(np.prod(shape)) * 8)

    def call(ctx, arr, m, s=None):
        if pir:
            sg.check(lib.shg_pir_expand_absorb(ctx.h, arr, levels, db.ptr, items, out.ptr, ct.ptr,
                                               m, s))
        else:
            sg.check(lib.shg_oblivious_expand(ctx.h, arr, levels, out.ptr, ct.ptr, m, s))

    def made():
        ctx = sg.Context(log_n, [q])
        keys = [sg.Key(ctx, [log_b], (n >> j) + 1, *rows[j]) for j in range(levels)]
        return ctx, keys, (ctypes.c_void_p * levels)(*[k.h for k in keys])

    ctx, keys, arr = made()
    call(ctx, arr, count)
    want = out.download(shape)
    ctx, keys, arr = made()
    # one lane of all members of the last level, and the expanded blocks
    members = count << (levels - 1)
    blocks = (count * 2 << levels) if pir else 0
    sg.check(lib.shg_context_reserve(ctx.h, (levels + members * (3 + dim) + blocks) * n * 8))
    call(ctx, arr, 2)
    got = _captured(sg, lambda s: call(ctx, arr, count, s), out, shape)
    assert np.array_equal(got, want)


def test_bfv_products(sg, oracle):
    lib, log_n, qs, ps, count = sg.lib(), 12, Q45[:2], Q45[2:5], 9
    n, L = 1 << log_n, 2
    a, b = (_batch(sg, oracle, qs, n, (count, 2, L, n), s) for s in (1, 2))
    shape = (count, 3, L, n)
    out = sg.DeviceBuffer(int(np.prod(shape)) * 8)

    def product(ctx, m, s=None):
        sg.check(lib.shg_bfv_mul(ctx.h, out.ptr, a.ptr, b.ptr, m, L, s))

    product(sg.Context(log_n, qs, ps=ps), count)
    want = out.download(shape)
    ctx = sg.Context(log_n, qs, ps=ps)
    sg.check(lib.shg_context_set_chunk(ctx.h, 1))
    product(ctx, 8)  # opens the side stream: two lanes of one pair
    sg.check(lib.shg_context_set_chunk(ctx.h, 4))
    product(ctx, 4)  # one lane of four
    got = _captured(sg, lambda s: product(ctx, count, s), out, shape)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("encrypt", [False, True])
def test_sampler(sg, oracle, encrypt):
    """Warmed with one limb (up to 4096 uniform words: no records), captured with two."""
    lib, log_n, qs, count, variance = sg.lib(), 12, Q45[:2], 8, 8
    n, L = 1 << log_n, 2
    seeds = np.random.RandomState(3).randint(0, 256, (count, 32)).astype(np.uint8)
    dseeds = sg.DeviceBuffer(seeds.nbytes)
    sg.check(lib.shg_memcpy_h2d(dseeds.ptr, seeds.ctypes.data, seeds.nbytes, None))
    secret = _batch(sg, oracle, qs, n, (L, n), 1)
    m = _batch(sg, oracle, qs, n, (count, L, n), 2)
    shape = (count, 2, L, n)
    out = sg.DeviceBuffer(int(np.prod(shape)) * 8)

    def call(ctx, limbs, s=None):
        if encrypt:
            sg.check(lib.shg_bgv_encrypt(ctx.h, out.ptr, secret.ptr, m.ptr, dseeds.ptr, limbs,
                                         count, variance, s))
        else:  # errors behind the uniform polynomials
            sg.check(lib.shg_sample_uniform_error(ctx.h, out.ptr, out.ptr + count * L * n * 8,
                                                  dseeds.ptr, limbs, count, variance, s))

    call(sg.Context(log_n, qs), L)
    want = out.download(shape)
    ctx = sg.Context(log_n, qs)
    call(ctx, 1)
    sg.check(lib.shg_context_set_chunk(ctx.h, count // 2))  # as many limbs at once as before
    got = _captured(sg, lambda s: call(ctx, L, s), out, shape)
    assert np.array_equal(got, want)
