"""The key switch in three auxiliary 30-bit primes (csrc/ks32.cu) against the
oracle, bit for bit, at the edges of its range: every ring degree it takes, odd
limb and digit counts, batches below, at and between its ciphertext groups, both
prime sets, and digits and keys of the largest magnitude."""
import numpy as np
import pytest

from conftest import Q45, Q50

pytestmark = pytest.mark.gpu


def _key(sg, oracle, ctx, rns, qs, log_bs, power, seed, count):
    k = rns.gadget_dim(log_bs)
    # the batch is large enough to take the path (ks32_for in csrc/capi.cu)
    L = len(qs)
    assert (k * L - 0.45 * (3 * k + 6 * L) - 2 * L) * count * ctx.n >= 1.75e6
    kb = oracle.uniform_limbs(seed, qs, ctx.n, k)
    ka = oracle.uniform_limbs(seed + 1, qs, ctx.n, k)
    key = sg.Key(ctx, log_bs, power, kb, ka)
    # the 32-bit form is there: 6 words beside the two 64-bit rows
    elems = k * len(qs) * ctx.n
    assert sg.lib().shg_key_device_bytes(key.h) >= elems * (16 + 24)
    return key, kb, ka


@pytest.mark.parametrize("log_n,qs,log_b,count", [
    (12, Q50, 20, 2), (12, Q50, 20, 5), (13, Q50[:9], 17, 3), (13, Q45[:4], 20, 18),
    (14, Q45, 20, 2), (14, Q45, 20, 7), (14, Q45[:5], 9, 18), (14, Q50[:7], 22, 4),
    (15, Q50, 20, 1), (15, Q50, 20, 2), (15, Q50[:4], 21, 9), (12, Q45[:4], 3, 23),
    (13, Q45[:5], 2, 4)])
def test_ks32_matches_oracle(sg, oracle, log_n, qs, log_b, count):
    lib, n, L = sg.lib(), 1 << log_n, len(qs)
    log_bs = [log_b] * L
    rns, ctx = oracle.Rns(log_n, qs), sg.Context(log_n, qs)
    a = oracle.uniform_limbs(1, qs, n, 2 * count).reshape(count, 2, L, n)
    b = oracle.uniform_limbs(2, qs, n, 2 * count).reshape(count, 2, L, n)
    da, db, out = (sg.DeviceBuffer.from_array(x) for x in (a, b, np.zeros_like(a)))
    key, kb, ka = _key(sg, oracle, ctx, rns, qs, log_bs, 1, 3, count)
    sg.check(lib.shg_bgv_mul_relin(ctx.h, key.h, out.ptr, da.ptr, db.ptr, count, None))
    got = out.download(a.shape)
    assert np.array_equal(got, rns.mul_relin_batch(a, b, kb, ka, log_bs, threads=8))
    power = pow(5, 3, 2 * n)
    gkey, kb, ka = _key(sg, oracle, ctx, rns, qs, log_bs, power, 5, count)
    sg.check(lib.shg_bgv_rotate(ctx.h, gkey.h, out.ptr, da.ptr, count, None))
    got = out.download(a.shape)
    for i in range(0, count, 3):
        sub = np.stack([rns.substitute(a[i, c], power) for c in (0, 1)])
        assert np.array_equal(got[i], rns.galois(sub, kb, ka, log_bs)), i


@pytest.mark.parametrize("log_n,qs,log_b,count", [(14, Q45, 20, 2), (15, Q50, 20, 1),
                                                  (12, Q50[:6], 24, 9)])
def test_ks32_largest_sums(sg, oracle, log_n, qs, log_b, count):
    """Every digit near its mask and every key coefficient at +-q/2: the sums
    reach the bound that the choice of the auxiliary primes rests on."""
    lib, n, L = sg.lib(), 1 << log_n, len(qs)
    log_bs = [log_b] * L
    rns, ctx = oracle.Rns(log_n, qs), sg.Context(log_n, qs)
    k = rns.gadget_dim(log_bs)
    primes = [oracle.Prime(q, log_n) for q in qs]
    kb = np.empty((k, L, n), np.uint64)
    ka = np.empty((k, L, n), np.uint64)
    ct = oracle.uniform_limbs(9, qs, n, 3 * count).reshape(count, 3, L, n)
    for l, q in enumerate(qs):
        kb[:, l] = primes[l].ntt_fwd(np.full(n, q // 2, np.uint64))
        ka[:, l] = primes[l].ntt_fwd(np.full(n, q // 2 + 1, np.uint64))
        v = (((q >> log_b) - 1) << log_b) | ((1 << log_b) - 1)
        ct[:, 2, l] = primes[l].ntt_fwd(primes[l].import_(np.full(n, v, np.uint64)))
    key = sg.Key(ctx, log_bs, 1, kb, ka)
    d, out = sg.DeviceBuffer.from_array(ct), sg.DeviceBuffer(count * 2 * L * n * 8)
    sg.check(lib.shg_relin_apply(ctx.h, key.h, out.ptr, d.ptr, count, None))
    got = out.download((count, 2, L, n))
    for i in (0, count - 1):
        assert np.array_equal(got[i], rns.relin(ct[i], kb, ka, log_bs))
