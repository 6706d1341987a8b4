"""The four-step row phases and the uncorrected inverse butterflies: the bounds on
the CPU, and on the GPU the transforms at the edges of the row groups (batches of
1 to 9 polynomials of one prime, several primes) and of the prime ranges (just
below 2^45, 2^53 and 2^58), with inputs that push every level to its bound."""
import random

import numpy as np
import pytest

from conftest import P58, Q45, Q50



def _is_prime(q):
    return all(pow(a, q - 1, q) == 1 for a in (2, 3, 5, 7, 11, 13, 17, 19, 23))


def _below(bits, count=1, above=False):
    q, out = (1 << bits) + 1, []
    while len(out) < count:
        q += (1 << 16) if above else -(1 << 16)
        if _is_prime(q):
            out.append(q)
    return out


@pytest.mark.parametrize("q", [Q45[0], Q50[3], P58[0], 12289, 3, 65537] + _below(53))
def test_reduce_1024(q):
    """csrc/modarith.cuh reduce_1024: x below 2^10 q lands in [0, 2q)."""
    shift = max(q.bit_length() - 16, 0)
    mul = (1 << (32 + shift)) // q
    assert mul < 1 << 32
    rng = random.Random(q)
    for _ in range(20000):
        x = rng.choice([rng.randrange(min(q << 10, 1 << 64)), rng.randrange(1 << 10) * q,
                        rng.randrange(1, 1 << 10) * q - 1])
        if x >> 64:
            continue
        assert (x >> shift) < 1 << 32
        r = x - (((x >> shift) * mul) >> 32) * q
        assert 0 <= r < 2 * q and r % q == x % q


def test_uncorrected_inverse_bounds():
    # level V: inputs below 2^(2 + V) q, difference plus offset below 2^(3 + V) q;
    # eight levels at most, primes below 2^53; reduce_1024 takes seven levels' sums
    for q in _below(53):
        assert (q << (3 + 7)) < 1 << 64
        assert (4 * q) << 7 <= q << 10


@pytest.mark.gpu
@pytest.mark.parametrize("log_n,qs,count", [
    (12, _below(53, 2), 1), (12, Q50[:3], 5), (13, _below(53, 1), 7), (13, P58[:2], 4),
    (14, Q45[:2], 3), (14, Q50[:1], 9), (14, _below(53, 1, above=True), 8),
    (15, _below(53, 2), 2), (15, P58[:1], 4), (15, _below(53, 1), 6)])
def test_transforms_at_the_edges(sg, oracle, log_n, qs, count):
    lib, n, L = sg.lib(), 1 << log_n, len(qs)
    ctx = sg.Context(log_n, qs)
    x = oracle.uniform_limbs(60 + count, qs, n, count)
    for l, q in enumerate(qs):
        x[0, l] = q - 1                      # the largest values everywhere
        if count > 1:
            x[1, l, ::2] = 0                 # and every other one
            x[1, l, 1::2] = q - 1
    primes = [oracle.Prime(q, log_n) for q in qs]
    for call, ref in ((lib.shg_ntt_forward, "ntt_fwd"), (lib.shg_ntt_inverse, "ntt_inv")):
        d = sg.DeviceBuffer.from_array(x)
        sg.check(call(ctx.h, d.ptr, count, L, None))
        got = d.download(x.shape)
        for i in range(count):
            for l in range(L):
                assert np.array_equal(got[i, l], getattr(primes[l], ref)(x[i, l])), (ref, i, l)
