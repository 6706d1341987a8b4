"""The side-by-side sampler against the oracle's sequential one: rings of one
block to many salts, ciphertexts with and without rejected words, primes that
reject often enough for the sequential kernel, and the widest error draws."""
import numpy as np
import pytest

from conftest import Q45, Q50, Q60

pytestmark = pytest.mark.gpu



def _prime_near(bits, two_n, skip):
    """The skip-th prime below 2^bits that is 1 mod two_n."""
    q = (1 << bits) + 1
    while True:
        q -= two_n
        if all(pow(a, q - 1, q) == 1 for a in (2, 3, 5, 7, 11, 13)):
            if skip == 0:
                return q
            skip -= 1


@pytest.mark.parametrize("log_n,qs,variance,count", [
    (6, Q45[:1], 8, 3), (7, Q50[:3], 1, 2), (10, [Q60], 256, 5), (12, Q45[:4], 33, 7),
    (14, Q45, 8, 40),
    # four in five, then half of these ciphertexts have rejected words, at positions
    # of their own
    (10, [_prime_near(24, 2048, 0)], 8, 150),
    (10, [_prime_near(28, 2048, s) for s in (0, 1, 2)], 8, 150),
    # some of these reject in the first limb and then meet, shifted across the
    # boundary, a word that only one of the two primes rejects
    (6, [_prime_near(17, 128, s) for s in (0, 1)], 8, 4000),
    # twelve rejections expected: the sequential kernel
    (11, [_prime_near(22, 4096, 0)], 3, 60)])
def test_sampler_matches_oracle(sg, oracle, log_n, qs, variance, count):
    lib, n, L = sg.lib(), 1 << log_n, len(qs)
    rns, ctx = oracle.Rns(log_n, qs), sg.Context(log_n, qs)
    seeds = np.random.RandomState(7 + log_n).randint(0, 256, (count, 32)).astype(np.uint8)
    buf = sg.DeviceBuffer(seeds.nbytes)
    sg.check(lib.shg_memcpy_h2d(buf.ptr, seeds.ctypes.data, seeds.nbytes, None))
    a, e = (sg.DeviceBuffer(count * L * n * 8) for _ in range(2))
    sg.check(lib.shg_sample_uniform_error(ctx.h, a.ptr, e.ptr, buf.ptr, L, count, variance, None))
    ga, ge = a.download((count, L, n)), e.download((count, L, n))
    for i in range(count):
        wa, we = rns.sample_uniform_error(L, variance, seeds[i].tobytes())
        assert np.array_equal(ga[i], wa), i
        assert np.array_equal(ge[i], we), i
