"""The side-by-side sampler's last resort: ciphertexts of more than 4096 uniform words
where a rejected word shifts a later one across a limb boundary and only one of the two
primes rejects that one.  The record of rejected words is then wrong, the redo by it
would be too, and the sequential kernel has to do the ciphertext.  Which ciphertexts
these are is found from the keystream on the host."""
import numpy as np
import pytest

import test_gpu_sample as base
from conftest import Q45, Q50


def _redo(raw, qs, n):
    """(uniform words as the redo by record gives them, whether it notices a mismatch);
    the first is None without rejected words."""
    total = n * len(qs)
    q = np.array(qs, np.uint64)
    mask = np.array([(1 << x.bit_length()) - 1 for x in qs], np.uint64)
    limb = np.arange(total) // n
    rejected = np.nonzero((raw[:total] & mask[limb]) >= q[limb])[0]
    if len(rejected) == 0:
        return None, False
    w = np.arange(total + len(rejected))
    o = w - np.searchsorted(rejected, w)  # each word's place, by the record
    listed = np.isin(w, rejected)
    limb = np.minimum(o, total - 1) // n
    v = raw[:len(w)] & mask[limb]
    inside = o < total
    out = np.empty(total, np.uint64)
    out[o[inside & ~listed]] = v[inside & ~listed]
    return out, bool((inside & (listed != (v >= q[limb]))).any())


CASES = [
    # a prime that rejects often first, then primes that hardly ever do
    (8, [base._prime_near(21, 512, 1)] + (Q45 + Q50)[:17], 1500),
    # the same prime last but one, and sixteen primes alike
    (8, (Q45 + Q50)[:16] + [base._prime_near(21, 512, 1), Q50[11]], 1500),
    (8, [base._prime_near(28, 512, s) for s in range(17)], 3000),
    (10, [base._prime_near(28, 2048, 11)] + Q45 + Q50[:1], 3000)]


def _ciphertexts(oracle, log_n, qs, count):
    n = 1 << log_n
    seeds = np.random.RandomState(11 + log_n).randint(0, 256, (count, 32)).astype(np.uint8)
    kinds = []
    for s in seeds:
        raw = np.frombuffer(bytes(oracle.prng_bytes(s.tobytes(), 0, 8 * (n * len(qs) + 64))),
                            np.uint64)
        kinds.append(_redo(raw, qs, n))
    return seeds, kinds


@pytest.mark.parametrize("log_n,qs,count", CASES)
def test_the_seeds_need_the_last_resort(oracle, log_n, qs, count):
    """Some ciphertexts of each set do, and for them the redo's words are wrong; for the
    others it is right."""
    seeds, kinds = _ciphertexts(oracle, log_n, qs, count)
    rns, L, n = oracle.Rns(log_n, qs), len(qs), 1 << log_n
    assert n * L > 4096 and sum(n * (1 - q / 2 ** q.bit_length()) for q in qs) < 1
    assert any(hard for _, hard in kinds)
    redone = [i for i, (out, hard) in enumerate(kinds) if out is not None and not hard]
    for i in [i for i, (_, hard) in enumerate(kinds) if hard] + redone[:20]:
        a, _ = rns.sample_uniform_error(L, 8, seeds[i].tobytes())
        assert np.array_equal(kinds[i][0], a.reshape(-1)) != kinds[i][1], i


@pytest.mark.gpu
@pytest.mark.parametrize("log_n,qs,count", CASES)
def test_last_resort_matches_oracle(sg, oracle, log_n, qs, count):
    lib, n, L, variance = sg.lib(), 1 << log_n, len(qs), 8
    rns, ctx = oracle.Rns(log_n, qs), sg.Context(log_n, qs)
    seeds, kinds = _ciphertexts(oracle, log_n, qs, count)
    buf = sg.DeviceBuffer(seeds.nbytes)
    sg.check(lib.shg_memcpy_h2d(buf.ptr, seeds.ctypes.data, seeds.nbytes, None))
    a, e = (sg.DeviceBuffer(count * L * n * 8) for _ in range(2))
    sg.check(lib.shg_sample_uniform_error(ctx.h, a.ptr, e.ptr, buf.ptr, L, count, variance, None))
    ga, ge = a.download((count, L, n)), e.download((count, L, n))
    hard = [i for i, (_, h) in enumerate(kinds) if h]
    for i in hard + list(range(0, count, 25)):
        wa, we = rns.sample_uniform_error(L, variance, seeds[i].tobytes())
        assert np.array_equal(ga[i], wa), i
        assert np.array_equal(ge[i], we), i
