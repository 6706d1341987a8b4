"""The uncorrected inverse butterflies (bf_gs_lazy in csrc/ntt.cuh) level by level in
exact integers: both four-step phases with every value at its largest, in the limits
that the sources state, for the largest prime that the host lets through and for one
that is too large."""
import os
import random
import re

import pytest

from conftest import PKG
from test_lazy_bounds import shoup_lazy4


def _source(name):
    with open(os.path.join(PKG, "csrc", name)) as f:
        return f.read()


def _one(pattern, text):
    found = re.findall(pattern, text)
    assert len(found) == 1, (pattern, found)
    return int(found[0])


# primes below 2^LIMIT take these butterflies; level V adds q << (OFFSET + V);
# rows of 2^ROW_BITS elements; reduce_1024 takes values below 2^10 q
LIMIT = _one(r"\(all\[i\] >> (\d+)\) != 0\) ctx->lazy_inv = 0", _source("capi.cu"))
OFFSET = _one(r"const uint64_t d = X - Y \+ \(q << \((\d+) \+ V\)\);", _source("ntt.cuh"))
ROW_BITS = _one(r"constexpr int kNtt4RowBits = (\d+);", _source("ntt4.cuh"))


def _prime_below(bits):
    q = (1 << bits) + 1
    while True:
        q -= 1 << 16
        if all(pow(a, q - 1, q) == 1 for a in (2, 3, 5, 7, 11, 13, 17, 19, 23)):
            return q


def _phase(q, levels, rng):
    """The largest sums of a phase whose inputs lie below 4q, or None where a difference
    goes below zero or a value leaves 64 bits.  X follows the sums of sums, the largest
    values there are; Y is the largest and the smallest that may meet it."""
    top = 4 * q - 1
    for v in range(levels):
        for x, y in ((top, 0), (0, top), (top, top), (rng.randrange(top), rng.randrange(top))):
            d = x - y + (q << (OFFSET + v))
            if d < 0 or d >> 64 or (x + y) >> 64:
                return None
            w = rng.randrange(q)
            r, _ = shoup_lazy4(d, w, (w << 64) // q, q)
            if r >= 4 * q or r % q != (x - y) * w % q:
                return None
        top = 2 * top  # products stay below 4q, no more than the sums
    return top


@pytest.mark.parametrize("log_n", [12, 13, 14, 15])
def test_largest_allowed_prime(log_n):
    rng, q = random.Random(log_n), _prime_below(LIMIT)
    rows = _phase(q, ROW_BITS, rng)
    assert rows is not None and rows < q << 10      # what reduce_1024 takes
    shift = max(q.bit_length() - 16, 0)
    mul = (1 << (32 + shift)) // q
    for x in [rows] + [rng.randrange(rows) for _ in range(1000)]:
        r = x - (((x >> shift) * mul) >> 32) * q
        assert 0 <= r < 4 * q and r % q == x % q    # the column phase's inputs
    assert _phase(q, log_n - ROW_BITS, rng) is not None


def test_a_larger_prime_does_not_fit():
    rng = random.Random(1)
    assert _phase(_prime_below(LIMIT + 3), 15 - ROW_BITS, rng) is None
