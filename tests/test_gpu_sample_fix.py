"""The side-by-side sampler's redo of ciphertexts with rejected words, above the 4096
uniform words up to which the sequential kernel runs, and the two sizes at that
line.  Primes just far enough below a power of two that about half of the
ciphertexts have rejections (0.4 to 0.9 expected in each)."""
import pytest

import test_gpu_sample as base

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,qs,count", [
    (13, [base._prime_near(30, 1 << 14, 0)], 80), (13, [base._prime_near(32, 1 << 14, 0)], 80),
    (12, [base._prime_near(30, 1 << 13, s) for s in (0, 1, 2)], 80),
    (12, [base._prime_near(31, 1 << 13, s) for s in (0, 1)], 80),
    (12, [base._prime_near(31, 1 << 13, 0)], 80),
    (11, [base._prime_near(28, 1 << 12, s) for s in (0, 1)], 80)])
def test_sampler_rejections_match_oracle(sg, oracle, log_n, qs, count):
    base.test_sampler_matches_oracle(sg, oracle, log_n, qs, 8, count)
