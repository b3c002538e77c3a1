"""The prime sieve at the edges of its segments, for each of its three segment
lengths (chosen by the window's length), against the oracle's primes."""
from __future__ import annotations

import pytest

import pgo

pytestmark = pytest.mark.gpu

SHORT, MID = 2 * 2**14, 2 * 2**16  # numbers per segment
MID_FROM = 2 * 128 * 2**16         # windows longer than this take the middle length


@pytest.mark.parametrize("lo", [3, 4, 1009, 999_999_999, 2**32 - 40_000, 10**10 + 1])
@pytest.mark.parametrize("n", [1, 2, SHORT - 2, SHORT, SHORT + 2, 5 * SHORT + 7])
def test_short_segments(sieve, lo, n):
    assert sieve.primes(lo, lo + n - 1) == pgo.primes(lo, lo + n - 1)


@pytest.mark.parametrize("n", [MID_FROM - 2, MID_FROM, MID_FROM + 2, MID_FROM + MID + 3])
def test_middle_segments(sieve, n):
    lo = 7_000_001
    assert sieve.primes(lo, lo + n - 1) == pgo.primes(lo, lo + n - 1)
