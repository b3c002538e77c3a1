"""Tests of lists whose numbers have many widths: bands for the residue form, the
rest and small lists for the limb form, every answer at its number's place."""
from __future__ import annotations

import random

import pytest

import prp_oracle as po

pytestmark = pytest.mark.gpu


def _some(rng, bits: int, count: int, primes: int) -> list[int]:
    nums = [rng.getrandbits(bits) | (1 << (bits - 1)) | 1 for _ in range(count)]
    for i in range(min(primes, count)):
        while not po.strong_prp2(nums[i]):
            nums[i] += 2
    return nums


# (width, how many) of each kind, every kind from a few different numbers
@pytest.mark.parametrize("kinds", [
    [(520, 9000), (1400, 1)],                       # one wide number beside a band
    [(1100, 7000), (1060, 7000)],                   # two bands
    [(800, 12000), (778, 50), (777, 50), (500, 300), (40, 300)],  # widths at a band's end, and a rest
    [(900, 20), (60, 30)],                          # the widest band alone
    [(900, 15), (925, 1)],                          # all through the limb form
    [(300, 20000), (1100, 3), (2950, 1)],           # wider than the residue form takes
    [(w, 7) for w in range(270, 800, 23)],          # no band
    [(4, 5), (8, 5), (253, 40)],
])
def test_lists_of_many_widths(sieve, kinds):
    rng = random.Random(repr(kinds))
    nums, want = [], []
    for bits, count in kinds:
        few = _some(rng, bits, min(count, 24), 6 if bits < 850 else 2 if bits < 1200 else 0)
        ok = [po.strong_prp2(n) if n > 7 else n in (2, 3, 5, 7) for n in few]
        nums += [few[i % len(few)] for i in range(count)]
        want += [ok[i % len(few)] for i in range(count)]
    at = list(range(len(nums)))
    rng.shuffle(at)
    assert any(want) and not all(want)
    assert sieve.prp_test([nums[i] for i in at]) == [want[i] for i in at]
