"""The tensor-core probable-prime tests (residue number system) against the
oracle's strong test, at the sizes where they can go wrong: the widths where the
number of residue slots changes, counts around a tile of 128 and a pair of 256
numbers, and numbers that leave the common path."""
from __future__ import annotations

import random

import pytest

import prp_oracle as po

pytestmark = pytest.mark.gpu

SMALL = [p for p in range(3, 4096) if all(p % q for q in range(2, int(p**0.5) + 1))]


def _numbers(rng, bits, count):
    return [rng.getrandbits(bits - 1) | (1 << (bits - 1)) | 1 for _ in range(count)]


# the last widths of one to nine chunks of 32 slots and the ones after them
@pytest.mark.parametrize("bits", [252, 253, 360, 361, 735, 736, 1103, 1104, 1463, 1464, 1813, 1814, 2147, 2148,
                                  2462, 2463, 2747, 2748, 2900, 2901])
def test_rns_widths(sieve, bits):
    rng = random.Random(bits)
    nums = _numbers(rng, bits, 20) + [(1 << bits) - 1, (1 << (bits - 1)) + 1]
    nums += _numbers(rng, bits - 19, 3) + _numbers(rng, bits - 21, 3) + _numbers(rng, 100, 2)
    if bits <= 800:  # primes
        for i in range(12):
            while not po.strong_prp2(nums[i]):
                nums[i] += 2
    assert sieve.prp_test(nums) == [po.strong_prp2(n) for n in nums]


@pytest.mark.parametrize("count", [1, 31, 127, 128, 129, 255, 256, 257, 1300])
def test_rns_counts(sieve, count):
    rng = random.Random(count)
    prime = rng.getrandbits(300) | (1 << 300) | 1
    while not po.strong_prp2(prime):
        prime += 2
    nums = _numbers(rng, 301, count)
    for i in range(0, count, 7):
        nums[i] = prime
    assert sieve.prp_test(nums) == [po.strong_prp2(n) for n in nums]


@pytest.mark.parametrize("p", [137, 151, 359, 1069])
def test_rns_pseudoprimes_and_near_misses(sieve, p):
    """(4^p + 1)/5 passes the strong test (2^(2p) = -1), (4^p - 1)/3 only
    Fermat's (2^p is another root of 1); multiples of the residue system's own
    primes; long runs of zeros in N - 1."""
    strong, fermat = (4**p + 1) // 5, (4**p - 1) // 3
    bits = 2 * p - 2
    assert po.strong_prp2(strong) and not po.strong_prp2(fermat) and pow(2, fermat - 1, fermat) == 1
    rng = random.Random(p)
    nums = [strong, fermat]
    nums += [q * (rng.getrandbits(bits - 12) | 1 << (bits - 12) | 1) for q in rng.sample(SMALL[-300:], 12)]
    for t in (2, 5, 9, 10, 40, bits // 2):
        nums.append((_numbers(rng, bits - t, 1)[0] << t) + 1)
    if bits < 800:  # primes that are 1 modulo a high power of two: many square roots on the way
        for t in (3, 4, 6, 8, 11):
            k = rng.getrandbits(bits - t) | 1 << (bits - t - 1)
            while not po.strong_prp2((k << t) + 1):
                k += 1
            nums.append((k << t) + 1)
    assert sieve.prp_test(nums) == [po.strong_prp2(n) for n in nums]


@pytest.mark.parametrize("bits,count", [(301, 20480), (720, 20000), (1000, 19457), (1300, 39169), (1700, 19713),
                                        (2100, 20100), (2300, 19460), (2800, 19460)])
def test_rns_more_numbers_than_one_wave(sieve, bits, count):
    """Several tiles per pair of CTAs: the same answers as a few numbers get, at
    every place (the last group of tiles not full)."""
    rng = random.Random(bits)
    few = _numbers(rng, bits, 37)
    if bits < 400:
        while not po.strong_prp2(few[5]):
            few[5] += 2
    few += [(4**p + 1) // 5 for p in (bits // 2, bits // 2 - 1, bits // 2 + 1) if all(p % q for q in SMALL if q < p)]
    want = [po.strong_prp2(n) for n in few]
    got = sieve.prp_test([few[i % len(few)] for i in range(count)])
    assert all(got[i] == want[i % len(few)] for i in range(count))


@pytest.mark.parametrize("bits", [300, 720, 1300, 2100, 2800])
def test_rns_multiples_of_the_bases_primes(sieve, bits):
    """N = q c with q a prime of the residue system and 2^(N-1) = 1 mod q, the
    ones that q alone does not rule out; also with two such factors."""
    rng = random.Random(bits)
    nums = []
    for q in [x for x in SMALL if x > 2600]:
        order = next(o for o in range(1, q) if pow(2, o, q) == 1)
        if order > 400:
            continue
        c = rng.getrandbits(bits - 12) | 1 << (bits - 12) | 1
        while (q * c) % (2 * order) != 1:
            c += 2
        nums += [q * c, q * c + 2]
        c = rng.getrandbits(bits - 24) | 1 << (bits - 24) | 1
        while (q * q * c) % (2 * order) != 1:
            c += 2
        nums.append(q * q * c)
    assert len(nums) == 60
    assert sieve.prp_test(nums) == [po.strong_prp2(n) for n in nums]


def test_rns_strong_pseudoprimes_with_a_factor_of_the_base(sieve):
    """(4^p + 1)/5 with a prime factor 4pk + 1 below 4096: probable primes whose
    chain runs without that factor."""
    nums = []
    for p in [x for x in SMALL if 131 <= x < 1000]:
        if any(q in SMALL and pow(4, p, q) == q - 1 for q in range(4 * p + 1, 4096, 4 * p)):
            nums += [(4**p + 1) // 5, (4**p + 1) // 5 + 2, (4**p - 1) // 3]
    assert len(nums) >= 12
    for n in nums:  # one width at a time: each its own plan
        assert sieve.prp_test([n, n]) == [po.strong_prp2(n)] * 2, n
