"""Numbers with several factors among the residue system's own primes, the ones that
no factor rules out by itself."""
from __future__ import annotations

import math
import random

import pytest

import prp_oracle as po

pytestmark = pytest.mark.gpu

SMALL = [p for p in range(3, 4096) if all(p % q for q in range(2, int(p**0.5) + 1))]


def _order(q: int) -> int:
    o, x = 1, 2 % q
    while x != 1:
        x, o = 2 * x % q, o + 1
    return o


def _cyclotomic(n: int) -> int:
    """Phi_n(2): 2 has order n modulo each of its primes (but those of n)."""
    primes, rest, q = [], n, 2
    while rest > 1:
        if rest % q == 0:
            primes.append(q)
            while rest % q == 0:
                rest //= q
        q += 1
    num = den = 1
    for pick in range(1 << len(primes)):
        e, sign = n, 1
        for i, p in enumerate(primes):
            if pick >> i & 1:
                e, sign = e // p, -sign
        if sign > 0:
            num *= 2**e - 1
        else:
            den *= 2**e - 1
    return num // den


# q1 q2 Phi_n(2) with 2^(N-1) = 1 mod N: two primes of base A of numbers of this width;
# the strong test passes where 2's order is divisible by the same power of 2 throughout
PSEUDOPRIMES = [(337, 673, 10800), (673, 1429, 8988), (1163, 2657, 4233), (1163, 2657, 8466), (1181, 4051, 7130),
                (1657, 2593, 6200), (1801, 4051, 2615), (2143, 3061, 1649), (2143, 3061, 3783), (2143, 3061, 3298)]


@pytest.mark.parametrize("q1,q2,n", PSEUDOPRIMES)
def test_pseudoprimes_with_two_factors_of_the_base(sieve, q1, q2, n):
    x = q1 * q2 * _cyclotomic(n)
    assert pow(2, x - 1, x) == 1
    assert po.strong_prp2(x) == (n == 8466)
    nums = [x] * 8 + [x + 2, x - 2]
    assert sieve.prp_test(nums) == [po.strong_prp2(y) for y in nums]


def _multiple(rng, bits: int, f: int, orders: int) -> int | None:
    """A multiple of f with N = 1 modulo the odd part of every order; None: there is none."""
    step = orders // (orders & -orders)
    if math.gcd(f, step) > 1:
        return None
    c = rng.getrandbits(bits - f.bit_length() - 1) | 1 << (bits - f.bit_length() - 1) | 1
    c += (pow(f, -1, step) - c) % step
    return f * (c if c % 2 else c + step)


@pytest.mark.parametrize("bits", [700, 1400, 2140, 2740, 2900])
def test_multiples_of_two_primes_and_of_squares(sieve, bits):
    rng = random.Random(bits)
    low = [q for q in SMALL if 300 < q and _order(q) < 60] + [q for q in SMALL if q < 90 and bits == 2900]
    nums = []
    for _ in range(10):
        a, b, c = rng.sample(low, 3)
        oa, ob, oc = _order(a), _order(b), _order(c)
        for f, o in ((a * b, oa * ob), (a * a, oa), (a * a * b, oa * ob), (a**3, oa), (a * b * c, oa * ob * oc)):
            nums.append(_multiple(rng, bits, f, o))
    for w in (1093, 3511):  # 2^(w-1) = 1 mod w^2
        nums += [_multiple(rng, bits, w * w, _order(w)), _multiple(rng, bits, w * w * low[-1], _order(w) * _order(low[-1]))]
    nums = [n for n in nums if n]
    assert len(nums) > 20 and all(n.bit_length() > bits - 24 for n in nums)
    assert sieve.prp_test(nums) == [po.strong_prp2(n) for n in nums]


def test_unsieved_numbers_of_the_widest(sieve):
    """Base A of the widest numbers takes every prime from 17 on: of 3000 numbers one or
    two are multiples of a square or of two primes that do not rule them out."""
    rng = random.Random(17)
    few = [rng.getrandbits(2900) | 1 << 2899 | 1 for _ in range(60)]
    few += [_multiple(rng, 2900, f, o) for f, o in ((17 * 17, 8), (23 * 31, 55), (17 * 31, 40), (31**2, 5))]
    want = [po.strong_prp2(n) for n in few]
    assert sieve.prp_test([few[i % 64] for i in range(640)]) == [want[i % 64] for i in range(640)]
