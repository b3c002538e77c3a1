"""first_entry of a prime modulus (the host build of the device header), the form
without the tie test, against a walk of the residues and against the general
form with the same early stop."""
from __future__ import annotations

import ctypes
import random

import pytest

import pgo
from test_arith_host import ah  # noqa: F401 (the host library as a fixture)

u64 = ctypes.c_uint64


def _call(fn, *args):
    out = (u64 * 6)()
    fn(*[u64(a) for a in args], out)
    return list(out)


@pytest.mark.parametrize("lo", [50, 1000, 60_000, 1_000_003])
def test_prime_entry_walk(ah, lo):  # noqa: F811
    rng = random.Random(lo)
    for p in pgo.primes(lo, lo + 400)[1:]:
        for _ in range(20):
            w = rng.randrange(2, max(3, p // 2))
            if p <= 2 * w:
                continue
            a, y0 = rng.randrange(1, p), rng.randrange(p)
            t, y = 0, y0
            while y >= w:
                t, y = t + 1, (y + a) % p
            got = _call(ah.ah_first_entry_prime, p, a, w, y0, 2**63)
            assert got[:2] == [t, y], (p, a, w, y0)


@pytest.mark.parametrize("bits", [20, 27, 31, 32, 33, 40, 45])
def test_prime_entry_equals_general_form(ah, bits):  # noqa: F811
    rng = random.Random(bits)
    primes = pgo.primes(2**bits - 3000, 2**bits - 1)
    for _ in range(4000):
        p = rng.choice(primes)
        w = rng.choice([2, 3, rng.randrange(2, 2**10), rng.randrange(2, min(p // 2, 2**17))])
        a = rng.choice([1, 2, w, p - 1, p // 2, rng.randrange(1, p), rng.randrange(1, p)])
        y0 = rng.choice([0, w - 1, w, p - 1, rng.randrange(p)])
        t_lim = rng.choice([2**63, 1, 5000, 50_000, rng.randrange(1, p)])
        full = _call(ah.ah_first_entry, p, a, w, y0)
        got = _call(ah.ah_first_entry_prime, p, a, w, y0, t_lim)
        if full[0] < t_lim:
            assert got == full, (p, a, w, y0, t_lim)
        else:
            assert got[0] >= t_lim, (p, a, w, y0, t_lim)


@pytest.mark.parametrize("bits,mi_hi", [(10, 1), (16, 700), (24, 5000), (31, 30_000), (45, 2**31 - 1)])
def test_whole_walk(ah, bits, mi_hi):  # noqa: F811
    """Every hit of a direct walk, by circle steps within the bound's count."""
    u32 = ctypes.c_uint32
    ah.ah_whole_walk_agrees.argtypes = [u32] * 9 + [ctypes.POINTER(u32), ctypes.c_size_t]
    rng = random.Random(bits)
    primes = pgo.primes(2**bits - 900, 2**bits - 1)
    cap = 1 << 20
    buf = (u32 * cap)()
    walked = 0
    for _ in range(300):
        p = rng.choice(primes)
        w = rng.choice([2, 3, max(2, p >> 14), rng.randrange(2, min((p - 1) // 2, 2**17))])
        hi = min(mi_hi, 100_000 * (p // w))
        t, y, kp, up, kn, dn = _call(ah.ah_first_entry_prime, p, rng.randrange(1, p), w, rng.randrange(p), hi)
        if t >= hi or y >= w:
            continue
        kp, kn = min(kp, hi), min(kn, hi)
        assert ah.ah_whole_walk_agrees(t, y, kp, up, kn, dn, w, hi, 2**32 - 1, buf, cap) == 1, (p, w, t, y)
        walked += 1
    assert walked > 20


@pytest.mark.parametrize("bits", [33, 34, 36, 40, 44])
def test_prime_entry_least_gap(ah, bits):  # noqa: F811
    """64-bit moduli whose descent ends in tiny gaps (step costs past 2^32) and
    windows at the line where the circle goes to 32 bits, w = floor(p / 2^32) + 1."""
    rng = random.Random(1000 + bits)
    primes = pgo.primes(2**bits - 2000, 2**bits - 1)
    for _ in range(1500):
        p = rng.choice(primes)
        least = (p >> 32) + 1
        w = max(2, rng.choice([least - 1, least, least + 1, 2 * least, 2**14]))
        k = rng.randrange(1, min(p, 2**rng.randrange(20, bits)))
        # k steps come to a small residue: gaps of a few units at the end
        a = rng.choice([pow(k, -1, p), p - pow(k, -1, p), rng.randrange(1, p)])
        y0 = rng.randrange(p)
        t_lim = rng.choice([2**31 - 1, 2**32 - 1, 100_000, 2**33])
        full = _call(ah.ah_first_entry, p, a, w, y0)
        got = _call(ah.ah_first_entry_prime, p, a, w, y0, t_lim)
        if full[0] < t_lim:
            assert got == full, (p, a, w, y0, t_lim)
        else:
            assert got[0] >= t_lim, (p, a, w, y0, t_lim)
