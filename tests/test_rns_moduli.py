"""The residue number system's moduli, from first principles: coprime, wide enough, and
every sum exact in single precision."""
from __future__ import annotations

import ctypes
import math
from fractions import Fraction

import pytest


@pytest.fixture(scope="module")
def lib():
    import build as pkg_build

    h = ctypes.CDLL(str(pkg_build.build_rns_host()))
    h.rh_a_count.argtypes = [ctypes.c_uint32, ctypes.c_uint32]
    return h


def _moduli(lib, n):
    a, b = (ctypes.c_uint32 * (32 * n))(), (ctypes.c_uint32 * (32 * n))()
    primes, bits = ctypes.c_uint32(), ctypes.c_double()
    k = lib.rh_moduli(n, a, b, ctypes.byref(primes), ctypes.byref(bits))
    return list(a)[:k], list(b), primes.value, bits.value


CHUNKS = range(1, 10)


@pytest.mark.parametrize("n", CHUNKS)
def test_moduli_hold_the_numbers_that_they_are_said_to(lib, n):
    assert lib.rh_chunks() == len(CHUNKS)
    a, b, b_primes, bits = _moduli(lib, n)
    real = [m for m in b if m > 1]
    assert all(m <= 4096 for m in a + b) and b[:b_primes] == real[:b_primes]
    for v in (a, real[:b_primes]):
        assert all(all(m % q for q in range(2, math.isqrt(m) + 1)) for m in v)
    assert math.prod(a) * math.prod(b) == math.lcm(*a, *b)  # pairwise coprime
    for width in range(max(97, int(bits) - 340), int(bits) + 1):
        k = lib.rh_a_count(n, width)
        c = Fraction(k, 2) + 1  # |x| <= c N
        A, B = math.prod(a[:k]), math.prod(b)
        assert 4 * c * c * 2**width <= A and 4 * c * 2**width <= B, width
        # floor(A / N) of numbers down to 24 bits narrower, in double precision: the start
        # A - q N stays below c N with room to spare
        mant, exp = 1.0, 0
        for m in a[:k]:
            mant, e = math.frexp(mant * m)
            exp += e
        off = abs(Fraction(mant) * Fraction(2) ** exp / A - 1) + Fraction(3, 2**53)
        assert off * A / 2 ** (width - 24) + 1 < c, width


@pytest.mark.parametrize("n", CHUNKS)
def test_sums_are_exact(lib, n):
    a, b, _, _ = _moduli(lib, n)
    for v in (a, b):
        worst = sum(m // 2 + 1 for m in v)  # of |xi|: balanced, one more for the quotient's rounding
        assert 32 * worst + (len(v) // 2 + 1) * 2048 < 2**24
    # the rank's column, 4096 / m in 11 bits of mantissa: a quarter would be too much
    rank = sum(Fraction(m // 2 + 1) * Fraction(1, 2**11) * Fraction(4096, m) for m in b if m > 1) / 4096
    assert rank < Fraction(1, 8)


def test_wide_moduli_are_refused(lib):
    """288 residues near 4096 would not fit: 2048 * 32 * 288 > 2^24."""
    for moduli, ok in (([4093] * 288, 0), ([4093] * 240, 1), ([1950] * 288, 1)):
        assert lib.rh_sums_exact((ctypes.c_uint32 * len(moduli))(*moduli), len(moduli)) == ok


def test_benchmark_counts_the_products_of_these_widths(lib):
    import bench

    assert list(bench.RNS_WIDTHS) == [int(_moduli(lib, n)[3]) for n in CHUNKS]
