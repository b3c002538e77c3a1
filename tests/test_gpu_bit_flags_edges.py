"""Bitcompressed rows and their parse at the edges of their words: live counts of a side
around a multiple of 32 (the last word of flags), bitmaps whose last group of 32 words
has 1, 31 or all of them; and offsets too many for the masks per residue."""
from __future__ import annotations

import math

import numpy as np
import pytest

import pgo
import pgsieve

pytestmark = pytest.mark.gpu

P = 503
PRIMES = [q for q in range(2, P + 1) if all(q % r for r in range(2, math.isqrt(q) + 1))]


def _spec(d: int, sl: int) -> pgsieve.JobSpec:
    return pgsieve.JobSpec(P, d, 1_000_001, 150, sl, 5_000_000, 2)


def _edges(d: int) -> dict:
    """The first accepted sieve length for each remainder of the live offsets of a side
    and of the bitmap's words by 32."""
    of_k = math.prod(q for q in PRIMES if d % q)
    live, found = 0, {}
    for dd in range(1, 5500):
        live += dd % 2 == d % 2 and math.gcd(dd, of_k) == 1
        if dd < 6 * P:
            continue
        par = dd & 1 if d % 2 == 0 else (dd + 1) & 1
        words = (dd + (par == 0) + 31) // 32
        for key in (("live", live % 32), ("words", words % 32)):
            if key[1] in (0, 1, 31) and key not in found and pgsieve.plan(_spec(d, dd))["rc"] == pgsieve.PGS_OK:
                found[key] = dd
    return found


@pytest.mark.parametrize("d", [1, 2, 6, 2190, 30030, 2 * 499])
def test_word_edges(sieve, d):
    found = _edges(d)
    assert sorted(found) == [(k, r) for k in ("live", "words") for r in (0, 1, 31)]
    for sl in sorted(set(found.values())):
        job = (P, d, 1_000_001, 150, sl, 5_000_000)
        want = pgo.method2_lists(*job, threads=8)
        got = sieve.parse_unknowns(_spec(d, sl), sieve.method2(_spec(d, sl)))
        for k in ("m", "n_prev", "n_next", "start", "dist"):
            assert np.array_equal(got[k], want[k]), (sl, k)


def test_offsets_beyond_the_masks(sieve):
    """A prime of d times the live offsets of a side, in bits, above 64 MB: the parse
    divides offset by offset.  The same lists as from plain rows."""
    job = (20011, 30030 * 19997, 1, 60, 440_000, 3_000_000)
    spec = pgsieve.JobSpec(*job, 2)
    assert pgsieve.plan(spec)["rc"] == pgsieve.PGS_OK
    plain = pgsieve.JobSpec(*job, 0)  # (wider than the oracle takes)
    want = sieve.parse_unknowns(plain, sieve.method2(plain))
    got = sieve.parse_unknowns(spec, sieve.method2(spec))
    assert len(want["dist"]) > 10_000
    # live offsets of a side: even, no factor 17 to 20011 but 19997
    flags = np.ones(440_001, dtype=bool)
    flags[1::2] = flags[0] = False
    for q in range(17, 20012):
        if q != 19997 and all(q % r for r in range(2, math.isqrt(q) + 1)):
            flags[q::q] = False
    assert 19997 * ((int(flags.sum()) + 31) // 32) * 4 > 64 << 20
    for k in ("m", "n_prev", "n_next", "start", "dist"):
        assert np.array_equal(got[k], want[k]), k
