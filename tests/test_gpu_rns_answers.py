"""Probable primes through every kernel of the residue form (one tile per pair of CTAs
with one to nine chunks, groups of tiles with one to six): at edges of tiles, in both CTAs
of a pair, in every tile of a group and in the last one that is not full."""
from __future__ import annotations

import ctypes
import random

import numpy as np
import pytest

import pgsieve
import prp_oracle as po

pytestmark = pytest.mark.gpu

WAVE = 76 * 256  # single tiles on 152 SMs
# a width of each chunk count, and the tiles of a group
WIDTHS = {1: (340, 4), 2: (700, 3), 3: (1060, 2), 4: (1420, 2), 5: (1780, 2), 6: (2120, 2), 7: (2440, 1),
          8: (2722, 1), 9: (2864, 1)}


def _few(bits: int) -> tuple[list[int], list[bool]]:
    """Numbers within 22 bits of the widest, every third a strong pseudoprime
    (4^p + 1)/5, 2p - 2 bits wide."""
    rng = random.Random(bits)
    p = [q for q in range(bits // 2 - 10, bits // 2 + 2) if all(q % r for r in range(2, int(q**0.5) + 1))]
    nums = []
    for i in range(12):
        nums.append((4 ** p[i % len(p)] + 1) // 5 if i % 3 == 0 else rng.getrandbits(bits) | (1 << (bits - 1)) | 1)
    assert all(bits - 22 <= n.bit_length() <= bits + 1 for n in nums)
    want = [po.strong_prp2(n) for n in nums]
    assert any(want) and not all(want)
    return nums, want


def _check(s, few, want, place):
    words = max(n.bit_length() for n in few) // 32 + 1
    limbs = np.frombuffer(b"".join(n.to_bytes(4 * words, "little") for n in few), dtype="<u4").reshape(-1, words)
    limbs = np.ascontiguousarray(limbs[place])
    out = np.full(len(place), 7, dtype=np.uint8)
    rc = s.lib.pgs_prp_test(s.h, limbs.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)), words, len(place), 1,
                            out.ctypes.data_as(ctypes.POINTER(ctypes.c_uint8)))
    assert rc == pgsieve.PGS_OK
    assert np.array_equal(out, np.array(want, dtype=np.uint8)[place])


@pytest.mark.parametrize("chunks", WIDTHS)
def test_single_tiles(sieve, chunks):
    few, want = _few(WIDTHS[chunks][0])
    rng = random.Random(chunks)
    prime, rest = want.index(True), [i for i, w in enumerate(want) if not w]
    for count in (1, 128, 129, 256, 257, 700):
        place = np.array([rng.randrange(12) for _ in range(count)])
        place[[i for i in (0, 127, 128, 255, 256, count - 1) if i < count]] = prime
        _check(sieve, few, want, place)
        place[-1] = rest[0]
        _check(sieve, few, want, place)


@pytest.mark.parametrize("chunks", [n for n, (_, tiles) in WIDTHS.items() if tiles > 1])
def test_groups_of_tiles(sieve, chunks):
    bits, tiles = WIDTHS[chunks]
    few, want = _few(bits)
    rng = random.Random(chunks)
    for extra in (1, 1300):
        place = np.array([rng.randrange(12) for _ in range((tiles - 1) * WAVE + extra)])
        place[[0, len(place) - 1]] = want.index(True)
        _check(sieve, few, want, place)


# the last widths of one to nine chunks and the ones after them
@pytest.mark.parametrize("bits", [253, 360, 361, 735, 736, 1103, 1104, 1463, 1464, 1813, 1814, 2147, 2148, 2462, 2463,
                                  2747, 2748, 2900])
def test_edges_of_the_widths(sieve, bits):
    rng = random.Random(bits)
    few = [rng.getrandbits(b) | (1 << (b - 1)) | 1 for b in (bits, bits, bits, bits - 19, bits - 21, bits - 22)]
    few += [(1 << bits) - 1, (1 << (bits - 1)) + 1]
    p = next(q for q in range(bits // 2 + 1, 0, -1) if all(q % r for r in range(2, int(q**0.5) + 1)))
    few += [(4**p + 1) // 5] * (2 * p - 2 >= bits - 22)
    want = [po.strong_prp2(n) for n in few]
    # so many that the residue form takes them at every width
    place = np.array([rng.randrange(len(few)) for _ in range(13_000 if bits < 765 else 16)])
    place[: len(few)] = range(len(few))
    _check(sieve, few, want, place)
