"""The residue form's device memory is a wave's, however many numbers or rows a
call has, and long lists go through it in slices."""
from __future__ import annotations

import ctypes
import random

import numpy as np
import pytest

import pgsieve
import prp_oracle as po

pytestmark = pytest.mark.gpu

# some 1 KB per number of 300 bits (32 slots of 15 halves), at most 4 tiles of 256
# numbers for each of 76 pairs of SMs: 75 MB; the rest of the calls below is their
# numbers, items, rows and results, under 200 bytes each
WAVE_BYTES = 100 << 20


def _free() -> int:
    import torch

    return torch.cuda.mem_get_info(0)[0]


def _limbs(nums: list[int], words: int) -> np.ndarray:
    return np.frombuffer(b"".join(n.to_bytes(4 * words, "little") for n in nums), dtype="<u4").reshape(-1, words)


def _prp_test(s, limbs: np.ndarray) -> np.ndarray:
    limbs = np.ascontiguousarray(limbs)
    out = np.full(len(limbs), 7, dtype=np.uint8)
    rc = s.lib.pgs_prp_test(s.h, limbs.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)), limbs.shape[1], len(limbs), 1,
                            out.ctypes.data_as(ctypes.POINTER(ctypes.c_uint8)))
    assert rc == pgsieve.PGS_OK
    return out


def _mixed(bits: int, count: int) -> list[int]:
    """Numbers of one width, some of them probable primes."""
    rng = random.Random(bits)
    nums = [rng.getrandbits(bits) | (1 << (bits - 1)) | 1 for _ in range(count)]
    for i in range(0, count, 3):
        while not po.strong_prp2(nums[i]):
            nums[i] += 2
    return nums


# slices of a group of tiles per pair, of single tiles, and a last one of a few numbers
# (a wave of 152 SMs: 19456 numbers a tile); 500 bits: waves of three tiles
@pytest.mark.parametrize("bits,count", [(300, 77824 * 2 + 19456 + 3), (300, 19456 + 1), (500, 58368 + 2 * 19456),
                                        (500, 58368 + 257), (900, 38912 + 1)])
def test_long_lists_in_slices(sieve, bits, count):
    few = _mixed(bits, 37 if bits < 900 else 12)
    want = np.array([po.strong_prp2(n) for n in few], dtype=np.uint8)
    limbs = _limbs(few, (bits + 31) // 32)
    place = np.arange(count) % len(few)
    assert np.array_equal(_prp_test(sieve, limbs[place]), want[place])


def test_slices_of_numbers_that_the_residue_form_leaves(sieve):
    """Places of numbers tested limb by limb after the last slice: 2^t k + 1 with more
    roots of 1 on the way than the residue form keeps."""
    bits, count = 300, 4 * 77824
    few = _mixed(bits, 40)
    rng = random.Random(1)
    k = rng.getrandbits(bits - 30) | 1 << (bits - 31) | 1
    while not po.strong_prp2((k << 30) + 1):
        k += 2
    few += [(k << 30) + 1, (4**149 + 1) // 5]
    want = np.array([po.strong_prp2(n) for n in few], dtype=np.uint8)
    limbs = _limbs(few, (bits + 31) // 32)
    place = np.array([random.Random(2).randrange(40) for _ in range(1000)] * (count // 1000 + 1))[:count]
    place[[0, 77823, 77824, 200_000, count - 1]] = [40, 41, 40, 40, 41]
    assert np.array_equal(_prp_test(sieve, limbs[place]), want[place])


def test_memory_of_a_long_list(built):
    with pgsieve.Sieve(0) as s:
        few = _mixed(300, 37)
        limbs = _limbs(few, 10)
        _prp_test(s, limbs)
        before = _free()
        count = 1_500_000
        place = np.arange(count) % len(few)
        want = np.array([po.strong_prp2(n) for n in few], dtype=np.uint8)
        assert np.array_equal(_prp_test(s, limbs[place]), want[place])
        assert before - _free() < WAVE_BYTES + 200 * count


def test_memory_of_a_search_of_many_rows(built):
    """Rows without unknowns: each side runs past the sieve length."""
    p, d, sl, rows = 251, 210, 1000, 200_000
    m = np.array([k for k in range(1_000_001, 1_000_001 + 5 * rows) if k % 2 and k % 3 and k % 5 and k % 7][:rows],
                 dtype=np.uint64)
    assert len(m) == rows
    zero = np.zeros(rows, dtype=np.uint32)
    lists = {"m": m, "start": np.zeros(rows, dtype=np.uint64), "n_prev": zero, "n_next": zero,
             "dist": np.zeros(0, dtype=np.uint32)}
    few = {k: v[:4] if k != "dist" else v for k, v in lists.items()}
    with pgsieve.Sieve(0) as s:
        s.prp_gaps(p, d, sl, few)
        before = _free()
        got, _ = s.prp_gaps(p, d, sl, lists)
        assert before - _free() < WAVE_BYTES + 200 * rows
    at = [0, 1, 77, rows // 2, rows - 1]
    some = {k: [int(x) for x in v[at]] if k != "dist" else v for k, v in lists.items()}
    assert [got[i] for i in at] == po.gap_search(po.primorial_k(p, d), sl, some)
