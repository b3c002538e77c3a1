"""Tests and searches where the device has no room for the residue form's
workspace: the limb form takes them, as it does numbers too wide for the other."""
from __future__ import annotations

import random

import pytest

import pgsieve
import prp_oracle as po

pytestmark = pytest.mark.gpu

# for the numbers, items, results and rows (4 MB of numbers); the workspaces below take
# 58 MB (20000 numbers in 96 slots of 15 halves) and more
ROOM = 40 << 20


def test_no_room_for_the_workspace(built):
    import torch

    rng = random.Random(3)
    nums = [rng.getrandbits(1100) | 1 << 1099 | 1 for _ in range(24)]
    for i in (0, 5, 23):
        while not po.strong_prp2(nums[i]):
            nums[i] += 2
    want = [po.strong_prp2(n) for n in nums]
    job = pgsieve.JobSpec(907, 2190, 1_000_001, 30, 11000, 20_000_000)
    with pgsieve.Sieve(0) as s, s.prepare(job) as prep:
        prep.run(False)
        free_want = prep.prp_gaps()[0]
        limbs = [nums[i % 24] for i in range(20000)]
        assert s.prp_test(limbs) == [want[i % 24] for i in range(20000)]
    with pgsieve.Sieve(0) as s, s.prepare(job) as prep:  # a context without blocks kept
        prep.run(False)
        free = torch.cuda.mem_get_info(0)[0]
        held = torch.empty(free - ROOM, dtype=torch.uint8, device="cuda:0")
        try:
            got = s.prp_test(limbs)
            gaps = prep.prp_gaps()[0]
        finally:
            del held
            torch.cuda.empty_cache()
        assert got == [want[i % 24] for i in range(20000)]
        assert gaps == free_want
        assert s.prp_test(limbs) == got  # and with room again
