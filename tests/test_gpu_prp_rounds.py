"""The gap search's rounds in both forms against the oracle: lists that end within a
round, empty and one-sided ones, few and many rows, rows with m far below the
largest."""
from __future__ import annotations

import random

import numpy as np
import pytest

import prp_oracle as po

pytestmark = pytest.mark.gpu


def _lists(k: int, sl: int, ms: list[int], lengths: list[int], rng) -> dict:
    start, n_prev, n_next, dist = [], [], [], []
    for i, m in enumerate(ms):
        odd = [x for x in range(1, sl) if (m * k + x) % 2]
        sides = [sorted(rng.sample(odd, min(lengths[(i + s) % len(lengths)], len(odd)))) for s in (0, 3)]
        start.append(len(dist))
        n_prev.append(len(sides[0]))
        n_next.append(len(sides[1]))
        dist += sides[0] + sides[1]
    return {"m": np.array(ms, dtype=np.uint64), "start": np.array(start, dtype=np.uint64),
            "n_prev": np.array(n_prev, dtype=np.uint32), "n_next": np.array(n_next, dtype=np.uint32),
            "dist": np.array(dist, dtype=np.uint32)}


@pytest.mark.parametrize("skip", [False, True])
@pytest.mark.parametrize("p,d,ms,lengths", [
    (101, 30, [1_000_003 + 2 * i for i in range(9)], [0, 1, 5, 600, 31]),       # limb form, a few searches
    (101, 30, [1_000_003 + 2 * i for i in range(300)], [3, 0, 40]),             # many short lists
    (307, 210, [1_000_003, 1_000_009], [20, 700]),                              # two chunks, few candidates
    (307, 210, [1_000_003 + 2 * i for i in range(120)], [200, 0, 350, 1]),      # and a wave of them
    (241, 210, [1_000_003 + 2 * i for i in range(40)], [64, 2]),                # one chunk
    (503, 210, [1, 11, (1 << 50) + 1, (1 << 50) + 3], [30, 2]),                 # half the rows far narrower
    (503, 210, [13] + [(1 << 40) + 2 * i + 1 for i in range(300)], [12]),       # one row far narrower
    (727, 2310, [1_000_003, 1_000_007], [90, 0, 7]),
])
def test_rounds(sieve, p, d, ms, lengths, skip):
    rng = random.Random(f"{p} {len(ms)}")
    k, sl = po.primorial_k(p, d), 2000
    lists = _lists(k, sl, ms, lengths, rng)
    got, stats = sieve.prp_gaps(p, d, sl, lists, min_merit=12.0, one_side_skip=skip)
    rows = sorted({0, 1, len(ms) - 1} | set(rng.sample(range(len(ms)), min(3, len(ms)))))  # the oracle's
    few = {key: v if key == "dist" else v[rows] for key, v in lists.items()}
    assert [got[i] for i in rows] == po.gap_search(k, sl, few, min_merit=12.0, one_side_skip=skip)
    assert stats["prp_tests"] >= sum(r[2] + r[3] for r in got)
