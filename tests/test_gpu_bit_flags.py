"""The device parse of bitcompressed rows, a word of 32 live offsets at a time, at
word edges (sieve lengths side by side), for d with no, few and large odd primes,
against the oracle's restatement of parse_unknown_line; and rows whose header or
length does not match their flags."""
from __future__ import annotations

import numpy as np
import pytest

import pgo
import pgsieve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 6, 2190, 30030, 2 * 499])
@pytest.mark.parametrize("sl", [3500, 3501, 3502, 3507, 3520, 3533, 4000, 4500])
def test_lists_of_bitcompressed_rows(sieve, d, sl):
    job = (503, d, 1_000_001, 150, sl, 5_000_000)
    spec = pgsieve.JobSpec(*job, 2)
    if pgsieve.plan(spec)["rc"] != pgsieve.PGS_OK:
        pytest.skip("the reference refuses this sieve length")
    want = pgo.method2_lists(*job, threads=8)
    got = sieve.parse_unknowns(spec, sieve.method2(spec))
    for k in ("m", "n_prev", "n_next", "start", "dist"):
        assert np.array_equal(got[k], want[k]), k


def test_rows_that_do_not_match_their_header(sieve):
    spec = pgsieve.JobSpec(907, 2190, 1, 200, 11000, 100_000_000, 2)
    text = sieve.method2(spec)
    lines = text.split(b"\n")
    m, rest = lines[-2].split(b" : ", 1)
    count, tail = rest.split(b" ", 1)
    sign = b"+" if count.startswith(b"+") else b""
    for wrong in (1, int(count) - 1, int(count) + 1, 2 * int(count)):
        bad = lines[:-2] + [m + b" : " + sign + str(wrong).encode() + b" " + tail, b""]
        with pytest.raises(pgsieve.PgsError) as e:
            sieve.parse_unknowns(spec, b"\n".join(bad))
        assert e.value.code == pgsieve.PGS_EINVAL
    got = sieve.parse_unknowns(spec, text)
    assert got["m"][-1] == int(m) and got["n_prev"][-1] + got["n_next"][-1] == int(count)
