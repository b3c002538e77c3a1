"""The work that is measured when this framework's speed is compared: what a
prime-gap search has it do, from the smallest sieve call to the gap search that
follows the sieve.

A search runs in three steps, and each has its cases here:

* the sieve (``Sieve.method2_view``, ``Sieve.method2_batch_views``,
  ``Prepared.run``): K = P#/d, a block of m, every offset up to the sieve
  length, every prime up to a limit; the file's bytes on the host, or the lists;
* reading the unknowns back (``Sieve.parse_unknowns``) for the statistics;
* the probable-prime tests (``Prepared.prp_gaps``, ``Sieve.prp_gaps`` and the
  C entry ``pgs_prp_test``), where nearly all the time of a search goes.

Sizes are those of the repository's benchmark configurations, its 64-job mix and
its tests.  Every output is whole numbers or bytes.  A file's length depends on m
by a part in a thousand: it is returned as a view of its first part and a copy of
the rest in an array of fixed size, so that every seed's outputs have one shape.
"""
from __future__ import annotations

import ctypes
import math
import random
import sys
from pathlib import Path

import numpy as np

_PKG = Path(__file__).resolve().parents[1] / "prime-gap_gb300"
if str(_PKG) not in sys.path:
    sys.path.insert(0, str(_PKG))

import pgsieve  # noqa: E402
import workloads  # noqa: E402

PLAIN, RLE, BITS = 0, 1, 2
TABLE_LIMIT = 4_000_000_000  # the mix's largest prime limit
HEAVIEST = 5e12  # operations of the heaviest drawn gap search or list of tests


def listed() -> list[dict]:
    return [
        # the smallest call: one short block of m, as the reference's own tests sieve it
        _sieve("sieve_tiny", 907, 2190, 200, 11000, 100_000_000),
        # the smallest benchmark configuration: a block that takes half a millisecond
        _sieve("sieve_small", 503, 210, 10_000, 5000, 100_000_000),
        # the benchmark's default: a block of a record search, text to the host
        _sieve("sieve_large", 1511, 2190, 100_000, 20_000, 2_000_000_000),
        # the widest configuration: primes past 2^32
        _sieve("sieve_wide", 3001, 2190, 100_000, 40_000, 10_000_000_000),
        # a bitcompressed file of a job of the mix's kind, of no round size
        _sieve("sieve_bits", 2003, 30030, 43_211, 16_500, 700_000_000, BITS),
        # an odd d (both parities of m are valid), run-length encoded
        _sieve("sieve_rle_odd", 1009, 1, 7_321, 9500, 300_000_000, RLE),
        # many uneven jobs in one call over the resident prime table
        {"name": "batch_16", "kind": "batch", "jobs": 16, "mix": 4},
        # the sieve kept on the device and its unknowns taken as lists (statistics without text)
        dict(_sieve("lists_large", 1511, 2190, 60_000, 20_000, 1_000_000_000), kind="lists"),
        # a bitcompressed file read back into lists
        dict(_sieve("parse_bits", 1511, 2190, 30_011, 20_000, 500_000_000, BITS), kind="parse"),
        # the gap search over a small block, both sides of every m
        _gaps("gaps_small", 503, 210, 4000, 5000, 100_000_000, 0),
        # the gap search of a record search's block, next side skipped where the previous gap is short
        _gaps("gaps_large", 1511, 2190, 16_001, 20_000, 2_000_000_000, 1),
        # a list of numbers of 2003#'s size to be tested, from the host
        {"name": "prp_list", "kind": "prp", "p": 2003, "d": 210, "count": 9001},
    ]


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["sieve", "sieve", "sieve", "batch", "lists", "parse", "gaps", "gaps", "gaps", "prp", "prp"])
    if kind == "batch":
        return {"kind": "batch", "jobs": round(_log_uniform(rng, 2, 16)), "mix": rng.randrange(10**6)}
    if kind == "prp":
        p = rng.choice([p for p in workloads.MIXED_P if p < 3001])
        c = {"kind": "prp", "p": p, "d": rng.choice(workloads.MIXED_D), "count": 0}
        top = min(20_000.0, HEAVIEST / _test_ops(_number_bits(c)))
        c["count"] = round(_log_uniform(rng, 600, top))
        return c
    p = rng.choice(workloads.MIXED_P)
    if kind == "gaps":  # m*K up to 4092 bits
        p = rng.choice([p for p in workloads.MIXED_P if p < 3001])
    d = rng.choice(workloads.MIXED_D)
    lo, hi = max(5000, 6 * p), min(40_000, 22 * p)
    sl = rng.randrange((lo + 499) // 500, hi // 500 + 1) * 500
    minc = round(_log_uniform(rng, 100, 100_000))
    limit = round(_log_uniform(rng, 1e7, 1e10 if kind == "sieve" else 4e9) / 1e6) * 1_000_000
    if kind == "gaps":
        c = _gaps(None, p, d, minc, sl, limit, rng.randrange(2))
        most = HEAVIEST / (work(dict(c, minc=100_000))["flops"] / 100_000)
        c["minc"] = round(_log_uniform(rng, 60, max(61.0, min(100_000.0, most))))
        return c
    c = _sieve(None, p, d, minc, sl, limit, rng.choice([PLAIN, PLAIN, RLE, BITS]))
    c["kind"] = kind
    return c


def prepare(case: dict, seed: int):
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "batch":
        _context().reserve_table(TABLE_LIMIT)
        jobs = workloads.mixed_jobs(case["jobs"], case["mix"])  # another seed moves m: the same work
        nominal = _nominal(case, jobs)
        for j in jobs:
            j.mstart = _mstart(rng, j.d)
        return _State(kind, jobs=jobs, cuts=nominal)
    if kind == "prp":
        return _State(kind, **_numbers(case, rng))
    job = pgsieve.JobSpec(case["p"], case["d"], _mstart(rng, case["d"]), case["minc"], case["sieve_length"],
                          case["max_prime"], case.get("compression", PLAIN))
    if kind == "sieve":
        return _State(kind, job=job, cuts=_nominal(case, [job]))
    if kind == "lists":
        return _State(kind, prep=_context().prepare(job), cuts=_nominal(case, [job]))
    if kind == "parse":
        return _State(kind, job=job, text=_context().method2(job), cuts=_nominal(case, [job]))
    if kind == "gaps":
        prep = _context().prepare(job)
        prep.run(False)
        return _State(kind, prep=prep, skip=bool(case["one_side_skip"]))
    raise ValueError(kind)


def run(state):
    return getattr(state, "run_" + state.kind)()


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "batch":
        each = [_sieve_work(j.p, j.d, j.minc, j.sieve_length, j.max_prime, PLAIN)
                for j in workloads.mixed_jobs(case["jobs"], case["mix"])]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if kind == "prp":
        bits = _number_bits(case)
        return {"bytes": case["count"] * (bits / 8 + 1), "flops": case["count"] * _test_ops(bits)}
    args = (case["p"], case["d"], case["minc"], case["sieve_length"], case["max_prime"])
    rows, unknowns = _rows(case["d"], case["minc"]), _unknowns(*args)
    if kind == "sieve":
        return _sieve_work(*args, case.get("compression", PLAIN))
    if kind == "lists":
        return {"bytes": 4 * unknowns + 24 * rows, "flops": _sieve_work(*args, PLAIN)["flops"]}
    if kind == "parse":
        return {"bytes": 4 * unknowns + 24 * rows + _text_bytes(*args, case["compression"]), "flops": 2 * unknowns}
    # gaps: tests until a probable prime on each side, nearest first
    bits = _number_bits(case)
    tests = 2 * rows * 0.6931 * bits / (1.781 * math.log(case["max_prime"]))
    if case["one_side_skip"]:
        tests *= 0.6
    return {"bytes": tests * 4 + 20 * rows, "flops": tests * _test_ops(bits)}


# ---- what the cases are made of -------------------------------------------


def _sieve(name, p, d, minc, sl, max_prime, compression=PLAIN) -> dict:
    c = {"kind": "sieve", "p": p, "d": d, "minc": minc, "sieve_length": sl, "max_prime": max_prime,
         "compression": compression}
    return dict(c, name=name) if name else c


def _gaps(name, p, d, minc, sl, max_prime, skip) -> dict:
    c = {"kind": "gaps", "p": p, "d": d, "minc": minc, "sieve_length": sl, "max_prime": max_prime,
         "one_side_skip": skip}
    return dict(c, name=name) if name else c


def _log_uniform(rng, lo, hi) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


_sieve_context = None


def _context() -> "pgsieve.Sieve":
    """The one library context that a program keeps."""
    global _sieve_context
    if _sieve_context is None:
        _sieve_context = pgsieve.Sieve(0)
    return _sieve_context


def _mstart(rng, d) -> int:
    """A start of eight digits after which every block has as many m coprime to d."""
    return rng.randrange(2 * 10**7 // d, 9 * 10**7 // d) * d + 1


_lengths: dict[str, list[tuple[int, int]]] = {}


def _nominal(case, jobs) -> list[tuple[int, int]]:
    """Per job of a case, how much of its file (or list of distances) every seed
    has, and room for the rest: from one run at a fixed m."""
    key = repr(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _lengths:
        got = []
        for j in jobs:
            at = pgsieve.JobSpec(j.p, j.d, 5 * 10**7 // j.d * j.d + 1, j.minc, j.sieve_length, j.max_prime, j.compression)
            stats: dict = {}
            with _context().method2_view(at, stats) as v:
                n = len(v) if case["kind"] in ("sieve", "batch") else stats["unknowns"]
            slack = int(0.002 * n + 6 * n / max(1, stats["rows"]) + 20 * math.sqrt(n)) + 64
            got.append((max(0, n - slack), 2 * slack))
        _lengths[key] = got
    return _lengths[key]


def _in_two(a, cut) -> list:
    head, room = cut
    if not head <= len(a) <= head + room:
        raise ValueError(f"an output of {len(a)} where {head} to {head + room} were expected")
    rest = np.zeros(room, dtype=a.dtype)
    rest[:len(a) - head] = a[head:]
    return [a[:head], rest, len(a)]


def _whole(lists: dict, cut) -> dict:
    """Lists as signed whole numbers, the distances in two parts."""
    out = {k: v.view(f"i{v.dtype.itemsize}") for k, v in lists.items()}
    out["dist"] = _in_two(out["dist"], cut)
    return out


class _State:
    """What a program holds before the call, and the views of its last call's
    results (given back when it calls again)."""

    def __init__(self, kind, **held):
        self.kind, self.views = kind, []
        self.__dict__.update(held)

    def _release(self):
        for v in self.views:
            v.close()
        self.views = []

    def __del__(self):
        self._release()
        if getattr(self, "prep", None) is not None:
            self.prep.close()

    def run_sieve(self):
        self._release()
        self.views = [_context().method2_view(self.job)]
        return _in_two(np.frombuffer(self.views[0].view, dtype=np.uint8), self.cuts[0])

    def run_batch(self):
        self._release()
        self.views = _context().method2_batch_views(self.jobs)
        return [_in_two(np.frombuffer(v.view, dtype=np.uint8), c) for v, c in zip(self.views, self.cuts)]

    def run_lists(self):
        self.prep.run(False)
        return _whole(self.prep.unknowns(), self.cuts[0])

    def run_parse(self):
        return _whole(_context().parse_unknowns(self.job, self.text), self.cuts[0])

    def run_gaps(self):
        gaps, _ = self.prep.prp_gaps(min_merit=18.0, one_side_skip=self.skip)
        return np.array(gaps, dtype=np.int64)

    def run_prp(self):
        s = _context()
        out = np.empty(len(self.limbs), dtype=np.uint8)
        rc = s.lib.pgs_prp_test(s.h, self.limbs.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)), self.limbs.shape[1],
                                len(self.limbs), 1, out.ctypes.data_as(ctypes.POINTER(ctypes.c_uint8)))
        if rc != pgsieve.PGS_OK:
            raise pgsieve.PgsError(rc, "pgs_prp_test")
        return out


def _primes(n: int) -> list[int]:
    flags = bytearray([1]) * (n + 1)
    flags[:2] = b"\0\0"
    for q in range(2, math.isqrt(n) + 1):
        if flags[q]:
            flags[q * q::q] = bytes(len(range(q * q, n + 1, q)))
    return [q for q in range(n + 1) if flags[q]]


def _numbers(case: dict, rng) -> dict:
    """Numbers m*K +- X without a factor up to P, as a sieve leaves them."""
    p, d = case["p"], case["d"]
    k = math.prod(_primes(p)) // d
    of_d = [q for q in _primes(100) if d % q == 0]
    words = (_number_bits(case) + 8 + 31) // 32
    nums = []
    while len(nums) < case["count"]:
        m, x = rng.randrange(10**6, 10**8), rng.randrange(1, 10 * p)
        if math.gcd(m, d) > 1 or math.gcd(k % x, x) > 1:
            continue
        n = m * k + (x if rng.random() < 0.5 else -x)
        if all(n % q for q in of_d):
            nums.append(n.to_bytes(4 * words, "little"))
    return {"limbs": np.frombuffer(b"".join(nums), dtype="<u4").reshape(case["count"], words).copy()}


def _number_bits(case: dict) -> int:
    """Bits of m*K, K = P#/d, m near 5e7."""
    return int(sum(math.log2(q) for q in _primes(case["p"])) - math.log2(case["d"]) + 25.6)


def _test_ops(bits: int) -> float:
    """Multiply-adds (two operations each) of 32-bit words in one base-2 test:
    per exponent bit a square (half the cross products) and its reduction."""
    n = bits / 32
    return bits * 2 * (0.5 * n * (n + 1) + n * n)


def _rows(d: int, minc: int) -> float:
    for q in (2, 3, 5, 7, 11, 13, 73):
        if d % q == 0:
            minc *= 1 - 1 / q
    return minc


def _unknowns(p, d, minc, sl, max_prime) -> float:
    return _rows(d, minc) * 2 * sl * 0.5615 / math.log(max_prime)


def _text_bytes(p, d, minc, sl, max_prime, compression) -> float:
    if compression == BITS:  # a bit for each offset coprime to K, 7 to a byte
        rest = math.prod(q / (q - 1) for q in (2, 3, 5, 7, 11, 13, 73) if d % q == 0)
        return _rows(d, minc) * (2 * sl * 0.5615 / math.log(p) * rest / 7 + 20)
    per = 2 if compression == RLE else 2 + math.log10(sl)
    return _unknowns(p, d, minc, sl, max_prime) * per + 20 * _rows(d, minc)


def _sieve_work(p, d, minc, sl, max_prime, compression) -> dict:
    """Bytes: the file.  Operations: for each prime K mod p (a multiply-add and
    its reduction per 32-bit word of K) and its first hit (a continued fraction
    of 0.843 ln(p/SL) levels, eight operations each), and six for each hit of a
    prime in an offset that no small prime takes."""
    limit = float(max_prime)
    primes = limit / (math.log(limit) - 1)
    words = 1.4427 * 0.97 * p / 32
    halves = 4 if d % 2 == 0 else 2
    hits = _rows(d, minc) * 2 * sl / halves * (math.log(math.log(limit)) - math.log(math.log(p)))
    levels = 0.843 * max(0.0, math.log(min(limit / sl, minc))) + 1
    return {"bytes": _text_bytes(p, d, minc, sl, max_prime, compression),
            "flops": primes * (6 * words + 8 * levels) + 6 * hits}
