"""Lists copied out of the library's block by several threads: the block is given
back after the last of them, also where the caller's wait ends early (an error in
one slice, an interrupt) or the threads take no more work."""
from __future__ import annotations

import ctypes
import gc
import threading

import numpy as np
import pytest

import pgsieve


class _Lib:
    """Stands in for the library: notes when the block is given back."""

    def __init__(self):
        self.freed = threading.Event()

    def pgs_unknowns_free(self, _):
        assert not self.freed.is_set()
        self.freed.set()


def _block(values: np.ndarray) -> pgsieve.Unknowns:
    u = pgsieve.Unknowns()
    u.rows, u.total = 1, len(values)
    one64, one32 = np.ones(1, dtype=np.uint64), np.ones(1, dtype=np.uint32)
    for name, a in (("m", one64), ("start", one64), ("n_prev", one32), ("n_next", one32), ("dist", values)):
        setattr(u, name, a.ctypes.data_as(type(getattr(u, name))))
    u.held = (one64, one32, values)
    return u


@pytest.fixture
def values():
    return np.arange(3 << 20, dtype=np.uint32)


def test_block_goes_back_once(values):
    lib = _Lib()
    out = pgsieve._unknowns_out(lib, _block(values))
    assert lib.freed.is_set() and np.array_equal(out["dist"], values)


@pytest.mark.parametrize("error", [MemoryError, KeyboardInterrupt])
def test_block_outlives_slices_under_way(values, monkeypatch, error):
    lib, go, copyto = _Lib(), threading.Event(), np.copyto
    freed_early = []

    def slow(dst, src):
        if src[0] == 0:
            raise error  # what the caller sees while the other slices are being copied
        assert go.wait(20)
        freed_early.append(lib.freed.is_set())
        copyto(dst, src)

    monkeypatch.setattr(np, "copyto", slow)
    with pytest.raises(error):
        pgsieve._unknowns_out(lib, _block(values))
    go.set()
    gc.collect()
    assert lib.freed.wait(20)  # when the last slice is done
    assert len(freed_early) == 7 and not any(freed_early)


def test_block_outlives_slices_of_threads_that_end(values, monkeypatch):
    """Threads that take some slices and then no more (the interpreter ends)."""
    from concurrent.futures import ThreadPoolExecutor

    lib, go, copyto = _Lib(), threading.Event(), np.copyto
    early, main = [], threading.get_ident()

    def slow(dst, src):
        if threading.get_ident() != main:
            assert go.wait(20)
            early.append(lib.freed.is_set())
        copyto(dst, src)

    class Ending(ThreadPoolExecutor):
        taken = 0

        def submit(self, *args, **kw):
            self.taken += 1
            if self.taken > 3:
                threading.Timer(0.2, go.set).start()
                raise RuntimeError("cannot schedule new futures after interpreter shutdown")
            return super().submit(*args, **kw)

    monkeypatch.setattr(np, "copyto", slow)
    monkeypatch.setattr(pgsieve, "_copiers", Ending(8))
    out = pgsieve._unknowns_out(lib, _block(values))
    assert np.array_equal(out["dist"], values)
    gc.collect()
    assert lib.freed.wait(20)
    assert len(early) == 3 and not any(early)
