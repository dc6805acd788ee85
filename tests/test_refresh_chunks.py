"""How a value refresh splits a matrix's slots into chunks (host only): the
chunks cover every slot once, in order, whatever the slot count (up to
2^32 - 1), and each holds its slices' entries."""
import ctypes as C

import numpy as np
import pytest


class Chunk(C.Structure):
    _fields_ = [("first", C.c_uint), ("slots", C.c_uint), ("entry", C.c_int),
                ("entries", C.c_int)]


def chunks(ispm, begin, lo, hi):
    L = ispm.lib_handle()
    L.ispm_refresh_chunks.argtypes = [C.c_int] + [C.c_void_p] * 4 + [C.c_int]
    begin, lo, hi = (np.ascontiguousarray(v, t) for v, t in
                     ((begin, np.uint32), (lo, np.int32), (hi, np.int32)))
    args = (len(lo), begin.ctypes.data, lo.ctypes.data, hi.ctypes.data)
    n = L.ispm_refresh_chunks(*args, None, 0)
    out = (Chunk * max(n, 1))()
    assert L.ispm_refresh_chunks(*args, out, n) == n
    return [(c.first, c.slots, c.entry, c.entries) for c in out[:n]]


def check(ch, begin, lo, hi):
    at = 0
    for first, slots, entry, entries in ch:
        assert first == at and 0 < slots <= 8192
        at += slots
        # the slices whose slots it holds
        a = np.searchsorted(begin, first, side="right") - 1
        b = np.searchsorted(begin, first + slots, side="left")
        real = [s for s in range(a, b) if lo[s] <= hi[s]]
        if real:
            assert entry <= min(lo[s] for s in real)
            assert entry + entries > max(hi[s] for s in real)
        assert entry >= 0 and entries <= 8192
    assert at == begin[-1]


@pytest.mark.parametrize("slots,count", [(1 << 20, 2300), (1 << 10, 700), (3, 50)])
def test_chunks_cover_every_slot(ispm, slots, count):
    begin = np.arange(count + 1, dtype=np.int64) * slots  # 2.4e9 slots in the first case
    width = min(slots, 900)
    lo = np.arange(count) * width
    hi = lo + width - 1
    lo[5::11], hi[5::11] = 0, -1  # padding alone
    check(chunks(ispm, begin, lo, hi), begin, lo, hi)


def test_long_slices_and_no_slices(ispm):
    begin = np.array([0, 10, 30, 60])
    assert chunks(ispm, begin, [0, 5, 20], [4, 5 + 8192, 30]) == []  # gathered
    assert len(chunks(ispm, begin, [0, 5, 20], [4, 5 + 8191, 30])) >= 1
    assert chunks(ispm, np.array([0]), [], []) == []
    # a taller slice among many short runs: gathered; most of them tall: chunks
    begin = np.arange(101) * 6000
    for every, form in ((10, False), (1, True)):
        width = np.where(np.arange(100) % every == 0, 6000, 2000)
        hi = np.cumsum(width)
        ch = chunks(ispm, begin, hi - width, hi - 1)
        assert bool(ch) == form
        if ch:
            check(ch, begin, hi - width, hi - 1)
