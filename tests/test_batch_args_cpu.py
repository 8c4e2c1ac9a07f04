"""Batch.step passes every sequence of whole numbers element by element, bytes
and bytearrays (small frame numbers) too: array.array takes those as raw memory,
which left the engine fewer entries to read than the batch has."""
import ctypes as C
from types import SimpleNamespace

import pytest

import fft3dcl_gb300 as F


def read(addr, kind, n):
    return list((kind * n).from_address(addr if isinstance(addr, int) else C.addressof(addr)))


@pytest.mark.parametrize("to", [list, tuple, bytes, bytearray, iter])
def test_whole_numbers_of_any_sequence(monkeypatch, to):
    n, got = 8, {}

    def step(h, fns, srcs, pitches, wins, lens, dsts, dst_pitches):
        got["fns"] = read(fns, C.c_int, n)
        for name, a in (("srcs", srcs), ("dsts", dsts)):
            got[name] = [v or 0 for v in read(a, C.c_void_p, n)]
        for name, a in (("pitches", pitches), ("dst_pitches", dst_pitches)):
            got[name] = read(a, C.c_size_t, n)
        at = [v or 0 for v in read(wins, C.c_void_p, n)]
        got["windows"] = [read(p, C.c_int, k) if k else [] for p, k in zip(at, read(lens, C.c_int, n))]
        return F.F3D_OK

    monkeypatch.setattr(F, "lib", lambda: SimpleNamespace(f3d_batch_step=step))
    b = F.Batch.__new__(F.Batch)
    b._h, b.engines = None, [None] * n
    fns, srcs, pitches = list(range(3, 3 + n)), list(range(64, 64 + n)), [96] * n
    dsts, dst_pitches = list(range(128, 128 + n)), [112] * n
    windows = [[i, i + 1, i + 2] if i != 5 else [] for i in range(n)]
    b.step(to(fns), to(srcs), to(pitches), [w if to is iter else to(w) for w in windows], to(dsts), to(dst_pitches))
    assert got == dict(fns=fns, srcs=srcs, pitches=pitches, dsts=dsts, dst_pitches=dst_pitches, windows=windows)
