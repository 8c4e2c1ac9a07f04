"""Batch.step with windows that can be gone through only once (an iterator): no
entry has an output, as with any argument shorter than the batch, and no window
pointer leads to memory that holds none."""
import ctypes as C
from types import SimpleNamespace

import fft3dcl_gb300 as F


def test_windows_from_an_iterator(monkeypatch):
    n, got = 3, {}

    def step(h, fns, srcs, pitches, wins, lens, dsts, dst_pitches):
        got["lens"] = list((C.c_int * n).from_address(lens if isinstance(lens, int) else C.addressof(lens)))
        got["fns"] = list((C.c_int * n).from_address(fns if isinstance(fns, int) else C.addressof(fns)))
        return F.F3D_OK

    monkeypatch.setattr(F, "lib", lambda: SimpleNamespace(f3d_batch_step=step))
    b = F.Batch.__new__(F.Batch)
    b._h, b.engines = None, [None] * n
    b.step([4, 5, 6], [64] * n, [96] * n, iter([[1, 2, 3]] * n), [128] * n, [96] * n)
    assert got == dict(lens=[0] * n, fns=[4, 5, 6])
