"""Fused sweeps of planes so small that every block row is a segment of its
own: each seam between two of them is finished, in the tolerances of the forms
(+-1 LSB at 8 bits)."""
import numpy as np
import pytest

import fft3dcl_gb300 as F
import oracle
from fft3dcl_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,bw", [("tc", 32), ("tc", 16), ("fast", 32), ("fast", 8)])
@pytest.mark.parametrize("size", [(16, 9), (40, 17), (239, 33), (320, 180), (640, 360)])
def test_planes_of_one_row_segments(form, bw, size):
    w, h = size
    frames = synth.moving_rects(w, h, 6, 5, lo=16, hi=235, noise=3.0)
    params = dict(bt=3, bw=bw, bh=bw, sigma=2.5, sharpen=0.3)
    ref = oracle.run_clip(frames, 8, threads=8, **params)
    with F.Engine(w, h, 8, form=form, **params) as e:
        for i in range(6):
            e.forward_raw(i, frames[i])
        for n in range(4):  # passes in a row: the seams' counts start again
            got = e.process_raw([n, n + 1, n + 2])
            assert int(np.abs(got.astype(int) - ref[n + 1].astype(int)).max()) <= 1
