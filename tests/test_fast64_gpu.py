"""The fast form's 64x64 kernels against the oracle: planes with aligned and
unaligned rows, blocks inside the plane and mirrored ones, each sample format,
chroma centering, every temporal mode; the form's tolerances (+-1 LSB at 8
bits, +-4 at 10, 1e-4 for float)."""
import numpy as np
import pytest

import fft3dcl_gb300 as F
import oracle
from fft3dcl_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(40, 30), (160, 144), (201, 133)])
@pytest.mark.parametrize("bits,chroma", [(8, False), (8, True), (10, True), (32, False)])
@pytest.mark.parametrize("bt", [-1, 1, 2, 3, 4])
def test_fast_64x64_blocks(size, bits, chroma, bt):
    w, h = size
    dtype = {8: np.uint8, 10: np.uint16, 32: np.float32}[bits]
    lo, hi, scale = (16, 235, 255.0) if bits != 10 else (64, 940, 1.0)
    frames = synth.moving_rects(w, h, 4, 11, lo=lo, hi=hi, noise=2.5, dtype=dtype, scale=scale,
                                maxval=255.0 if bits == 8 else 1023.0)
    params = dict(bt=bt, bw=64, bh=64, sigma=2.5, sharpen=0.3)
    need, cur = (bt, 2 if bt == 4 else 1) if bt >= 2 else (1, 0)
    ref = oracle.run_clip(frames, bits, threads=8, chroma=chroma, **params)[cur]
    with F.Engine(w, h, bits, int(bits == 32), chroma=chroma, form="fast", **params) as e:
        assert e.info().form == F.FORMS["fast"]
        for i in range(need):
            if bits == 32:
                e.forward(i, frames[i])
            else:
                e.forward_raw(i, frames[i])
        got = e.process(list(range(need))) if bits == 32 else e.process_raw(list(range(need)))
    worst = float(np.abs(got.astype(np.float64) - ref.astype(np.float64)).max())
    assert worst <= {8: 1, 10: 4, 32: 1e-4}[bits]
