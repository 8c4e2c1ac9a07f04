"""Overlap-add + packing of the separate kernels: groups of four samples
(overlaps that are multiples of four) and single samples (others), planes
whose width leaves every remainder and pitches that are not aligned, each
sample format, against the oracle bit for bit."""
import numpy as np
import pytest

import fft3dcl_gb300 as F
import oracle
from fft3dcl_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ow", [4, 6, 8, 10, 16])
@pytest.mark.parametrize("width", [61, 62, 63, 64, 129])
@pytest.mark.parametrize("bits", [8, 10, 32])
def test_overlap_add_bits(ow, width, bits):
    dtype = {8: np.uint8, 10: np.uint16, 32: np.float32}[bits]
    lo, hi, scale = (16, 235, 255.0) if bits != 10 else (64, 940, 1.0)
    frames = synth.moving_rects(width, 45, 2, 7, lo=lo, hi=hi, noise=2.0, dtype=dtype, scale=scale,
                                maxval=255.0 if bits == 8 else 1023.0)
    params = dict(bt=1, sigma=3.0, bw=32, bh=16, ow=ow, oh=min(ow, 8))
    fmt = F.VideoFormat("gray", bits, 1 if bits == 32 else 0)
    got = F.FFT3DCL([[f] for f in frames], fmt, form="exact", **params)
    ref = oracle.run_clip(frames, bits, **params)
    for g, r in zip(got, ref):
        np.testing.assert_array_equal(g[0], r)
