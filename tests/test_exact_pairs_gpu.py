"""The exact form's inverse on lane groups (32x32 and 64x64 blocks) against the
oracle, bit for bit: from one row of blocks up, every temporal mode with
sharpening and degrid on and off, integer and float output."""
import numpy as np
import pytest

import fft3dcl_gb300 as F
import oracle
from fft3dcl_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(20, 17), (129, 97), (160, 144)])
@pytest.mark.parametrize("bw,opts", [(32, {}), (32, dict(sharpen=0.4, degrid=0.7)), (64, dict(sharpen=0.4)),
                                     (32, dict(ow=8, oh=8, degrid=1.0))])
@pytest.mark.parametrize("bits", [8, 32])
@pytest.mark.parametrize("bt", [-1, 0, 1, 2, 3, 4])
def test_bits_of_square_blocks(size, bw, opts, bits, bt):
    w, h = size
    frames = synth.moving_rects(w, h, 5, 19, lo=16, hi=235, noise=2.5,
                                dtype=np.uint8 if bits == 8 else np.float32, scale=255.0, maxval=255.0)
    params = dict(bt=bt, bw=bw, bh=bw, sigma=2.5, **opts)
    ref = oracle.run_clip(frames, bits, threads=8, **params)
    need, cur = (bt, 2 if bt == 4 else 1) if bt >= 2 else (1, 0)
    with F.Engine(w, h, bits, int(bits == 32), form="exact", **params) as e:
        for i in range(5):
            (e.forward if bits == 32 else e.forward_raw)(i, frames[i])
        # Kalman: in frame order, the state goes from one output to the next.
        for n in range(5 - need + 1):
            win = list(range(n, n + need))
            got = e.process(win) if bits == 32 else e.process_raw(win)
            np.testing.assert_array_equal(got, ref[n + cur])
