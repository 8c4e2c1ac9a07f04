"""The tensor-core filter built for fixed switches (degrid alone, degrid with
sharpen) and for any: a batch whose planes differ in their switches runs the
latter for all of them, each plane alone its own, and the outputs are the same
bits. Plane sizes leave the last group of blocks partly filled."""
import numpy as np
import pytest

import fft3dcl_gb300 as F
from fft3dcl_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SWITCHES = [dict(), dict(sharpen=0.4), dict(degrid=0.0), dict(sigma2=1.0, sigma3=3.0, sigma4=4.0, sharpen=0.2)]


@pytest.mark.parametrize("bw", [16, 32])
@pytest.mark.parametrize("bt", [-1, 1, 2, 3, 4])
@pytest.mark.parametrize("size", [(33, 17), (200, 136), (333, 95)])
def test_mixed_switches_equal_each_alone(bw, bt, size):
    w, h = size
    need = max(bt, 1)
    frames = synth.moving_rects(w, h, need, 3, lo=64, hi=940, noise=12.0, dtype=np.uint16, maxval=1023.0)
    src = [torch.from_numpy(f.view(np.int16)).cuda() for f in frames]
    win = list(range(need))
    alone = []
    for sw in SWITCHES:
        with F.Engine(w, h, 10, form="tc", bt=bt, bw=bw, bh=bw, sigma=3.0, **sw) as e:
            for i, f in enumerate(frames):
                e.forward_raw(i, f)
            alone.append(e.process_raw(win))
    st = torch.cuda.Stream()
    engines = [F.Engine(w, h, 10, form="tc", bt=bt, bw=bw, bh=bw, sigma=3.0, stream=st.cuda_stream, **sw)
               for sw in SWITCHES]
    out = [torch.empty((h, w), dtype=torch.int16, device="cuda") for _ in engines]
    torch.cuda.synchronize()
    for e in engines:
        for i, f in enumerate(src):
            e.forward_device(i, f.data_ptr(), 2 * w)
    with F.Batch(engines, graph=False, autotune=False) as b:
        n = len(engines)
        b.step([-1] * n, [0] * n, [0] * n, [win] * n, [o.data_ptr() for o in out], [2 * w] * n)
        torch.cuda.synchronize()
    for o, a in zip(out, alone):
        np.testing.assert_array_equal(o.cpu().numpy().view(np.uint16), a)
    for e in engines:
        e.close()
