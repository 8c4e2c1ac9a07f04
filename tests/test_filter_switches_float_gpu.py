"""Float outputs, to the last bit, of planes whose filter switches differ in one
batch (the kernels that read the switches) and of each plane alone (those built
for its switches), in both forms that have such kernels."""
import numpy as np
import pytest

import fft3dcl_gb300 as F
from fft3dcl_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SWITCHES = [dict(), dict(sharpen=0.4), dict(degrid=0.0), dict(sigma2=1.0, sigma3=3.0, sigma4=4.0, sharpen=0.2)]
W, H = 333, 95


@pytest.mark.parametrize("form,bw", [("tc", 16), ("tc", 32), ("fast", 8), ("fast", 16), ("fast", 32)])
@pytest.mark.parametrize("bt", [-1, 1, 2, 3, 4])
def test_mixed_switches_equal_each_alone(form, bw, bt):
    need = max(bt, 1)
    frames = synth.moving_rects(W, H, need, 3, lo=0.06, hi=0.92, noise=0.02, dtype=np.float32)
    src = [torch.from_numpy(f).cuda() for f in frames]
    st, win = torch.cuda.Stream(), list(range(need))
    torch.cuda.synchronize()
    engines = [F.Engine(W, H, 32, 1, form=form, bt=bt, bw=bw, bh=bw, sigma=3.0, stream=st.cuda_stream, **sw)
               for sw in SWITCHES]
    alone, out = [torch.zeros((len(engines), H, W), device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    for e, a in zip(engines, alone):
        for i, f in enumerate(src):
            e.forward_device(i, f.data_ptr(), 4 * W)
        e.process_device(win, a.data_ptr(), 4 * W)
    with F.Batch(engines, graph=False, autotune=False) as b:
        n = len(engines)
        b.step([-1] * n, [0] * n, [0] * n, [win] * n, [o.data_ptr() for o in out], [4 * W] * n)
        torch.cuda.synchronize()
    assert alone.abs().sum(dim=(1, 2)).min() > 0
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), alone.cpu().numpy().view(np.uint32))
    for e in engines:
        e.close()
