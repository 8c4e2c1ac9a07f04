"""Kernel stamps do not hold up kernels of many short CTAs: the forward of 8 x 8
blocks at 3840x2160 (65,000 CTAs), stamped by the engine's call, takes no more
than a quarter longer than unstamped in a batch step without outputs."""
import pytest

import fft3dcl_gb300 as F

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

W, H, N = 3840, 2160, 40


def test_stamped_forward():
    st = torch.cuda.Stream()
    src = torch.randint(0, 256, (H, W), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with F.Engine(W, H, 8, form="fast", bt=1, bw=8, bh=8, stream=st.cuda_stream) as e, F.Batch([e]) as b:

        def us(forward):
            best = 1e9
            for _ in range(4):
                t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                t0.record(st)
                for fn in range(N):
                    forward(fn)
                    e.prune(fn + 1, fn + 1)
                t1.record(st)
                t1.synchronize()
                best = min(best, t0.elapsed_time(t1) / N * 1e3)
            return best

        plain = us(lambda fn: b.step([fn], [src.data_ptr()], [W], [[]], [0], [0]))
        stamped = us(lambda fn: e.forward_device(fn, src.data_ptr(), W))
    assert stamped <= 1.25 * plain, f"{stamped:.1f} us, {plain:.1f} without stamps"
