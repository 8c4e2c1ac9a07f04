"""What an engine and a batch need zeroed (the sweep's seam counters, the kernel
clocks) is zero when their create call returns, whatever the streams are doing:
created while the caller's stream records a graph, over memory that held other
values, both give the right outputs without that graph ever running; and a batch
created while the legacy stream is busy keeps the times of its first step."""
import warnings

import numpy as np
import pytest

import fft3dcl_gb300 as F
from fft3dcl_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

W, H, N = 640, 360, 5


@pytest.fixture(scope="module")
def clip():
    frames = synth.moving_rects(W, H, N, 9, lo=16, hi=235, noise=2.0)
    return frames, torch.from_numpy(np.stack(frames)).cuda()


def two_outputs(b, e, src, out):
    for i in range(4):
        e.forward_device(i, src[i].data_ptr(), W)
    b.step([-1, -1], [0, 0], [0, 0], [[0, 1, 2], [1, 2, 3]], [o.data_ptr() for o in out], [W, W])


@pytest.mark.parametrize("form", ["fast", "tc"])
def test_created_while_the_stream_is_captured(clip, form):
    frames, src = clip
    ref = F.FFT3DCL(frames, bits=8, form=form, bt=3)
    out = torch.zeros((2, H, W), dtype=torch.uint8, device="cuda")
    st = torch.cuda.Stream()
    junk = [torch.full((4 << 20,), 0x55, dtype=torch.uint8, device="cuda") for _ in range(32)]
    torch.cuda.synchronize()
    del junk
    torch.cuda.empty_cache()
    g = torch.cuda.CUDAGraph()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")  # the graph stays empty
        with torch.cuda.graph(g, stream=st, capture_error_mode="relaxed"):
            e = F.Engine(W, H, 8, form=form, bt=3, stream=st.cuda_stream)
            b = F.Batch([e, e], graph=False, autotune=False)
    with e, b:
        for _ in range(2):  # the counters are zero again after a step
            out.zero_()
            torch.cuda.synchronize()
            two_outputs(b, e, src, out)
            torch.cuda.synchronize()
            for i in range(2):
                np.testing.assert_array_equal(out[i].cpu().numpy(), ref[i + 1])


def test_times_with_a_busy_legacy_stream(clip):
    _, src = clip
    out = torch.zeros((2, H, W), dtype=torch.uint8, device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    with F.Engine(W, H, 8, form="tc", bt=3, stream=st.cuda_stream) as e:
        torch.cuda._sleep(100_000_000)  # the default stream: some 50 ms
        with F.Batch([e, e], graph=False, autotune=False) as b:
            two_outputs(b, e, src, out)
            st.synchronize()
            torch.cuda.synchronize()
            assert all(t > 0 for t in b.last_kernel_ms())
