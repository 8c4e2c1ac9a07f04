"""Kernel times need the engine's own kernels to have ended and nothing else:
they are there while other work is queued on the same stream, -1 while the
kernels themselves wait behind such work, and a batch's are not kept back by
work queued after its step. After a captured pass was replayed they are those of
the replay."""
import time

import numpy as np
import pytest

import fft3dcl_gb300 as F
from fft3dcl_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

W, H = 640, 360
BUSY = 1_000_000_000  # cycles: about half a second


@pytest.fixture(scope="module")
def src():
    return torch.from_numpy(np.stack(synth.moving_rects(W, H, 5, 9, lo=16, hi=235, noise=2.0))).cuda()


@pytest.mark.parametrize("form,params,third", [
    ("exact", dict(bt=3), True), ("exact", dict(bt=1, bw=128, bh=64), True), ("fast", dict(bt=3), False),
    ("fast", dict(bt=3, ow=8, oh=8), True), ("tc", dict(bt=3), True), ("tc", dict(bt=3, ow=8, oh=8), True)])
def test_engine_times_with_work_queued(src, form, params, third):
    st, dst = torch.cuda.Stream(), torch.zeros((H, W), dtype=torch.uint8, device="cuda")
    done = torch.cuda.Event()
    torch.cuda.synchronize()

    def one(e):
        for i in range(3):
            e.forward_device(i, src[i].data_ptr(), W)
        e.process_device([0, 1, 2], dst.data_ptr(), W)
        e.prune(100, 100)

    with F.Engine(W, H, 8, form=form, stream=st.cuda_stream, **params) as e, torch.cuda.stream(st):
        one(e)
        e.synchronize()
        first = e.last_kernel_ms()
        assert first[0] > 0 and first[1] > 0 and (first[2] > 0) == third
        one(e)
        done.record(st)
        torch.cuda._sleep(BUSY)
        done.synchronize()
        a, b, c = e.last_kernel_ms()
        assert not st.query()
        assert a > 0 and b > 0 and (c > 0 if third else c == 0)
        one(e)
        ms = e.last_kernel_ms()
        assert not st.query()
        assert ms == (-1.0, -1.0, -1.0)
        e.synchronize()
        assert min(e.last_kernel_ms()[:2]) > 0


@pytest.mark.parametrize("form", ["fast", "tc"])
def test_batch_times_do_not_wait_for_later_work(src, form):
    st, dst = torch.cuda.Stream(), torch.zeros((2, H, W), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with F.Engine(W, H, 8, form=form, bt=3, stream=st.cuda_stream) as e, torch.cuda.stream(st):
        for i in range(4):
            e.forward_device(i, src[i].data_ptr(), W)
        with F.Batch([e, e], graph=False, autotune=False) as b:
            for fwd in (-1, 4):  # the second step's frame enters beside the outputs
                b.step([-1, fwd], [0, src[4].data_ptr()], [0, W], [[0, 1, 2], [1, 2, 3]], [d.data_ptr() for d in dst], [W, W])
                torch.cuda._sleep(BUSY)
                t0 = time.perf_counter()
                ms = b.last_kernel_ms()
                assert time.perf_counter() - t0 < 0.2 and not st.query()
                assert ms[0] > 0 and (ms[1] > 0) == (form == "tc")
                st.synchronize()


def test_engine_times_of_a_replay(src):
    st, dst = torch.cuda.Stream(), torch.zeros((H, W), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with F.Engine(W, H, 8, form="tc", bt=3, stream=st.cuda_stream) as e:
        for i in range(3):
            e.forward_device(i, src[i].data_ptr(), W)
        e.process_device([0, 1, 2], dst.data_ptr(), W)  # sets kernel attributes outside the capture
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            e.process_device([0, 1, 2], dst.data_ptr(), W)
        for _ in range(3):
            g.replay()
        torch.cuda.synchronize()
        assert min(e.last_kernel_ms()) > 0
        e.process_device([0, 1, 2], dst.data_ptr(), W)
        e.synchronize()
        assert min(e.last_kernel_ms()) > 0
