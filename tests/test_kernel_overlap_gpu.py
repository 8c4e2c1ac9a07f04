"""Kernels start before the one ahead of them on the stream has ended: outputs
queued without a wait between them, on buffers that the next output overwrites,
equal those of the same calls waited for one by one, directly and from a
captured graph in which a call also waits for another stream's copy."""
import numpy as np
import pytest

import fft3dcl_gb300 as F
from fft3dcl_gb300 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

N = 24


def outputs(form, params, size, wait, graph=False):
    w, h = size
    frames = torch.from_numpy(np.stack(synth.moving_rects(w, h, N, 3, lo=16, hi=235, noise=3.0))).cuda()
    need = max(params["bt"], 1)
    src = torch.zeros((h, w), dtype=torch.uint8, device="cuda")
    dst = torch.zeros_like(src)
    got = torch.zeros((N, h, w), dtype=torch.uint8, device="cuda")
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()

    def one(e, i):
        # One input and one output buffer: the copy in and the copy out are
        # ordered with the kernels by the stream alone.
        with torch.cuda.stream(side):
            side.wait_stream(main)
            src.copy_(frames[i])
        main.wait_stream(side)
        with torch.cuda.stream(main):
            e.forward_device(i, src.data_ptr(), w)
            if i >= need - 1:
                e.process_device(list(range(i - need + 1, i + 1)), dst.data_ptr(), w)
                got[i].copy_(dst)
            e.prune(i - need + 2, i)
        if wait:
            torch.cuda.synchronize()

    with F.Engine(w, h, 8, form=form, stream=main.cuda_stream, **params) as e:
        if graph:
            one(e, 0)  # first launches set kernel attributes: not in the capture
            one(e, 1)
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=main):
                for i in range(2, N):
                    one(e, i)
            g.replay()
        else:
            for i in range(N):
                one(e, i)
        torch.cuda.synchronize()
    return got.cpu().numpy()


@pytest.mark.parametrize("form,params", [
    ("exact", dict(bt=2)), ("exact", dict(bt=0)), ("exact", dict(bt=2, bw=64, bh=64)),
    ("exact", dict(bt=1, bw=128, bh=64)), ("fast", dict(bt=2)), ("fast", dict(bt=2, ow=8, oh=8)),
    ("fast", dict(bt=2, bw=64, bh=64)), ("fast", dict(bt=0, bw=32, bh=16)), ("tc", dict(bt=2)),
    ("tc", dict(bt=2, ow=8, oh=8)), ("tc", dict(bt=2, bw=16, bh=16))])
@pytest.mark.parametrize("size", [(96, 64), (640, 360)])
def test_queued_equals_waited(form, params, size):
    want = outputs(form, params, size, wait=True)
    assert want[max(params["bt"], 1) - 1:].any(axis=(1, 2)).all()
    np.testing.assert_array_equal(outputs(form, params, size, wait=False), want)


@pytest.mark.parametrize("form", ["exact", "fast", "tc"])
def test_captured_equals_waited(form):
    want = outputs(form, dict(bt=2), (320, 180), wait=True)
    np.testing.assert_array_equal(outputs(form, dict(bt=2), (320, 180), wait=False, graph=True), want)
