"""The argument forms Batch.step takes: lists, tuples, numpy arrays, and None
for the pointers of an entry without a frame or without an output. All give
the engine's own output; a missing output pointer is refused as before."""
import numpy as np
import pytest

import fft3dcl_gb300 as F
from fft3dcl_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

W, H = 96, 64


@pytest.mark.parametrize("kind", ["list", "tuple", "numpy", "none"])
def test_step_argument_forms(kind):
    frames = synth.moving_rects(W, H, 4, 9, lo=16, hi=235, noise=2.0)
    ref = F.FFT3DCL(frames, bits=8, form="tc", bt=3)
    src = torch.from_numpy(np.stack(frames)).cuda()
    out = torch.empty((2, H, W), dtype=torch.uint8, device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    with F.Engine(W, H, 8, form="tc", bt=3, stream=st.cuda_stream) as e:
        for i in range(3):
            e.forward_device(i, src[i].data_ptr(), W)
        with F.Batch([e, e], graph=False, autotune=False) as b:
            to = {"tuple": tuple, "numpy": np.array}.get(kind, list)
            no = None if kind == "none" else 0
            # Entry 0: output 1. Entry 1: frame 3 enters, no output.
            b.step(to([-1, 3]), to([no, src[3].data_ptr()]), to([0, W]), [to([0, 1, 2]), to([])],
                   to([out[0].data_ptr(), no]), to([W, 0]))
            b.step(to([-1, -1]), to([no, no]), to([0, 0]), [to([1, 2, 3]), to([])],
                   to([out[1].data_ptr(), no]), to([W, 0]))
            torch.cuda.synchronize()
            with pytest.raises(F.F3DError, match="bad output plane"):
                b.step([-1, -1], [0, 0], [0, 0], [[0, 1, 2], []], [no, no], [W, 0])
    np.testing.assert_array_equal(out[0].cpu().numpy(), ref[1])
    np.testing.assert_array_equal(out[1].cpu().numpy(), ref[2])
