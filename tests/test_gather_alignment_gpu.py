"""Device planes at any address and pitch: the forward kernels read rows in
whole loads where they are aligned and otherwise as their samples allow. The
spectra are the same bits for every placement of the same samples."""
import numpy as np
import pytest

import fft3dcl_gb300 as F
from fft3dcl_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,bw", [("exact", 32), ("fast", 8), ("fast", 16), ("fast", 32), ("fast", 64),
                                     ("tc", 16), ("tc", 32)])
@pytest.mark.parametrize("bits", [8, 10, 16, 32])
def test_spectra_do_not_depend_on_placement(form, bw, bits):
    w, h = 150, 90
    dtype = {8: np.uint8, 32: np.float32}.get(bits, np.uint16)
    lo, hi, scale, peak = {8: (16, 235, 1.0, 255.0), 10: (64, 940, 1.0, 1023.0), 16: (4096, 60000, 1.0, 65535.0),
                           32: (16, 235, 255.0, 255.0)}[bits]
    plane = synth.moving_rects(w, h, 1, 21, lo=lo, hi=hi, noise=2.0, dtype=dtype, scale=scale, maxval=peak)[0]
    raw = torch.from_numpy(np.ascontiguousarray(plane).view(np.uint8).reshape(h, -1).copy()).cuda()
    row, bps = raw.shape[1], plane.itemsize
    ref = None
    with F.Engine(w, h, bits, int(bits == 32), form=form, bt=1, bw=bw, bh=bw) as e:
        fn = 0
        for pitch in (row, row + bps, (row + 15) // 16 * 16, (row + 15) // 16 * 16 + 4 * bps, row + 7 * bps):
            for start in (0, bps, 3 * bps, 4 * bps, 16):
                buf = torch.zeros(h * pitch + 64, dtype=torch.uint8, device="cuda")
                buf[start:start + h * pitch].view(h, pitch)[:, :row] = raw
                torch.cuda.synchronize()
                e.forward_device(fn, buf.data_ptr() + start, pitch)
                got = e.spectra(fn)
                e.prune(1 << 20, 1 << 20)
                ref = got if ref is None else ref
                np.testing.assert_array_equal(got.view(np.uint32), ref.view(np.uint32), err_msg=f"{pitch} {start}")


@pytest.mark.parametrize("bits", [8, 10])
def test_graph_steps_with_other_placements(bits):
    # A batch replays its graph for planes placed alike; a frame at another
    # alignment is another graph. Outputs equal the engine's own.
    w, h, nfr = 192, 96, 9
    dtype = np.uint8 if bits == 8 else np.uint16
    peak = (1 << bits) - 1.0
    frames = synth.moving_rects(w, h, nfr, 5, lo=peak * 0.1, hi=peak * 0.9, noise=2.0, dtype=dtype, maxval=peak)
    ref = F.FFT3DCL(frames, bits=bits, form="tc", bt=3)
    bps = frames[0].itemsize
    pitch = w * bps + 16
    bufs, ptrs = [], []
    for i, f in enumerate(frames):
        start = [0, bps, 16, 3 * bps][i % 4]
        buf = torch.zeros(h * pitch + 64, dtype=torch.uint8, device="cuda")
        buf[start:start + h * pitch].view(h, pitch)[:, :w * bps] = torch.from_numpy(f.view(np.uint8).reshape(h, -1).copy()).cuda()
        bufs.append(buf)
        ptrs.append(buf.data_ptr() + start)
    st = torch.cuda.Stream()
    out = torch.empty((nfr, h, w * bps), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with F.Engine(w, h, bits, form="tc", bt=3, stream=st.cuda_stream) as e:
        e.forward_device(0, ptrs[0], pitch)
        with F.Batch([e], graph=True, autotune=False) as b:
            for n in range(nfr):
                win = [max(n - 1, 0), n, min(n + 1, nfr - 1)]
                fn = n + 1 if n + 1 < nfr else -1
                b.step([fn], [ptrs[fn] if fn >= 0 else 0], [pitch], [win], [out[n].data_ptr()], [w * bps])
                e.prune(n, n + 2)
            torch.cuda.synchronize()
    got = out.cpu().numpy()
    for n in range(nfr):
        np.testing.assert_array_equal(got[n].view(dtype), ref[n])
