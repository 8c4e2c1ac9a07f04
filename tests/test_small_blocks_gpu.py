"""Exact form, blocks four wide or high: filter and inverse take no longer for
their bins than those of 8 x 8 blocks, give or take a tenth (4 x 8 has 3/4 of a
bin a sample, 8 x 8 has 5/8)."""
import statistics

import pytest

import fft3dcl_gb300 as F

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

W, H = 3840, 2160


def inverse_us(bw, bh):
    st = torch.cuda.Stream()
    src = torch.randint(0, 1024, (H, W), dtype=torch.int16, device="cuda")
    out = torch.empty_like(src)
    torch.cuda.synchronize()
    us = []
    with F.Engine(W, H, 10, bt=4, bw=bw, bh=bh, stream=st.cuda_stream) as e:
        for fn in range(4):
            e.forward_device(fn, src.data_ptr(), 2 * W)
        for _ in range(15):
            e.process_device([0, 1, 2, 3], out.data_ptr(), 2 * W)
            st.synchronize()
            us.append(e.last_kernel_ms()[1] * 1e3)
    return statistics.median(us)


@pytest.mark.parametrize("bw,bh", [(4, 8), (8, 4)])
def test_inverse_time_by_bins(bw, bh):
    small, square = inverse_us(bw, bh), inverse_us(8, 8)
    assert small <= 1.1 * (3 / 4) / (5 / 8) * square, f"{bw}x{bh}: {small:.1f} us, 8x8: {square:.1f}"
