"""Kernel times without events: every form's kernels stamp the engine's clocks,
the times are positive and fit the calls' own duration, and a fused fast engine
reports no third kernel."""
import time

import numpy as np
import pytest

import fft3dcl_gb300 as F
from fft3dcl_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,params,third", [
    ("exact", dict(bt=3), True), ("exact", dict(bt=0, bw=64, bh=64), True), ("exact", dict(bt=1, bw=128, bh=64), True),
    ("exact", dict(bt=2, mode=0), True), ("fast", dict(bt=3), False), ("fast", dict(bt=3, ow=8, oh=8), True),
    ("fast", dict(bt=3, bw=64, bh=64), True), ("fast", dict(bt=1, bw=32, bh=16), True), ("tc", dict(bt=4), True),
    ("tc", dict(bt=4, bw=16, bh=16), True), ("tc", dict(bt=2, ow=8, oh=8), True)])
def test_times_of_the_last_calls(form, params, third):
    frames = synth.moving_rects(320, 192, 4, 2, lo=16, hi=235, noise=2.0)
    need = max(params["bt"], 1)
    with F.Engine(320, 192, 8, form=form, **params) as e:
        assert e.last_kernel_ms() == (-1.0, -1.0, -1.0)
        for n in range(2):
            t0 = time.perf_counter()
            for i in range(need):
                e.forward_raw(i, frames[i])
            e.process_raw(list(range(need)))
            e.synchronize()
            ms = (time.perf_counter() - t0) * 1e3
            a, b, c = e.last_kernel_ms()
            assert a > 0 and b > 0 and (c > 0 if third else c == 0)
            assert a + b + c <= ms
            e.prune(100, 100)
