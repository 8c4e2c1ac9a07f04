"""The work whose speed is measured, as cases of plain values.

A case is one steady-state pass of a running filter: the frame (or frames)
that enter the temporal window are transformed and one output (or one batch
step of outputs) is produced, through the calls a user's program makes:

* ``call`` "engine": one plane per call, frames resident in device memory
  (``Engine.forward_device`` / ``process_device`` / ``prune``);
* ``call`` "batch": several planes or consecutive outputs per step, the next
  step's frames forwarded in the same step (``Batch.step``);
* ``call`` "filter": whole frames from and to host memory through the clip
  driver with the plugin's semantics (``Filter.get_frame``).

``listed()`` holds the cases, ``draw()`` gives more of the same ranges,
``prepare()`` makes what a program has in hand before the pass (frames, the
engine with its window resident), ``run()`` makes the pass, ``work()`` counts
what it cannot do without, ``exact()`` evaluates it in 64 bits where the
output is floating point.
"""
import math

import numpy as np
import torch

import fft3dcl_gb300 as F

DEVICE = torch.device("cuda", 0)
PARAMS = ("sigma", "sigma2", "sigma3", "sigma4", "beta", "bt", "bw", "bh", "ow", "oh", "sharpen", "degrid", "kratio")


def listed():
    return [
        # A small grey clip one frame at a time: the latency of one output
        # (a preview, a low-resolution stream).
        dict(name="gray8_360p_bt3", call="engine", form="tc", family="gray", width=640, height=360, bits=8, outputs=1,
             sigma=2.0, bt=3, bw=32, bh=32),
        # The same clip filtered ahead, sixteen outputs per step.
        dict(name="gray8_360p_bt3_step16", call="batch", form="tc", family="gray", width=640, height=360, bits=8,
             outputs=16, sigma=2.0, bt=3, bw=32, bh=32),
        # 4K 10-bit luma with sharpening, one output per call: a frame server
        # that asks for one frame at a time.
        dict(name="luma10_2160p_bt4", call="engine", form="tc", family="gray", width=3840, height=2160, bits=10,
             outputs=1, sigma=3.0, bt=4, bw=32, bh=32, sharpen=0.4),
        # The same clip transcoded: ten consecutive outputs per step.
        dict(name="luma10_2160p_bt4_step10", call="batch", form="tc", family="gray", width=3840, height=2160, bits=10,
             outputs=10, sigma=3.0, bt=4, bw=32, bh=32, sharpen=0.4),
        # A 1080p 4:2:0 frame, its three planes in one step.
        dict(name="yuv8_1080p_bt4_planes", call="batch", form="tc", family="yuv", width=1920, height=1080, bits=8,
             outputs=1, sigma=2.5, bt=4, bw=32, bh=32, sharpen=0.4),
        # 16-bit scan with odd sides and a quarter overlap.
        dict(name="gray16_1365x767_bt2_ow8", call="engine", form="tc", family="gray", width=1365, height=767, bits=16,
             outputs=1, sigma=2.0, beta=1.2, bt=2, bw=32, bh=32, ow=8, oh=8),
        # Float samples, small blocks, odd sides.
        dict(name="grays_1919x1079_bt3_bw16", call="engine", form="tc", family="gray", width=1919, height=1079, bits=32,
             outputs=1, sigma=2.0, bt=3, bw=16, bh=16, sharpen=0.3),
        # Kalman mode with a sigma pattern and scene cuts on float samples.
        dict(name="grays_720p_kalman_bw64", call="engine", form="exact", family="gray", width=1280, height=720, bits=32,
             outputs=1, sigma=2.0, sigma2=1.5, sigma3=2.5, sigma4=3.0, kratio=2.0, bt=0, bw=64, bh=64),
        # The default form of the Python calls: the reference's own bits.
        dict(name="luma10_1080p_bt4_exact", call="engine", form="exact", family="gray", width=1920, height=1080, bits=10,
             outputs=1, sigma=3.0, bt=4, bw=32, bh=32, sharpen=0.4),
        # Large blocks, spatial and temporal, on 8-bit material.
        dict(name="gray8_1080p_bt3_bw64", call="engine", form="tc", family="gray", width=1920, height=1080, bits=8,
             outputs=1, sigma=2.0, bt=3, bw=64, bh=64),
        # The plain fp32 transforms at the largest plane size.
        dict(name="luma10_2160p_bt4_fast", call="engine", form="fast", family="gray", width=3840, height=2160, bits=10,
             outputs=1, sigma=3.0, bt=4, bw=32, bh=32, sharpen=0.4),
        # Whole 720p 4:2:0 frames from and to host memory, as a plugin host
        # or the command line runs the filter.
        dict(name="yuv8_720p_bt3_filter", call="filter", form="tc", family="yuv", width=1280, height=720, bits=8,
             outputs=1, sigma=2.0, bt=3, bw=32, bh=32),
    ]


def draw(rng):
    """One more case: sizes over 360p to 2160p on a logarithm, odd ones among
    them, every temporal mode, block size, sample format and call."""
    scale = 2.0 ** rng.uniform(0.0, math.log2(5.5))
    width, height = int(640 * scale), int(360 * scale * rng.uniform(0.75, 1.3))
    width, height = min(width, 3840), min(height, 2160)
    if rng.random() < 0.5:
        width, height = width & ~15, height & ~7
    call = rng.choice(["engine", "engine", "engine", "batch", "batch", "filter"])
    case = dict(call=call, form="tc", family="gray", width=width, height=height, outputs=1,
                bits=rng.choice([8, 8, 10, 10, 16, 32]), sigma=round(rng.uniform(1.5, 4.0), 2),
                bt=rng.choice([1, 2, 3, 3, 4, 4]), bw=rng.choice([16, 32, 32]))
    if call == "engine":
        case["form"] = rng.choice(["tc", "tc", "fast", "exact"])
        case["bw"] = rng.choice([16, 32, 32, 64])
        if rng.random() < 0.2:
            case.update(form="exact", bt=0, bits=32, bw=rng.choice([32, 64]))
        elif rng.random() < 0.25:
            case["ow"] = case["oh"] = case["bw"] // 4
    else:
        if rng.random() < 0.5:
            case["family"] = "yuv"
        if call == "batch":
            case["form"] = rng.choice(["tc", "tc", "tc", "fast"])
            if case["family"] == "gray":
                case["outputs"] = rng.choice([2, 4, 8, 10])
        else:
            case["bits"] = min(case["bits"], 16)
        if case["family"] == "yuv":
            case["width"], case["height"] = width & ~1, height & ~1
    case["bh"] = case["bw"]
    if rng.random() < 0.5:
        case["sharpen"] = round(rng.uniform(0.2, 0.7), 2)
    if rng.random() < 0.2:
        case["degrid"] = 0.0
    if rng.random() < 0.2 or case["bt"] == 0:
        case.update(sigma2=round(case["sigma"] * 0.75, 2), sigma3=round(case["sigma"] * 1.25, 2),
                    sigma4=round(case["sigma"] * 1.5, 2))
    return case


# ---- inputs -----------------------------------------------------------------

def _planes(case):
    """(width, height, chroma) of the planes filtered."""
    w, h = case["width"], case["height"]
    if case["family"] == "gray":
        return [(w, h, False)]
    return [(w, h, False), (w // 2, h // 2, True), (w // 2, h // 2, True)]


def _window(case):
    """Frames a window reads, and where its output frame stands in it."""
    bt = case["bt"]
    return (bt, 2 if bt == 4 else 1) if bt >= 2 else (1, 0)


def _frames(case):
    """Frames of the clip, which is read in a circle: every frame of one pass
    and of the window before it is another one."""
    return _window(case)[0] + 2 * case["outputs"] + 3


def _clip(case, seed, p):
    """Plane p of a seeded clip on the GPU: a ramp (luma), rectangles that
    move by two samples per frame, a scene cut half way, Gaussian noise; u8,
    u16 as int16 bits, or float32 in about [0, 1]."""
    w, h, chroma = _planes(case)[p]
    dev = DEVICE
    gen = torch.Generator(device=dev).manual_seed(seed * 4 + p)
    rng = np.random.default_rng(seed * 4 + p)
    nfr = _frames(case)
    base = torch.full((w,), 126.0, device=dev) if chroma else torch.linspace(16.0, 235.0, w, device=dev)
    out = []
    for f in range(nfr):
        if f % ((nfr + 1) // 2) == 0:
            rects = [(int(rng.integers(0, w)), int(rng.integers(0, h)), int(rng.integers(max(1, w // 16), w // 4 + 2)),
                      int(rng.integers(max(1, h // 16), h // 4 + 2)), float(rng.uniform(16, 240)),
                      int(rng.integers(-1, 2)) * 2, int(rng.integers(-1, 2)) * 2) for _ in range(12)]
        img = base.expand(h, w).clone()
        for x, y, rw, rh, level, vx, vy in rects:
            x0, y0 = (x + vx * f) % w, (y + vy * f) % h
            img[y0:y0 + rh, x0:x0 + rw] = level
        img += torch.randn((h, w), generator=gen, device=dev) * (1.5 if chroma else 2.5)
        if case["bits"] == 32:
            out.append((img / 255.0).to(torch.float32))
        elif case["bits"] == 8:
            out.append(img.round_().clamp_(0, 255).to(torch.uint8))
        else:
            peak = float((1 << case["bits"]) - 1)
            img = (img * float(1 << (case["bits"] - 8))).round_().clamp_(0, peak).to(torch.int32)
            out.append(img.to(torch.int16))  # the low 16 bits
    return torch.stack(out)


class _Frames:
    """The clip as a frame server gives it: a long sequence of frames, each a
    list of planes in host memory."""

    def __init__(self, planes):
        self.planes = planes

    def __len__(self):
        return 1 << 20

    def __getitem__(self, n):
        return [p[n % len(p)] for p in self.planes]


def _params(case):
    return {k: case[k] for k in PARAMS if k in case}


_stream = []


def _the_stream():
    """The program's CUDA stream: one filter's passes follow each other on it."""
    if not _stream:
        _stream.append(torch.cuda.Stream())
    return _stream[0]


def _engine(case, w, h, chroma):
    return F.Engine(w, h, case["bits"], 1 if case["bits"] == 32 else 0, chroma=chroma, form=case["form"],
                    stream=_the_stream().cuda_stream, **_params(case))


def prepare(case, seed):
    clips = [_clip(case, seed, p) for p in range(len(_planes(case)))]
    need, cur = _window(case)
    if case["call"] == "filter":
        dt = np.uint8 if case["bits"] == 8 else np.uint16
        host = _Frames([c.cpu().numpy().view(dt) for c in clips])
        fmt = F.VideoFormat("gray" if case["family"] == "gray" else "yuv", case["bits"], 0,
                            int(case["family"] == "yuv"), int(case["family"] == "yuv"))
        flt = F.Filter(host, fmt, form=case["form"], plane=0 if case["family"] == "gray" else 4, **_params(case))
        s = dict(case=case, filter=flt, n=cur + 1)
        flt.get_frame(cur)  # the frame before: its window is resident
        return s
    engines = [_engine(case, w, h, c) for w, h, c in _planes(case)]
    slots = [(p, r) for p in range(len(engines)) for r in range(case["outputs"])]
    s = dict(case=case, clips=clips, engines=engines, slots=slots, n=cur,
             outs=[torch.empty_like(clips[p][0]) for p, _ in slots])
    torch.cuda.synchronize()
    if case["bt"] == 0:  # the state after two frames
        for n in range(2):
            _engine_pass(s)
    elif case["call"] == "engine":
        for fn in range(need - 1):
            _forward(s, 0, fn)
    else:
        s["batch"] = F.Batch([engines[p] for p, _ in slots])
        for p in range(len(engines)):  # the windows of the first step
            for fn in range(need + case["outputs"] - 1):
                _forward(s, p, fn)
    torch.cuda.synchronize()
    return s


def _forward(s, p, fn):
    c = s["clips"][p]
    s["engines"][p].forward_device(fn, c[fn % len(c)].data_ptr(), c.stride(1) * c.element_size())


def _engine_pass(s):
    need, cur = _window(s["case"])
    e, out, n = s["engines"][0], s["outs"][0], s["n"]
    win = [n - cur + i for i in range(need)]
    for fn in win:
        if not e.has(fn):
            _forward(s, 0, fn)
    e.process_device(win, out.data_ptr(), out.stride(0) * out.element_size())
    e.prune(n - cur + 1, n - cur + need)
    s["n"] = n + 1
    return out


def run(state):
    case = state["case"]
    if case["call"] == "filter":
        state["n"] += 1
        return state["filter"].get_frame(state["n"] - 1)
    if case["call"] == "engine":
        return _engine_pass(state)
    need, cur = _window(case)
    n, k = state["n"], case["outputs"]
    src, pitch, fns, wins = [], [], [], []
    for (p, r), out in zip(state["slots"], state["outs"]):
        c = state["clips"][p]
        wins.append([n + r - cur + i for i in range(need)])
        fns.append(n + r - cur + need - 1 + k)  # a frame of the next step's windows
        src.append(c[fns[-1] % len(c)].data_ptr())
        pitch.append(out.stride(0) * out.element_size())
    outs = state["outs"]
    state["batch"].step(fns, src, pitch, wins, [o.data_ptr() for o in outs], pitch)
    for e in state["engines"]:
        e.prune(n + k - cur, n + 2 * k - cur + need - 1)
    state["n"] = n + k
    return outs


# ---- what a pass cannot do without ------------------------------------------

def _grid(case, w, h):
    """bw, bh, ow, oh and the block grid (columns, rows) of a plane."""
    bw, bh = case["bw"], case["bh"]
    ow, oh = case.get("ow", bw // 2), case.get("oh", bh // 2)
    if bw == 2 * ow and bh == 2 * oh:
        nx, ny = int((w + bw * 1.5 - 1) / bw), int((h + bh * 1.5 - 1) / bh)
    else:
        nx, ny = ((w + ow - 1) // (bw - ow) + 2) // 2, ((h + oh - 1) // (bh - oh) + 2) // 2
    return bw, bh, ow, oh, 2 * nx, 2 * ny


def work(case):
    """Per output: the entering plane and the finished one, the window's
    spectra read once each (consecutive outputs share them; an entering frame
    that the pass itself uses need not be read back) and the entering frame's
    written; Kalman: its state read and written. Operations: the real 2D FFT
    of each block and its inverse, and about 60 per bin for the filter."""
    need, _ = _window(case)
    k = case["outputs"]
    bps = {8: 1, 32: 4}.get(case["bits"], 2)
    nbytes = flops = 0.0
    for w, h, _ in _planes(case):
        bw, bh, _, _, nc, nr = _grid(case, w, h)
        bins = nc * nr * bh * (bw // 2 + 1)
        nbytes += 2 * k * w * h * bps
        if case["bt"] == 0:
            nbytes += 32 * bins
        elif case["call"] == "batch":
            nbytes += 8 * bins * (need + k - 1 + k)
        else:
            nbytes += 8 * bins * need
        flops += k * (5.0 * nc * nr * bw * bh * math.log2(bw * bh) + 60.0 * bins)
    return {"bytes": nbytes, "flops": flops}


# ---- the same in 64 bits ----------------------------------------------------

def _axis(n, o, odd=False):
    """One axis of the mode-1 window (window type 0, analysis and synthesis
    alike): cosine ramps over the overlap, flat between. odd: the synthesis
    window of odd block columns, whose falling ramp follows the rising one at
    once (the same window at half overlap)."""
    i = torch.arange(o, dtype=torch.float64, device=DEVICE)
    r = torch.cos(math.pi * (i - o + 0.5) / (2.0 * o))
    a = torch.ones(n, dtype=torch.float64, device=DEVICE)
    a[:o] = r
    if odd:
        a[o:2 * o] = r.flip(0)
    else:
        a[n - o:] = r.flip(0)
    return a


def _mirror(x, n):
    p = torch.remainder(x, 2 * n)
    return torch.where(p >= n, 2 * n - 1 - p, p)


def _shrink(z, sy, beta):
    psd = z.real ** 2 + z.imag ** 2 + 1e-37
    return z * torch.where(psd > beta * sy, 1.0 - sy / psd, torch.full_like(psd, (beta - 1.0) / beta))


def exact(case, seed):
    """The output plane of the first pass, for float samples through the
    engine: gather, FFT, filter, inverse and overlap-add in 64 bits."""
    if case["call"] != "engine" or case["bits"] != 32:
        return None
    w, h = case["width"], case["height"]
    bw, bh, ow, oh, nc, nr = _grid(case, w, h)
    fbw, bt, btn = bw // 2 + 1, case["bt"], max(case["bt"], 1)
    dev, f64 = DEVICE, torch.float64
    clip = _clip(case, seed, 0)
    win = _axis(bh, oh)[:, None] * _axis(bw, ow)[None, :]
    xs = -ow + torch.arange(nc, device=dev)[:, None] * (bw - ow) + torch.arange(bw, device=dev)[None, :]
    ys = -oh + torch.arange(nr, device=dev)[:, None] * (bh - oh) + torch.arange(bh, device=dev)[None, :]

    def spectra(fn):
        v = clip[fn % len(clip)].to(f64)
        b = v[_mirror(ys, h).reshape(-1)][:, _mirror(xs, w).reshape(-1)]
        b = b.reshape(nr, bh, nc, bw).permute(0, 2, 1, 3) * win
        return torch.fft.rfft2(b)

    sig = [case.get("sigma", 2.0)] + [case.get(k, case.get("sigma", 2.0)) for k in ("sigma2", "sigma3", "sigma4")]
    s, s2, s3, s4 = [(v / 255.0) ** 2 * btn * bw * bh for v in sig]
    sy = torch.tensor(s, dtype=f64, device=dev)
    fyi = torch.arange(bh, dtype=f64, device=dev)
    fxi = torch.arange(fbw, dtype=f64, device=dev)
    if sig[0] != sig[1] or sig[2] != sig[3] or sig[0] != sig[2]:
        f = torch.sqrt((((bh - 2.0 * (fyi - bh / 2.0).abs()) / bh)[:, None] ** 2 + (fxi / fbw)[None, :] ** 2) * 0.5)
        f2, f3 = math.sqrt(0.5) / 2.0, math.sqrt(0.5) / 4.0
        sy = torch.where(f < f3, s4 + (s3 - s4) * f / f3,
                         torch.where(f < f2, s3 + (s2 - s3) * (f - f3) / (f2 - f3), s + (s2 - s) * (1.0 - f) / (1.0 - f2)))
    beta, degrid = case.get("beta", 1.0), case.get("degrid", 1.0)
    need, cur = _window(case)
    grid = torch.fft.rfft2(win)
    grid = grid / grid[0, 0].real * degrid

    if bt == 0:
        cn = sy
        last, cov, proc = None, cn + torch.zeros((nr, nc, bh, fbw), dtype=f64, device=dev), cn
        for n in range(3):
            c = spectra(n)
            last = c if last is None else last
            d = c - last
            jump = torch.maximum(d.real ** 2, d.imag ** 2) > case.get("kratio", 2.0) ** 2 * cn
            sm = cov + proc
            gain = sm / (sm + cn)
            last = torch.where(jump, c, gain * c + (1.0 - gain) * last)
            proc, cov = torch.where(jump, cn, gain * gain * cn), torch.where(jump, cn, (1.0 - gain) * sm)
        z = last
        corr = c[..., :1, :1].real * grid
    else:
        fr = [spectra(i) for i in range(need)]
        corr = fr[cur][..., :1, :1].real * grid
        z = 0.0
        for q in range(need):  # the temporal DFT's frequencies, shrunk, summed at the output frame
            t = sum(fr[i] * complex(math.cos(2 * math.pi * q * (i - cur) / need),
                                    -math.sin(2 * math.pi * q * (i - cur) / need)) for i in range(need))
            # degrid applies to the temporal mean; with four frames to the
            # first harmonic, as the filter's source has it.
            at = 3 if bt == 4 else 0
            t = t - (need * corr if q == at else 0.0)
            z = z + _shrink(t, sy, beta)
        z = z / need + corr
    if case.get("sharpen", 0.0):
        smin, smax = [(v / 255.0) ** 2 * bw * bh * btn for v in (4.0, 20.0)]
        dj = torch.where(fyi >= bh / 2, bh - fyi, fyi)
        d2 = (dj ** 2 / (bh / 2.0) ** 2)[:, None] + (fxi ** 2 / (bw / 2.0) ** 2)[None, :]
        lut = case["sharpen"] * (1.0 - torch.exp(-d2 / (2.0 * 0.3 * 0.3)))
        z = z - corr
        psd = z.real ** 2 + z.imag ** 2 + 1e-37
        z = z * (1.0 + lut * torch.sqrt(psd * smax / ((psd + smin) * (psd + smax)))) + corr
    # The reference completes the half spectrum by symmetry and keeps the real
    # part: a complex inverse over the completed spectrum.
    full = torch.empty((nr, nc, bh, bw), dtype=torch.complex128, device=dev)
    full[..., :fbw] = z
    rows = (bh - torch.arange(bh, device=dev)) % bh
    full[..., fbw:] = z[..., rows, :][..., torch.arange(bw - fbw, 0, -1, device=dev)].conj()
    blocks = torch.fft.ifft2(full).real
    blocks[:, 0::2] *= win
    blocks[:, 1::2] *= _axis(bh, oh)[:, None] * _axis(bw, ow, odd=True)[None, :]
    out = torch.zeros((h + 2 * bh, w + 2 * bw), dtype=f64, device=dev)
    for m in range(nr):
        y0 = int(ys[m, 0]) + bh
        for par in (0, 1):  # blocks of one parity do not overlap
            y1 = min(y0 + bh, h + 2 * bh)
            sel = blocks[m, par::2]
            row = torch.zeros((bh, w + 2 * bw), dtype=f64, device=dev)
            xi = (xs[par::2] + bw).reshape(-1)
            ok = (xi >= 0) & (xi < w + 2 * bw)
            row[:, xi[ok]] = sel.permute(1, 0, 2).reshape(bh, -1)[:, ok]
            if y1 > y0:
                out[y0:y1] += row[: y1 - y0]
    return out[bh:bh + h, bw:bw + w]
