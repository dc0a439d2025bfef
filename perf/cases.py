"""The work a user of this library has it do, as cases that can be timed and
compared: one frame, a frame of a clip with its history, a batch of frames,
frames served from host memory, the noise model of a frame; each through the
public entry points, over the sizes, debayers, output formats and stages that
are used in earnest.

A case is a dict of plain values. listed() gives the fixed ones, draw(rng)
one more of the same ranges; prepare(case, seed) makes what a program holds
before the call, run(state) makes the call; work(case) is what it cannot do
without, and exact(case, seed) its result in 64 bits, from the definitions
and without the library.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

import libcraw_gb300 as L

BLACK, WHITE = 256, 4095                 # 12-bit samples
RANGE = WHITE - BLACK
WB = (2.0, 1.0, 1.5)                     # as-shot gains of the camera
CAMERA = ((0.6850, 0.1640, 0.1015), (0.2950, 0.7700, -0.0650), (0.0100, 0.0400, 1.0390))
CHANNEL = (0, 1, 1, 2)                   # of the RGGB sites

DEBAYERS = {"bilinear": L.DEBAYER_BILINEAR, "mhc": L.DEBAYER_MHC, "rcd": L.DEBAYER_RCD}
SPACES = {"bt709": L.CS_BT709, "bt2020": L.CS_BT2020, "p3": L.CS_P3D65, "ap0": L.CS_ACES_AP0,
          "ap1": L.CS_ACES_AP1}
FORMATS = {"rgba16f": L.FORMAT_RGBA16F, "rgba32f": L.FORMAT_RGBA32F, "rgb32f": L.FORMAT_RGB32F}
PIXEL_BYTES = {"rgba16f": 8, "rgba32f": 16, "rgb32f": 12}

#: A frame's settings where a case does not say otherwise.
PLAIN = dict(path="frame", debayer="rcd", space="bt709", format="rgba32f", storage="fp32", denoise=0.0,
             temporal=0.0, chroma=0.0, exact_rounding=False, highlights=False, awb=True, clamp=False,
             stops=0.0, noise_a=4.0, noise_b=40.0)


def _case(**kw) -> dict:
    return {**PLAIN, **kw}


def listed() -> list[dict]:
    return [
        # A camera's live view with a closed white-balance loop: one small
        # frame, and its histogram read before the next is developed.
        _case(name="live_preview", path="live", width=640, height=360, debayer="bilinear",
              format="rgba16f", noise_a=2.0, noise_b=16.0),
        # HD monitoring: no denoise, full float output.
        _case(name="hd_bilinear", width=1920, height=1080, debayer="bilinear", noise_a=2.0, noise_b=16.0),
        # UHD playback: half storage and output, negatives clamped, no statistic.
        _case(name="uhd_mhc_half", width=3840, height=2160, debayer="mhc", space="p3", format="rgba16f",
              storage="fp16", awb=False, clamp=True),
        # A cinema frame of a ragged size with the library's default rounding.
        _case(name="cinema_denoise", width=4098, height=2162, space="bt2020", denoise=1.0),
        # The full chain on one 5760x3240 frame, its codes rounded as 64 bits round them.
        _case(name="frame_exact_ap1", width=5760, height=3240, space="ap1", format="rgb32f", denoise=1.0,
              exact_rounding=True),
        # A clip's frame with its history and the chroma denoise.
        _case(name="clip_chroma", path="clip", width=5760, height=3240, debayer="mhc", space="p3",
              denoise=1.0, temporal=0.8, chroma=0.5),
        # An HD stream's frame with its history.
        _case(name="clip_hd_ap0", path="clip", width=1920, height=1080, space="ap0", format="rgb32f",
              denoise=1.0, temporal=0.8),
        # A large still whose highlights clip, pushed a stop.
        _case(name="still_highlights", width=6000, height=4000, space="ap1", format="rgb32f",
              highlights=True, stops=1.0, noise_a=2.0, noise_b=16.0),
        # A contact sheet: previews of uneven sizes in one batch.
        _case(name="batch_previews", path="batch", sizes="640x360*24,480x320*12,518x262*12",
              space="bt2020", format="rgba16f", denoise=1.0),
        # A day's mixed footage and stills in one batch.
        _case(name="batch_mix", path="batch", sizes="1920x1080*6,3840x2160*4,5760x3240*4,6000x4000*2",
              space="bt2020", format="rgb32f", denoise=1.0),
        # The noise model of a camera that has none, from one frame on the device.
        _case(name="noise_model", path="noise", width=5760, height=3240),
        # Four clips served from and to host memory, two frames each.
        _case(name="serve_hd", path="serve", sizes="1920x1080*2,1280x720*2", frames=2, space="ap0",
              format="rgba16f", denoise=1.0, temporal=0.8),
    ]


def draw(rng) -> dict:
    def size(lo, hi):
        w = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        a = rng.choice((16 / 9, 3 / 2, 4 / 3, 2.39, 1.0)) * rng.uniform(0.97, 1.03)
        return int(w) // 2 * 2, max(32, int(w / a) // 2 * 2)

    noise = dict(noise_a=round(rng.uniform(1.0, 8.0), 2), noise_b=round(rng.uniform(10.0, 80.0), 1))
    look = dict(space=rng.choice(tuple(SPACES)), format=rng.choice(tuple(FORMATS)),
                stops=rng.choice((0.0, 0.0, 0.5, -1.0)), clamp=rng.random() < 0.25, **noise)
    debayer = rng.choice(("bilinear", "mhc", "rcd", "rcd"))
    strength = round(rng.uniform(0.5, 2.0), 2)
    kind = rng.choice(("frame", "frame", "denoise", "denoise", "exact", "clip", "clip", "chroma", "still",
                       "live", "batch", "batch", "noise", "serve"))
    if kind == "batch":
        many = rng.random() < 0.5
        sizes = [size(256, 960) if many else size(960, 6000) for _ in range(4)]
        n = rng.randint(2, 10) if many else rng.randint(1, 2)
        return _case(path="batch", sizes=",".join("%dx%d*%d" % (w, h, n) for w, h in sizes), debayer=debayer,
                     denoise=strength, **look)
    if kind == "serve":
        sizes = [size(480, 2048) for _ in range(rng.randint(2, 4))]
        return _case(path="serve", sizes=",".join("%dx%d*1" % s for s in sizes), frames=2, debayer=debayer,
                     denoise=strength, temporal=round(rng.uniform(0.4, 0.9), 2),
                     **{**look, "format": "rgba16f"})
    if kind == "noise":
        w, h = size(1920, 6000)
        return _case(path="noise", width=w, height=h, **noise)
    w, h = size(320, 1280) if kind == "live" else size(320, 6000)
    if kind in ("denoise", "clip", "chroma") and w * h < 1900000:
        # A proxy's format. (Below this size the denoise's timed choice of
        # tile differs from run to run, and with it the rounding of a few
        # codes, which a 32-bit output would show.)
        look["format"] = "rgba16f"
    more = {
        "live": dict(path="live"),
        "frame": dict(awb=rng.random() < 0.7, storage=rng.choice(("fp32", "fp32", "fp16"))),
        "denoise": dict(denoise=strength),
        "exact": dict(denoise=strength, exact_rounding=True, debayer="rcd"),
        "clip": dict(path="clip", denoise=strength, temporal=round(rng.uniform(0.4, 0.9), 2)),
        "chroma": dict(path="clip", denoise=strength, temporal=round(rng.uniform(0.4, 0.9), 2),
                       chroma=round(rng.uniform(0.2, 1.0), 2)),
        "still": dict(highlights=True),
    }[kind]
    return _case(**{**dict(width=w, height=h, debayer=debayer), **look, **more})


def _sizes(case) -> list[tuple[int, int]]:
    if "sizes" not in case:
        return [(case["width"], case["height"])]
    out = []
    for part in case["sizes"].split(","):
        wh, n = part.split("*")
        w, h = wh.split("x")
        out += [(int(w), int(h))] * int(n)
    return out


# ------------------------------------------------------------------ inputs


def scene(w: int, h: int, seed: int, case: dict, step: int = 0, ramp: bool = False) -> torch.Tensor:
    """One (h, w) int32 RGGB mosaic on the GPU: a gradient, flat rectangles
    (every third moves by `step` frames), a zone plate, and sensor noise of
    variance a s + b; with the highlights clipped where the case rebuilds
    them. `ramp`: the gradient alone, as a chart for the noise model."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + w * 31 + h)
    rng = np.random.RandomState(seed % (1 << 32))
    y = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
    x = torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
    if ramp:
        lo, hi = rng.uniform(0.005, 0.02), rng.uniform(0.85, 0.95)
        sig = (lo + (hi - lo) * x / (w - 1)).expand(h, w).clone()
    else:
        tone = rng.uniform(0.6, 1.0, 3)
        base = (0.08 + 0.55 * (0.6 * x / w + 0.4 * y / h))
        rgb = torch.stack([base * float(t) for t in tone])
        for i in range(48):
            x0, y0 = int(rng.uniform(-0.05, 0.95) * w), int(rng.uniform(-0.05, 0.95) * h)
            rw, rh = int(rng.uniform(0.02, 0.25) * w) + 2, int(rng.uniform(0.02, 0.25) * h) + 2
            colour = rng.uniform(0.02, 0.9, 3)
            if i % 3 == 0:
                x0 += 5 * step
            rgb[:, max(0, y0):max(0, y0 + rh), max(0, x0):max(0, x0 + rw)] = torch.tensor(
                colour, device="cuda", dtype=torch.float32)[:, None, None]
        cx, cy, r = rng.uniform(0.2, 0.8) * w, rng.uniform(0.2, 0.8) * h, 0.18 * min(w, h)
        d2 = (x - cx) ** 2 + (y - cy) ** 2
        rgb = torch.where(d2 < r * r, 0.4 + 0.3 * torch.cos(d2 * (math.pi / (2 * r))), rgb)
        if case["highlights"]:
            rgb = rgb * 1.6
            for _ in range(3):
                cx, cy, r = rng.uniform(0, w), rng.uniform(0, h), rng.uniform(0.04, 0.12) * min(w, h)
                rgb = rgb + 2.0 * (1.0 - ((x - cx) ** 2 + (y - cy) ** 2).sqrt() / r).clamp(0.0, 1.0)
        sig = torch.empty((h, w), device="cuda")
        for s in range(4):
            sig[s >> 1::2, s & 1::2] = rgb[CHANNEL[s], s >> 1::2, s & 1::2] / WB[CHANNEL[s]]
        if case["highlights"]:
            sig = sig * max(WB)
    sig = sig * RANGE
    # A frame of its own noise for each step of a clip.
    n = torch.randn((h, w), generator=g, device="cuda")
    for _ in range(step):
        n = torch.randn((h, w), generator=g, device="cuda")
    v = BLACK + sig + n * (case["noise_a"] * sig + case["noise_b"]).clamp_min(0.0).sqrt()
    return v.round().clamp(0, WHITE).to(torch.int32)


def _inputs(case, seed) -> list[torch.Tensor]:
    """The mosaics a pass of the case reads, in order."""
    path = case["path"]
    if path == "clip":
        return [scene(case["width"], case["height"], seed, case, step) for step in range(2)]
    if path == "serve":
        return [scene(w, h, seed + 7 * i, case, step)
                for i, (w, h) in enumerate(_sizes(case)) for step in range(case["frames"])]
    return [scene(w, h, seed + 7 * i, case, ramp=path == "noise") for i, (w, h) in enumerate(_sizes(case))]


# ------------------------------------------------------- the library's side


def profile() -> L.Profile:
    p = L.profile_init()
    for s in range(4):
        p.black_level[s], p.white_level[s] = BLACK / 65535.0, WHITE / 65535.0
    for c in range(3):
        p.as_shot_wb[c] = WB[c]
        for j in range(3):
            p.as_shot_matrix[c][j] = CAMERA[c][j]
    p.as_shot_cct = 5500.0
    return p


def _device_mosaic(m: torch.Tensor) -> tuple[torch.Tensor, L.Image]:
    h, w = m.shape
    t = torch.zeros((h, (w + 7) // 8 * 8), dtype=torch.int16, device="cuda")
    t[:, :w] = m.to(torch.int16)
    return t, L.Image(t.data_ptr(), t.stride(0) * 2, L.FORMAT_R16_UNORM, w, h)


def _output(case, w, h, host=False) -> tuple[torch.Tensor, int]:
    """An output image, and its row pitch in bytes."""
    where = dict(pin_memory=True) if host else dict(device="cuda")
    fmt = case["format"]
    if fmt == "rgb32f":
        row = (3 * w + 3) // 4 * 4
        t = torch.empty((h, row), dtype=torch.float32, **where)
        return t[:, :3 * w].unflatten(1, (w, 3)), row * 4
    t = torch.empty((h, w, 4), dtype=torch.float16 if fmt == "rgba16f" else torch.float32, **where)
    return t, t.stride(0) * t.element_size()


def _pipeline_params(case, w, h) -> L.PipelineParams:
    flags = ((L.FLAG_AWB_HISTOGRAM if case["awb"] else 0) | (L.FLAG_DENOISE if case["denoise"] else 0) |
             (L.FLAG_TEMPORAL_DENOISE if case["temporal"] else 0) |
             (L.FLAG_CHROMA_DENOISE if case["chroma"] else 0) |
             (L.FLAG_EXACT_ROUNDING if case["exact_rounding"] else 0) |
             (L.FLAG_HIGHLIGHT_RECONSTRUCTION if case["highlights"] else 0))
    return L.pipeline_params(w, h, debayer=DEBAYERS[case["debayer"]], out_space=SPACES[case["space"]],
                             out_format=FORMATS[case["format"]], flags=flags,
                             storage=L.STORAGE_FP16 if case["storage"] == "fp16" else L.STORAGE_FP32)


def _frame_params(case, prof, **kw) -> L.FrameParams:
    return L.frame_params(
        prof, exposure_stops=case["stops"], denoise_strength=case["denoise"],
        denoise_temporal_strength=case["temporal"], denoise_chroma_strength=case["chroma"],
        noise_override=(case["noise_a"] / RANGE, case["noise_b"] / RANGE ** 2),
        **{"flags": (L.FRAME_CLAMP_NEGATIVE if case["clamp"] else 0) |
           (L.FRAME_HIGHLIGHT_RECONSTRUCTION if case["highlights"] else 0), **kw})


class _DeviceImage:
    """A device image of a pipeline's own as torch reads it; the tensor
    over it keeps this object, and so the pipeline and its memory."""

    def __init__(self, pipe: L.Pipeline, img: L.Image, typestr: str):
        self.pipe = pipe
        self.__cuda_array_interface__ = {
            "shape": (img.height, img.width), "typestr": typestr, "data": (img.data, False),
            "strides": (img.pitch, int(typestr[2:])), "version": 3}


class State:
    """What a program keeps between passes."""


def prepare(case: dict, seed: int) -> State:
    st = State()
    st.path = case["path"]
    st.profile = profile()
    st.ctx = L.Context(0)
    st.stream = torch.cuda.current_stream().cuda_stream
    mosaics = _inputs(case, seed)
    sizes = _sizes(case)
    if st.path == "serve":
        st.host = [torch.empty(m.shape, dtype=torch.int16, pin_memory=True).copy_(m) for m in mosaics]
        st.server = L.Server(st.ctx, L.server_params(hbm_budget=16 << 30, max_inflight=8, slots_per_stream=2))
        ids = [st.server.open(L.server_stream_params(_pipeline_params(case, w, h))) for w, h in sizes]
        st.out, st.jobs = [], []
        # A clip's first frame starts without a history.
        fps = [_frame_params(case, st.profile, flags=L.FRAME_TEMPORAL_RESET if k == 0 else 0)
               for k in range(case["frames"])]
        for k in range(case["frames"]):
            for i, (w, h) in enumerate(sizes):
                src = st.host[i * case["frames"] + k]
                out, pitch = _output(case, w, h, host=True)
                st.out.append(out)
                st.jobs.append((ids[i], src.data_ptr(), src.stride(0) * 2, out.data_ptr(), pitch, fps[k]))
        return st
    pairs = [_device_mosaic(m) for m in mosaics]
    st.tensors, srcs = [t for t, _ in pairs], [im for _, im in pairs]
    if st.path == "noise":
        st.src = srcs[0]
        return st
    fmt = FORMATS[case["format"]]
    st.fp = _frame_params(case, st.profile)
    st.out, st.src, st.dst = [], srcs, []
    for w, h in sizes:
        out, pitch = _output(case, w, h)
        st.out.append(out)
        st.dst.append(L.Image(out.data_ptr(), pitch, fmt, w, h))
    if st.path == "batch":
        st.batch = L.Batch(st.ctx, L.batch_params(
            max(w for w, _ in sizes), max(h for _, h in sizes), max_frames=len(sizes),
            debayer=DEBAYERS[case["debayer"]], out_space=SPACES[case["space"]], out_format=fmt,
            flags=L.FLAG_DENOISE))
        st.fps = [st.fp] * len(sizes)
        return st
    w, h = sizes[0]
    st.pipe = L.Pipeline(st.ctx, _pipeline_params(case, w, h))
    if st.path == "clip":
        # The clip's first frame, then the frame that run() develops: a
        # replay develops it again from the same history.
        for k in range(2):
            st.pipe.record(st.stream, srcs[k], st.dst[0], st.fp)
        st.fp = _frame_params(case, st.profile, denoise_temporal_replay=True)
        st.src = srcs[1:]
        torch.cuda.current_stream().synchronize()
        level, var = st.pipe.temporal_state()
        st.out += [torch.as_tensor(_DeviceImage(st.pipe, level, "<f4"), device="cuda"),
                   torch.as_tensor(_DeviceImage(st.pipe, var, "|u1"), device="cuda")]
    return st


def run(st: State):
    if st.path == "serve":
        for i, (sid, src, pitch, dst, dst_pitch, fp) in enumerate(st.jobs):
            st.server.submit(sid, src, pitch, dst, dst_pitch, fp, user=i)
        st.server.drain()
        for r in st.server.poll(len(st.jobs)):
            if r.status:
                raise L.CrawError(r.status, "a served frame")
        return st.out
    if st.path == "noise":
        e = L.noise_estimate_cuda(st.src, st.profile, stream=st.stream)
        return {"a": e.model.a, "b": e.model.b, "fit_rms": e.fit_rms, "read_noise": e.read_noise_lsb,
                "bins": e.nb_bins, "inliers": e.nb_inliers}
    if st.path == "batch":
        st.batch.record(st.stream, st.src, st.dst, st.fps)
        return st.out
    st.pipe.record(st.stream, st.src[0], st.dst[0], st.fp)
    if st.path == "live":
        # The loop needs this frame's reading before the next frame.
        torch.cuda.current_stream().synchronize()
        hist = st.pipe.awb_histogram()
        return [st.out[0], hist.count, hist.weight, hist.weight_bright]
    return st.out


def work(case: dict) -> dict:
    bytes_, flops = 0, 0
    for w, h in _sizes(case):
        n = w * h * case.get("frames", 1)
        if case["path"] == "noise":
            bytes_ += 2 * n
            flops += n * (81 + 15)
            continue
        bytes_ += n * (2 + PIXEL_BYTES[case["format"]])
        flops += n * {"bilinear": 10, "mhc": 20, "rcd": 110}[case["debayer"]] + 20 * n
        if case["denoise"]:
            flops += n * 49 * 13
        if case["temporal"]:
            bytes_ += n * 10                 # the state read and written
            flops += n * 40
        if case["chroma"]:
            flops += n // 16 * 81 * 14 + n * 30
        if case["highlights"]:
            flops += n * 20
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------------- in 64 bits


def _pad(v, r):
    return F.pad(v[None, None], (r, r, r, r), mode="reflect")[0, 0]


def _around(v, r):
    """at(dx, dy): v moved by (dx, dy), mirrored at its edges."""
    h, w = v.shape
    p = _pad(v, r)
    return lambda dx, dy: p[r + dy:r + dy + h, r + dx:r + dx + w]


def _box3(v):
    """3x3 sums of the inside of v."""
    return F.avg_pool2d(v[None, None], 3, 1)[0, 0] * 9.0


def _levels():
    b, w = float(np.float32(BLACK / 65535.0)), float(np.float32(WHITE / 65535.0))
    return b, w - b


class _Transform:
    """The variance-stabilising transform of a noise model."""

    def __init__(self, case):
        self.a = float(np.float32(case["noise_a"] / RANGE))
        b = float(np.float32(case["noise_b"] / RANGE ** 2))
        self.c = 3.0 * self.a ** 2 / 8.0 + b
        self.sc = math.sqrt(self.c)
        self.t0 = 2.0 / self.a * self.sc

    def forward(self, u):
        root = 2.0 / self.a * (self.a * u.clamp_min(0.0) + self.c).sqrt()
        return torch.where(u >= 0, root, self.t0 + u / self.sc)

    def inverse(self, t):
        return torch.where(t >= self.t0, self.a / 4.0 * t * t - self.c / self.a, (t - self.t0) * self.sc)


def _nlm(t, var, inv_h2):
    """Non-local means of one plane: 7x7 search, 3x3 patches."""
    h, w = t.shape
    p = _pad(t, 4)
    vp = _pad(var, 4) if var is not None else None
    own = p[3:h + 5, 3:w + 5]
    acc, total = torch.zeros_like(t), torch.zeros_like(t)
    for dy in range(-3, 4):
        for dx in range(-3, 4):
            d2 = _box3((own - p[3 + dy:h + 5 + dy, 3 + dx:w + 5 + dx]).square()) * (inv_h2 / 9.0)
            if vp is None:
                wt = (2.0 - d2).clamp_max(0.0).exp()
            else:
                wt = ((var + vp[4 + dy:h + 4 + dy, 4 + dx:w + 4 + dx] - d2).clamp_max(0.0) / var).exp()
            acc += wt * p[4 + dy:h + 4 + dy, 4 + dx:w + 4 + dx]
            total += wt
    return acc / total


def _denoised(case, mosaic, history=None):
    """The denoised mosaic's codes, and the next state (level, variance)."""
    tr, (black, rng) = _Transform(case), _levels()
    inv_h2 = 1.0 / float(np.float32(case["denoise"])) ** 2 if case["denoise"] else 1.0
    alpha = float(np.float32(case["temporal"]))
    out = torch.empty_like(mosaic, dtype=torch.float64)
    level, variance = torch.empty_like(out), torch.ones_like(out)
    for s in range(4):
        at = (slice(s >> 1, None, 2), slice(s & 1, None, 2))
        u0 = (mosaic[at].double() / 65535.0 - black) / rng
        t, var = tr.forward(u0), None
        if history is not None:
            prev = tr.forward(history[0][at])
            a = alpha * (2.0 - _box3(_pad(prev - t, 1).square()) * (inv_h2 / 9.0)).clamp_max(0.0).exp()
            var = ((1.0 - a).square() + a.square() * history[1][at]).clamp_min(float(np.float32(1e-4)))
            t = t * (1.0 - a) + prev * a
            variance[at] = ((var.clamp(0.0, 1.0).sqrt() * 255.0).round() / 255.0).square()
        level[at] = tr.inverse(t)
        u = tr.inverse(_nlm(t, var, inv_h2)) if case["denoise"] else level[at]
        lo, hi = float(np.float32(0.9)), 1.0
        guard = ((u0 - lo) / (hi - lo)).clamp(0.0, 1.0)
        u = u + (u0 - u) * guard
        out[at] = ((black + u * rng).clamp(0.0, 1.0) * 65535.0).round()
    return out, (level, variance)


def _site_masks(h, w):
    s = (torch.arange(h, device="cuda")[:, None] % 2) * 2 + torch.arange(w, device="cuda")[None, :] % 2
    return [s == i for i in range(4)]


def _assemble(own, masks, at_r, at_gr, at_gb, at_b):
    """RGB planes from what each site knows of (R, G, B); None: its own."""
    out = torch.empty((3,) + own.shape, dtype=own.dtype, device=own.device)
    for m, values in zip(masks, (at_r, at_gr, at_gb, at_b)):
        for c in range(3):
            out[c] = torch.where(m, own if values[c] is None else values[c], out[c])
    return out


def _bilinear(v):
    n = _around(v, 1)
    edge = 0.25 * (n(0, -1) + n(0, 1) + n(-1, 0) + n(1, 0))
    corner = 0.25 * (n(-1, -1) + n(1, -1) + n(-1, 1) + n(1, 1))
    hz, vt = 0.5 * (n(-1, 0) + n(1, 0)), 0.5 * (n(0, -1) + n(0, 1))
    return _assemble(v, _site_masks(*v.shape), (None, edge, corner), (hz, None, vt), (vt, None, hz),
                     (corner, edge, None))


def _mhc(v):
    n = _around(v, 2)
    h1, v1 = n(-1, 0) + n(1, 0), n(0, -1) + n(0, 1)
    h2, v2 = n(-2, 0) + n(2, 0), n(0, -2) + n(0, 2)
    diag = n(-1, -1) + n(1, -1) + n(-1, 1) + n(1, 1)
    g = (4.0 * v + 2.0 * (h1 + v1) - (h2 + v2)) / 8.0
    d = (6.0 * v + 2.0 * diag - 1.5 * (h2 + v2)) / 8.0
    hz = (5.0 * v + 4.0 * h1 - (diag + h2) + 0.5 * v2) / 8.0
    vt = (5.0 * v + 4.0 * v1 - (diag + v2) + 0.5 * h2) / 8.0
    return _assemble(v, _site_masks(*v.shape), (None, g, d), (hz, None, vt), (vt, None, hz), (d, g, None))


def _rcd(v):
    eps = float(np.float32(1e-5))
    n = _around(v, 2)
    masks = _site_masks(*v.shape)
    low = (4.0 * v + 2.0 * (n(0, -1) + n(0, 1) + n(-1, 0) + n(1, 0)) + n(-1, -1) + n(1, -1) + n(-1, 1) +
           n(1, 1)) / 16.0

    def strength(dx, dy):
        d = (n(-dx, -dy) - n(dx, dy)).abs() + (2.0 * v - n(-2 * dx, -2 * dy) - n(2 * dx, 2 * dy)).abs()
        return _box3(_pad(d, 1)) / 9.0

    vs, hs, ps, qs = strength(0, 1), strength(1, 0), strength(1, -1), strength(1, 1)
    wv, wp = hs / (hs + vs + eps), qs / (ps + qs + eps)
    del vs, hs, ps, qs
    l0 = low.clamp_min(0.0)
    l = _around(l0, 2)

    def ratio(dx, dy):
        return 1.0 + (l0 - l(dx, dy)) / (l0 + l(dx, dy) + eps)

    gv = 0.5 * (n(0, -1) * ratio(0, -2) + n(0, 1) * ratio(0, 2))
    gh = 0.5 * (n(-1, 0) * ratio(-2, 0) + n(1, 0) * ratio(2, 0))
    green = torch.where(masks[1] | masks[2], v, wv * gv + (1.0 - wv) * gh)
    del gv, gh, low, l0
    d = _around(v - green, 1)                # colour minus green
    cross = green + 0.5 * (wp * (d(-1, 1) + d(1, -1)) + (1.0 - wp) * (d(-1, -1) + d(1, 1)))
    o = _around(cross - green, 1)            # the other colour minus green, at R and B
    ch = green + 0.5 * (wv * (o(0, -1) + o(0, 1)) + (1.0 - wv) * (d(-1, 0) + d(1, 0)))
    cv = green + 0.5 * (wv * (d(0, -1) + d(0, 1)) + (1.0 - wv) * (o(-1, 0) + o(1, 0)))
    return _assemble(v, masks, (None, green, cross), (ch, None, cv), (cv, None, ch), (cross, green, None))


def _chroma(rgb, strength):
    """Denoises the colour differences on quarter-resolution block means."""
    _, h, w = rgb.shape
    qh, qw = (h + 3) // 4, (w + 3) // 4
    diff = torch.stack([rgb[0] - rgb[1], rgb[2] - rgb[1], rgb[1]])
    fill = (0, 4 * qw - w, 0, 4 * qh - h)
    count = F.avg_pool2d(F.pad(torch.ones_like(rgb[:1]), fill)[None], 4)[0]
    down = F.avg_pool2d(F.pad(diff, fill)[None], 4)[0] / count
    n = [_around(down[c], 4) for c in range(3)]
    inv = 1.0 / (float(np.float32(0.35)) * (down[2].clamp_min(0.0) + float(np.float32(0.02))))
    acc, total = [torch.zeros_like(inv) for _ in range(2)], torch.zeros_like(inv)
    for dy in range(-4, 5):
        for dx in range(-4, 5):
            far = sum(((n[c](dx, dy) - down[c]) * inv).square() for c in range(3))
            wt = (-(dx * dx + dy * dy) / 8.0 - far).exp()
            total += wt
            for c in range(2):
                acc[c] += wt * n[c](dx, dy)
    change = torch.stack([acc[c] / total - down[c] for c in range(2)])

    def taps(size, q):
        f = (torch.arange(size, device="cuda", dtype=torch.float64) + 0.5) * 0.25 - 0.5
        lo = f.floor()
        return lo.long().clamp(0, q - 1), (lo.long() + 1).clamp(0, q - 1), f - lo

    y0, y1, ty = taps(h, qh)
    x0, x1, tx = taps(w, qw)
    rows = change[:, y0] * (1.0 - ty)[:, None] + change[:, y1] * ty[:, None]
    up = rows[:, :, x0] * (1.0 - tx) + rows[:, :, x1] * tx
    k = float(np.float32(strength))
    return torch.stack([rgb[0] + k * up[0], rgb[1], rgb[2] + k * up[1]])


def _rebuilt(u, wb):
    """The balanced mosaic of levels u with its clipped highlights lifted,
    at half precision: a pyramid of the log chroma of the unclipped quads,
    pulled up to one texel and pushed down again, and each site near the
    clip lifted toward what its neighbours and that colour field predict."""
    h, w = u.shape
    f32 = lambda x: float(np.float32(x))                                   # noqa: E731
    lo, hi, eps = f32(0.92), f32(0.98), f32(1e-4)
    s = ((u - lo) / (hi - lo)).clamp(0.0, 1.0)
    clipped = s * s * (3.0 - 2.0 * s)
    quads = lambda v: [v[i >> 1::2, i & 1::2] for i in range(4)]           # noqa: E731
    amax = F.max_pool2d(torch.stack(quads(clipped)).amax(0)[None, None], 7, 1, 3)[0, 0]
    us = quads(u)
    bright = torch.stack(us).amax(0).clamp_max(1.0)
    wq = (1.0 - amax) * bright * bright
    g = (0.5 * wb[1] * (us[1] + us[2])).clamp_min(eps)
    chroma = [(wb[c] * us[i]).clamp_min(eps).div(g).log().clamp(-2.0, 2.0) for c, i in ((0, 0), (2, 3))]
    level = torch.stack([wq * chroma[0], wq * chroma[1], wq])

    def halve(t):
        t = F.pad(t, (0, t.shape[2] % 2, 0, t.shape[1] % 2))
        return t[:, 0::2, 0::2] + t[:, 0::2, 1::2] + t[:, 1::2, 0::2] + t[:, 1::2, 1::2]

    pyramid = [halve(level)]
    while pyramid[-1].shape[1:] != (1, 1):
        pyramid.append(halve(pyramid[-1]))

    def sample(c, fy, fx):
        y0, x0 = fy.floor(), fx.floor()
        ty, tx = (fy - y0)[:, None], fx - x0
        ys = [(y0.long() + i).clamp(0, c.shape[1] - 1) for i in (0, 1)]
        xs = [(x0.long() + i).clamp(0, c.shape[2] - 1) for i in (0, 1)]
        rows = [c[:, y][:, :, xs[0]] * (1.0 - tx) + c[:, y][:, :, xs[1]] * tx for y in ys]
        return rows[0] * (1.0 - ty) + rows[1] * ty

    def grid(size, scale, shift):
        return torch.arange(size, device="cuda", dtype=torch.float64) * scale + shift

    top = pyramid[-1]
    field = torch.where(top[2] > 0, top[:2] / top[2], torch.zeros_like(top[:2]))
    for t in reversed(pyramid[:-1]):
        field = sample(field, grid(t.shape[1], 0.5, -0.25), grid(t.shape[2], 0.5, -0.25))
        mean = torch.where(t[2] > 0, t[:2] / t[2], field)
        field = field + t[2].clamp(0.0, 1.0) * (mean - field)
    field = sample(field, grid(h // 2, 0.5, -0.25), grid(w // 2, 0.5, -0.25))
    rho = torch.stack([field[0], torch.zeros_like(field[0]), field[1]])

    balanced = torch.empty_like(u)
    for i in range(4):
        balanced[i >> 1::2, i & 1::2] = us[i] * wb[CHANNEL[i]]
    at = {(dx, dy): (_around(balanced, 1)(dx, dy), _around(clipped, 1)(dx, dy))
          for dx in (-1, 0, 1) for dy in (-1, 0, 1) if (dx, dy) != (0, 0)}
    out = torch.empty_like(u)
    for i in range(4):
        q = (slice(i >> 1, None, 2), slice(i & 1, None, 2))
        own = CHANNEL[i]
        x, a = balanced[q], clipped[q]
        logs, spare = [], []
        for k in (c for c in range(3) if c != own):
            near = [(p[0][q], p[1][q]) for (dx, dy), p in at.items()
                    if CHANNEL[((i >> 1) ^ (dy & 1)) * 2 + ((i & 1) ^ (dx & 1))] == k]
            mean = sum(p for p, _ in near) / len(near)
            logs.append(mean.clamp_min(eps).log() - rho[k])
            spare.append(1.0 - torch.stack([c for _, c in near]).amax(0))
        l_own = x.clamp_min(eps).log() - rho[own]
        full = torch.maximum(l_own, torch.maximum(*logs)).exp()
        room = spare[0] + spare[1]
        part = ((spare[0] * logs[0] + spare[1] * logs[1]) / room.clamp_min(1e-300)).exp()
        part = torch.where(room > 0, part, full)
        lift = (full + room.clamp_max(1.0) * (part - full)) * rho[own].exp() - x
        out[q] = torch.where(a > 0, x + a * lift.clamp_min(0.0), x)
    return out.half().double()


def _matrix(space):
    """XYZ (D65) to the space's linear RGB, from its primaries and white."""
    prim = {"bt709": ((0.64, 0.33), (0.30, 0.60), (0.15, 0.06)),
            "bt2020": ((0.708, 0.292), (0.170, 0.797), (0.131, 0.046)),
            "p3": ((0.680, 0.320), (0.265, 0.690), (0.150, 0.060)),
            "ap0": ((0.7347, 0.2653), (0.0, 1.0), (0.0001, -0.0770)),
            "ap1": ((0.713, 0.293), (0.165, 0.830), (0.128, 0.044))}[space]
    xyz = lambda x, y: np.array([x / y, 1.0, (1.0 - x - y) / y])           # noqa: E731
    d65, aces = xyz(0.3127, 0.3290), xyz(0.32168, 0.33767)
    white = aces if space in ("ap0", "ap1") else d65
    m = np.stack([xyz(*p) for p in prim], 1)
    m = m * np.linalg.solve(m, white)
    if white is aces:
        cone = np.array([[0.8951, 0.2664, -0.1614], [-0.7502, 1.7135, 0.0367], [0.0389, -0.0685, 1.0296]])
        m = np.linalg.solve(cone, np.diag(cone @ d65 / (cone @ aces)) @ cone) @ m
    return np.linalg.inv(m)


def _coloured(case, rgb):
    m = _matrix(case["space"]) @ np.array(CAMERA, np.float32).astype(np.float64) * 2.0 ** case["stops"]
    out = torch.stack([sum(float(m[r, c]) * rgb[c] for c in range(3)) for r in range(3)])
    if case["space"] == "ap1":               # the ACES reference gamut compression
        limit, thr, power = (1.147, 1.264, 1.312), (0.815, 0.803, 0.880), 1.2
        ach = out.amax(0)
        mag = ach.abs()
        for c in range(3):
            scale = (limit[c] - thr[c]) / (((1 - thr[c]) / (limit[c] - thr[c])) ** -power - 1) ** (1 / power)
            d = (ach - out[c]) / mag
            nd = ((d - thr[c]) / scale).clamp_min(0.0)
            d = torch.where(d < thr[c], d, thr[c] + scale * nd / (1.0 + nd ** power) ** (1 / power))
            out[c] = torch.where(ach == 0, out[c], ach - d * mag)
    if case["clamp"]:
        out = out.clamp_min(0.0)
    return out


def _image(case, codes):
    """A developed frame from its (denoised) codes, as the format holds it."""
    black, rng = _levels()
    u = (codes.double() / 65535.0 - black) / rng
    if case["highlights"]:
        v = _rebuilt(u, WB)
    else:
        v = u
        for s in range(4):
            v[s >> 1::2, s & 1::2] *= WB[CHANNEL[s]]
        v = v.clamp_max(1.0)
    rgb = {"bilinear": _bilinear, "mhc": _mhc, "rcd": _rcd}[case["debayer"]](v)
    if case["chroma"]:
        rgb = _chroma(rgb, case["chroma"])
    out = _coloured(case, rgb)
    if case["format"] != "rgb32f":
        out = torch.cat([out, torch.ones_like(out[:1])])
    return out.permute(1, 2, 0)


def _noise_model(mosaic):
    """The noise model var = a u + b of one mosaic: bins by the 9x9 mean of
    each plane, the median absolute 3x3 high-pass of a bin for its noise, a
    least-trimmed-squares line through them and a robust refinement."""
    black, rng = _levels()
    bins = 128
    kernel = torch.tensor([[1.0, -2.0, 1.0], [-2.0, 4.0, -2.0], [1.0, -2.0, 1.0]], dtype=torch.float64,
                          device="cuda")[None, None] / 6.0
    means, noise = [], []
    for s in range(4):
        p = ((mosaic[s >> 1::2, s & 1::2].double() / 65535.0 - black) / rng)[None, None]
        means.append(F.avg_pool2d(p, 9, 1).flatten())
        noise.append(F.conv2d(p[..., 3:-3, 3:-3], kernel).flatten().abs())
    mean, hp = torch.cat(means), torch.cat(noise)
    keep = (mean > 0) & (mean <= float(np.float32(0.98)))
    mean, hp = mean[keep], hp[keep]
    b = (mean.sqrt() * bins).long().clamp(0, bins - 1)
    hp, order = hp.sort()
    b, order2 = b[order].sort(stable=True)
    hp = hp[order2].cpu().numpy()
    mean = mean[order][order2]
    count = torch.bincount(b, minlength=bins).cpu().numpy()
    start = np.concatenate([[0], np.cumsum(count)])
    m, v, n = [], [], []
    for i in range(bins):
        if count[i] < 20000:
            continue
        sigma = hp[start[i] + count[i] // 2] / 0.674489750196081746
        if sigma > 0:
            m.append(float(mean[start[i]:start[i + 1]].mean()))
            v.append(sigma ** 2)
            n.append(float(count[i]))
    m, v, n = np.array(m), np.array(v), np.array(n)
    lv, nb = np.log(v), len(m)
    keep = nb * 2 // 3 + 1
    best = (math.inf, 0.0, 0.0)
    for i in range(nb):
        for j in range(i + 1, nb):
            if m[j] - m[i] < 1e-5:
                continue
            ca = (v[j] - v[i]) / (m[j] - m[i])
            cb = v[i] - ca * m[i]
            if ca > 0 and not cb < 0:
                cost = float(np.sort((lv - np.log(ca * m + cb)) ** 2)[:keep].sum())
                if cost < best[0]:
                    best = (cost, ca, cb)
    la, lb = math.log(best[1]), math.log(max(best[2], 1e-16))
    scale = max(math.sqrt(best[0] / keep), 0.02)
    for it in range(40):
        ea, eb = math.exp(la), math.exp(lb)
        den = ea * m + eb
        res = lv - np.log(den)
        if it % 8 == 0:
            scale = max(1.4826 * np.sort(np.abs(res))[nb // 2], 0.02)
        q = res / (4.685 * scale)
        wt = np.where(np.abs(q) < 1.0, (1.0 - q * q) ** 2, 0.0) * np.log1p(n)
        ja, jb = ea * m / den, eb / den
        aa, ab, bb = (wt * ja * ja).sum() + 1e-9, (wt * ja * jb).sum(), (wt * jb * jb).sum() + 1e-9
        ra, rb = (wt * ja * res).sum(), (wt * jb * res).sum()
        det = aa * bb - ab * ab
        if not abs(det) > 1e-30:
            break
        d0 = min(0.5, max(-0.5, (bb * ra - ab * rb) / det))
        d1 = min(0.5, max(-0.5, (aa * rb - ab * ra) / det))
        la, lb = la + d0, max(-40.0, lb + d1)
        if abs(d0) < 1e-9 and abs(d1) < 1e-9:
            break
    a, b = math.exp(la), 0.0 if lb <= -40.0 else math.exp(lb)
    d = lv - np.log(a * m + b)
    d = d[np.abs(d) < 0.35]
    return {"a": a, "b": b, "fit_rms": math.sqrt((d * d).sum() / max(1, len(d))),
            "read_noise": math.sqrt(b) * rng * 65535.0, "bins": None, "inliers": None}


def exact(case: dict, seed: int):
    path = case["path"]
    mosaics = _inputs(case, seed)
    if path == "noise":
        return {k: v if v is None else torch.tensor(v, dtype=torch.float64)
                for k, v in _noise_model(mosaics[0]).items()}
    if path == "clip":
        _, state = _denoised(case, mosaics[0])
        codes, (level, _) = _denoised(case, mosaics[1], state)
        return [_image(case, codes), level, None]
    if path == "serve":
        out, nf = {}, case["frames"]
        for i in range(len(_sizes(case))):
            state = None
            for k in range(nf):
                codes, state = _denoised(case, mosaics[i * nf + k], state)
                out[k, i] = _image(case, codes)
        return [out[k, i] for k in range(nf) for i in range(len(_sizes(case)))]
    images = [_image(case, _denoised(case, m)[0] if case["denoise"] else m) for m in mosaics]
    return [images[0], None, None, None] if path == "live" else images
