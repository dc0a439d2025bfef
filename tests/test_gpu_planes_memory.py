"""GPU: creating a pipeline with a temporal history on a device that is nearly
full (craw_debug_limit_alloc): its averaged planes are optional, so they never
take the memory of what it needs."""
import ctypes as C

import numpy as np
import pytest

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from gpu_util import develop

pytestmark = pytest.mark.gpu

W2, H2 = 2078, 1046
SLACK = 1 << 16


def params(h=H2):
    return L.pipeline_params(W2, h, debayer=L.DEBAYER_BILINEAR, out_space=L.CS_BT709, out_format=L.FORMAT_RGBA32F,
                             flags=L.FLAG_DENOISE | L.FLAG_TEMPORAL_DENOISE)


def frame_params():
    return L.frame_params(W.make_profile(), denoise_strength=1.0, denoise_temporal_strength=0.8,
                          noise_override=W.noise_model(4.0, 40.0))


def clip(pipe):
    fp = frame_params()
    return [develop(pipe, W.synth_frame(W2, H2, 7, frame=f, rects=16, noise_a_dn=4.0, noise_b_dn=40.0,
                                        movers=[(3.0, 0.5)]), fp) for f in range(3)]


def created(ctx, limit, h=H2):
    L.debug_limit_alloc(limit)
    try:
        return L.Pipeline(ctx, params(h))
    except L.CrawError as e:
        assert e.errno == 12
        return None
    finally:
        L.debug_limit_alloc(0)


def need(ctx, h=H2):
    """The least memory (to SLACK) a pipeline of a shape without planes is
    created in, its shape not timed."""
    L.debug_force_denoise_shape(L.DN_SHAPES.index("2x4 f32x2"))
    lo, hi = 0, 64 * W2 * h
    while hi - lo > SLACK:
        mid = (lo + hi) // 2
        pipe = created(ctx, mid, h)
        lo, hi = (lo, mid) if pipe else (mid, hi)
        if pipe:
            pipe.close()
    L.debug_force_denoise_shape(-1)
    return hi


@pytest.fixture(scope="module")
def ctx():
    c = L.Context(0)
    yield c
    L.debug_force_denoise_shape(-1)
    L.debug_limit_alloc(0)
    c.close()


# The timing of the shapes takes 7 bytes a pixel beside the pipeline's own (a
# mosaic, a state's level and variance), the planes over 8. A size each, since
# a size is timed once a process.
@pytest.mark.parametrize("i,over", list(enumerate([7, 8, 9, 10, 12, 14, 16, 18])))
def test_created_where_only_the_planes_do_not_fit(ctx, i, over):
    h = H2 + 2 + 2 * i
    pitches = 3 * 256 * h          # rows rounded up to 256 bytes
    pipe = created(ctx, need(ctx, h) + over * W2 * h + pitches + SLACK, h)
    assert pipe is not None
    pipe.close()


def test_same_frames_with_and_without(ctx):
    least = need(ctx)
    L.debug_force_denoise_shape(L.DN_SHAPES.index("2x8 f32x2"))
    try:
        with L.Pipeline(ctx, params()) as pipe:
            want = clip(pipe)
        pipe = created(ctx, least)          # nothing for the planes
        assert pipe is not None
        with pipe:
            got = clip(pipe)
    finally:
        L.debug_force_denoise_shape(-1)
    for a, b in zip(want, got):
        assert np.array_equal(a, b)


class ContextWithLog(L.Context):
    """A context that keeps the formats of what is logged."""

    def __init__(self):
        self.said = []
        self._cb = C.CFUNCTYPE(None, C.c_void_p, C.c_int, C.c_char_p, C.c_void_p)(
            lambda opaque, level, fmt, args: self.said.append(fmt.decode()))
        opts = L.ContextOptions()
        opts.log_cb = C.cast(self._cb, C.c_void_p).value
        opts.log_level = 8             # verbose
        self._h, self._children, self.device = C.c_void_p(), [], 0
        assert L.lib().craw_context_create(C.byref(self._h), C.byref(L.CudaInitParams(0, None)), C.byref(opts)) == 0


def test_shape_timed_without_planes_is_not_remembered():
    """The history's shape timed where its planes did not fit is timed again
    by the next pipeline of the size, and that one's is remembered."""
    h = H2 + 18
    with ContextWithLog() as ctx:
        least = need(ctx, h) + 7 * W2 * h + 3 * 256 * h + SLACK
        timed = []
        for limit in (least, 0, 0):
            ctx.said.clear()
            created(ctx, limit, h).close()
            timed.append(sum(m.startswith("autotune") for m in ctx.said))
    assert timed == [2, 1, 0]          # with and without a history; with; neither
