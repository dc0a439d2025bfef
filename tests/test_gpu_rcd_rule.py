"""GPU: the RCD of AP1 frames at the sizes where the library goes over from
tiles to walking warps (180000 pixels, 800000, with a kept intermediate or FP16
storage 1000000, borders two tiles wide, after a denoise): its choice, the
tiles and the walking warps give the same bits."""
import numpy as np
import pytest
import torch

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from gpu_util import alloc_rgba, develop, download_image, upload_mosaic

pytestmark = pytest.mark.gpu

SIZES = [(8, 8), (64, 48), (130, 98), (480, 374), (480, 376), (640, 362), (642, 362), (640, 356),
         (1000, 800), (1002, 800), (1250, 800), (1252, 800)]
FORMS = [(L.FORMAT_RGBA32F, L.STORAGE_FP32, 0), (L.FORMAT_RGB32F, L.STORAGE_FP32, L.FLAG_AWB_HISTOGRAM),
         (L.FORMAT_RGBA16F, L.STORAGE_FP16, L.FLAG_AWB_HISTOGRAM),
         (L.FORMAT_RGBA32F, L.STORAGE_FP32, L.FLAG_KEEP_INTERMEDIATE),
         (L.FORMAT_RGBA16F, L.STORAGE_FP32, L.FLAG_DENOISE | L.FLAG_AWB_HISTOGRAM)]


@pytest.fixture(scope="module")
def ctx():
    c = L.Context(0)
    L.debug_force_denoise_shape(L.DN_SHAPES.index("2x4 f32x2"))
    yield c
    L.debug_force_denoise_shape(-1)
    L.debug_rcd_strips(1)
    c.close()


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("fmt,storage,flags", FORMS)
def test_choice_gives_the_same_bits(ctx, w, h, fmt, storage, flags):
    if flags & L.FLAG_DENOISE and min(w, h) < 10:
        pytest.skip("denoising needs a frame of at least 10x10")
    m = W.highlight_frame(w, h, w + h)
    fp = L.frame_params(W.make_profile(), denoise_strength=1.0 if flags & L.FLAG_DENOISE else 0.0,
                        noise_override=W.noise_model(4.0, 40.0))
    pp = L.pipeline_params(w, h, debayer=L.DEBAYER_RCD, out_space=L.CS_ACES_AP1, out_format=fmt, storage=storage,
                           flags=flags)
    got = []
    with L.Pipeline(ctx, pp) as pipe:
        for mode in (1, 0, 2):
            L.debug_rcd_strips(mode)
            r = [develop(pipe, m, fp, fmt)]
            if flags & L.FLAG_AWB_HISTOGRAM:
                hist = pipe.awb_histogram()
                r += [hist.count, hist.weight, hist.weight_bright]
            if flags & L.FLAG_KEEP_INTERMEDIATE:
                r.append(download_image(pipe.intermediate()[0], "rgba32f"))
            got.append(r)
        assert pipe.kernel_errors() == 0
    L.debug_rcd_strips(1)
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


FRAMES = 4


def recorded(graph, out_space, frame_space):
    """Frames of a clip recorded by tiles back to back into their own images
    (in a graph, the process's first use of the kernels): outputs, histograms."""
    w, h = 640, 362
    srcs = [upload_mosaic(W.highlight_frame(w, h, 5 + i)) for i in range(FRAMES)]
    outs = [alloc_rgba(w, h) for _ in srcs]
    kw = {} if frame_space is None else dict(out_space=frame_space, out_space_set=True)
    fp = L.frame_params(W.make_profile(), **kw)
    pp = L.pipeline_params(w, h, debayer=L.DEBAYER_RCD, out_space=out_space, out_format=L.FORMAT_RGBA32F,
                           flags=L.FLAG_AWB_HISTOGRAM, nb_awb_slots=FRAMES)
    with L.Context(0) as c, L.Pipeline(c, pp) as pipe:
        s = torch.cuda.Stream()
        torch.cuda.synchronize()

        def frames(wait):
            for (_, src), (_, dst) in zip(srcs, outs):
                pipe.record(s.cuda_stream, src, dst, fp)
                if wait:
                    torch.cuda.synchronize()
        if graph:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                frames(False)
            g.replay()
        else:
            frames(graph is None)
        torch.cuda.synchronize()
        assert pipe.kernel_errors() == 0
        hist = [pipe.awb_histogram(i) for i in range(FRAMES)]
    return [o.cpu().numpy() for o, _ in outs] + [a for x in hist for a in (x.count, x.weight, x.weight_bright)]


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("frame_space", [None, L.CS_ACES_AP1])
def test_back_to_back(graph, frame_space):
    space = L.CS_ACES_AP1 if frame_space is None else L.CS_BT709
    got, want = recorded(graph, space, frame_space), recorded(None, L.CS_ACES_AP1, None)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
