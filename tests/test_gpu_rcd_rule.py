"""GPU: the RCD of AP1 frames at the sizes where the library goes over from
tiles to walking warps (180000 pixels, 800000, with a kept intermediate or FP16
storage 1000000, borders two tiles wide, after a denoise): its choice, the
tiles and the walking warps give the same bits."""
import numpy as np
import pytest

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from gpu_util import develop, download_image

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
