"""GPU: the packed denoise shapes against each other, bit for bit: 2x8 (rows
of the patch block read again from the tile; with a history the temporal
average by its own kernel into padded planes) and 2x4 (the average inside the
tile). Sequences of three frames with moving rectangles, their denoised
mosaic, output and next state, at the smallest frame, at sizes one short of
and one over a 32 x 16 plane tile, and with the tile copies by plain loads."""
import numpy as np
import pytest

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from gpu_util import develop, download_image

pytestmark = pytest.mark.gpu

SIZES = [(12, 12), (14, 30), (62, 34), (64, 32), (66, 30), (130, 62), (518, 262)]


@pytest.fixture(scope="module")
def ctx():
    c = L.Context(0)
    yield c
    L.debug_force_denoise_shape(-1)
    L.debug_denoise_tma(True)
    c.close()


def sequence(ctx, w, h, shape, temporal, tma=True):
    L.debug_force_denoise_shape(L.DN_SHAPES.index(shape))
    L.debug_denoise_tma(tma)
    flags = L.FLAG_DENOISE | L.FLAG_KEEP_INTERMEDIATE | (L.FLAG_TEMPORAL_DENOISE if temporal else 0)
    pp = L.pipeline_params(w, h, debayer=L.DEBAYER_BILINEAR, out_space=L.CS_BT709, out_format=L.FORMAT_RGBA32F,
                           flags=flags)
    fp = L.frame_params(W.make_profile(), denoise_strength=1.2, denoise_temporal_strength=0.8 if temporal else 0.0,
                        noise_override=W.noise_model(4.0, 40.0))
    out = []
    with L.Pipeline(ctx, pp) as pipe:
        for f in range(3):
            m = W.synth_frame(w, h, 19 * w + h, frame=f, rects=16, noise_a_dn=4.0, noise_b_dn=40.0,
                              movers=[(3.0, 0.5)])
            out.append(develop(pipe, m, fp))
            out.append(download_image(pipe.intermediate()[1], "r16"))
            if temporal:
                level, var = pipe.temporal_state()
                out += [download_image(level, "r32f"), download_image(var, "r8")]
        assert pipe.kernel_errors() == 0
    L.debug_force_denoise_shape(-1)
    L.debug_denoise_tma(True)
    return out


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("temporal", [False, True])
def test_packed_shapes_agree(ctx, w, h, temporal):
    a = sequence(ctx, w, h, "2x8 f32x2", temporal)
    for b in (sequence(ctx, w, h, "2x4 f32x2", temporal), sequence(ctx, w, h, "2x8 f32x2", temporal, tma=False)):
        assert len(a) == len(b)
        for x, y in zip(a, b):
            assert np.array_equal(np.ascontiguousarray(x).view(np.uint8), np.ascontiguousarray(y).view(np.uint8))
