"""GPU: the RCD's border by walking warps against the per-pixel tiles, bit
for bit: frames that are all border, down to the smallest; interiors of one
tile; borders of a few pixels and of nearly two tiles on the right and below;
widths and heights that leave parts of AWB and chroma blocks; a kept
intermediate, FP16 storage, the chroma path and the histogram."""
import numpy as np
import pytest

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from gpu_util import develop, download_image

pytestmark = pytest.mark.gpu

SIZES = [(12, 12), (14, 64), (132, 12), (70, 40), (134, 38), (134, 54), (196, 38), (202, 70), (262, 52), (410, 230),
         (1030, 86)]


@pytest.fixture(scope="module")
def ctx():
    c = L.Context(0)
    yield c
    L.debug_rcd_strips(1)
    c.close()


def both(ctx, pp, run):
    out = []
    for mode in (0, 1):
        L.debug_rcd_strips(mode)
        with L.Pipeline(ctx, pp) as pipe:
            r = run(pipe)
            out.append((r, pipe.awb_histogram()))
            assert pipe.kernel_errors() == 0
    L.debug_rcd_strips(1)
    (a, ha), (b, hb) = out
    for x, y in zip(a, b):
        bad = np.argwhere((x.view(np.uint8) != y.view(np.uint8)).reshape(x.shape[0], x.shape[1], -1).any(-1))
        assert not len(bad), (len(bad), bad[:8].tolist(), bad[-4:].tolist())
    assert np.array_equal(ha.count, hb.count) and np.array_equal(ha.weight, hb.weight) and \
        np.array_equal(ha.weight_bright, hb.weight_bright)


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("keep,storage", [(False, L.STORAGE_FP32), (True, L.STORAGE_FP32), (True, L.STORAGE_FP16)])
def test_border_bits(ctx, w, h, keep, storage):
    m = W.synth_frame(w, h, 5 * w + h, rects=24, noise_a_dn=4.0, noise_b_dn=40.0)
    pp = L.pipeline_params(w, h, debayer=L.DEBAYER_RCD, out_space=L.CS_ACES_AP1 if h % 4 else L.CS_BT2020,
                           out_format=L.FORMAT_RGBA32F, storage=storage,
                           flags=L.FLAG_AWB_HISTOGRAM | (L.FLAG_KEEP_INTERMEDIATE if keep else 0))
    fp = L.frame_params(W.make_profile())

    def run(pipe):
        out = [develop(pipe, m, fp)]
        if keep:
            out.append(download_image(pipe.intermediate()[0], "rgba16f" if storage == L.STORAGE_FP16 else "rgba32f"))
        return out
    both(ctx, pp, run)


@pytest.mark.parametrize("w,h", [s for s in SIZES if min(s) >= 38])
@pytest.mark.parametrize("storage", [L.STORAGE_FP32, L.STORAGE_FP16])
def test_border_chroma(ctx, w, h, storage):
    """The block means, through the whole chroma denoise."""
    m = W.synth_frame(w, h, 5 * w + h, rects=24, noise_a_dn=4.0, noise_b_dn=40.0)
    pp = L.pipeline_params(w, h, debayer=L.DEBAYER_RCD, out_space=L.CS_BT2020, out_format=L.FORMAT_RGBA32F,
                           storage=storage, flags=L.FLAG_AWB_HISTOGRAM | L.FLAG_CHROMA_DENOISE)
    fp = L.frame_params(W.make_profile(), denoise_chroma_strength=0.7)
    both(ctx, pp, lambda pipe: [develop(pipe, m, fp)])
