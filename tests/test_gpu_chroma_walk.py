"""GPU: the chroma band's way back into the pixels by walking warps, at
widths where a lane, a quarter texel, an AWB block or a strip of 120 pixels
hangs over the edge and heights that end inside a quarter row: the kept
intermediate's histogram against the CPU builder, and every output layout,
from float and half storage, with and without it kept, against each other."""
import numpy as np
import pytest

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from gpu_util import develop, download_image

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = L.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("w,h", [(20, 20), (38, 22), (118, 26), (122, 34), (244, 62), (246, 70)])
@pytest.mark.parametrize("storage", [L.STORAGE_FP32, L.STORAGE_FP16])
def test_layouts_and_histogram(ctx, w, h, storage):
    m = W.synth_frame(w, h, 7 * w + h, rects=12, noise_a_dn=4.0, noise_b_dn=40.0)
    fp = L.frame_params(W.make_profile(), denoise_chroma_strength=0.8)
    out, hist = {}, []
    for fmt in (L.FORMAT_RGBA32F, L.FORMAT_RGB32F, L.FORMAT_RGBA16F):
        for keep in (0, L.FLAG_KEEP_INTERMEDIATE):
            pp = L.pipeline_params(w, h, debayer=L.DEBAYER_MHC, out_space=L.CS_ACES_AP1, out_format=fmt, storage=storage,
                                   flags=L.FLAG_AWB_HISTOGRAM | L.FLAG_CHROMA_DENOISE | keep)
            with L.Pipeline(ctx, pp) as pipe:
                out[fmt, keep] = develop(pipe, m, fp, fmt)
                hist.append(pipe.awb_histogram())
                if keep:
                    rgb = download_image(pipe.intermediate()[0], "rgba16f" if storage == L.STORAGE_FP16 else "rgba32f")
                assert pipe.kernel_errors() == 0
    cnt, wgt, brt = L.awb_histogram_from_rgb(rgb.astype(np.float32), W.WB)
    for g in hist:
        assert np.array_equal(g.count, cnt) and np.array_equal(g.weight, wgt) and np.array_equal(g.weight_bright, brt)
    full = out[L.FORMAT_RGBA32F, 0]
    for (fmt, _), o in out.items():
        want = full.astype(np.float16).astype(np.float32) if fmt == L.FORMAT_RGBA16F else full
        assert np.array_equal(o[..., :3], want[..., :3])
