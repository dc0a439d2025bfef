"""GPU: a pipeline's AWB slots over more frames than slots: each frame's
histogram is its own (the device's is back at zeros after each frame), for
every number of slots, with frames of one colour (every block in one bin,
the most contended) among them."""
import numpy as np
import pytest
import torch

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from gpu_util import alloc_rgba, download_image, upload_mosaic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots", [1, 2, 4])
@pytest.mark.parametrize("deb,w,h", [(L.DEBAYER_MHC, 246, 134), (L.DEBAYER_RCD, 330, 118)])
def test_histogram_of_each_frame(slots, deb, w, h):
    frames = [W.synth_frame(w, h, 31 + i, rects=16, noise_a_dn=4.0, noise_b_dn=40.0) for i in range(3)]
    flat = np.full((h, w), 1200, np.uint16)
    order = [frames[0], flat, frames[1], flat, frames[2], frames[0]]
    pp = L.pipeline_params(w, h, debayer=deb, out_space=L.CS_BT709, out_format=L.FORMAT_RGBA32F,
                           nb_awb_slots=slots, flags=L.FLAG_AWB_HISTOGRAM | L.FLAG_KEEP_INTERMEDIATE)
    fp = L.frame_params(W.make_profile())
    want = []
    with L.Context(0) as ctx, L.Pipeline(ctx, pp) as pipe:
        out, dst = alloc_rgba(w, h)
        for m in order:
            _, src = upload_mosaic(m)
            pipe.record(torch.cuda.current_stream().cuda_stream, src, dst, fp)
            torch.cuda.synchronize()
            want.append(L.awb_histogram_from_rgb(download_image(pipe.intermediate()[0], "rgba32f"), W.WB))
            for back in range(min(slots, len(want))):
                got = pipe.awb_histogram(back)
                cnt, wgt, brt = want[-1 - back]
                assert np.array_equal(got.count, cnt), (len(want), back)
                assert np.array_equal(got.weight, wgt) and np.array_equal(got.weight_bright, brt)
        assert pipe.kernel_errors() == 0
