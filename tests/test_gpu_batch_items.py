"""GPU: a batch's items where their layout branches, against the frames one
by one, bit for bit: RCD frames that are all border, with interiors of one
tile and of several strips and segments, one or many in a batch (the two
denoise shapes, on either side of two tiles an SM), every output layout,
fused and not, denoised and not in one batch."""
import numpy as np
import pytest
import torch

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from gpu_util import alloc_rgba, develop, upload_mosaic

pytestmark = pytest.mark.gpu

SIZES = [(12, 12), (132, 12), (70, 40), (134, 38), (196, 54), (262, 52), (410, 230), (1030, 150), (640, 360)]


@pytest.fixture(scope="module")
def ctx():
    c = L.Context(0)
    # The batch's search is the packed one: so is the frames' one by one.
    L.debug_force_denoise_shape(2)
    yield c
    L.debug_force_denoise_shape(-1)
    c.close()


@pytest.mark.parametrize("sizes", [SIZES[2:3], SIZES[6:7], SIZES, SIZES + SIZES[::-1] + SIZES[5:]])
@pytest.mark.parametrize("fmt", [L.FORMAT_RGBA32F, L.FORMAT_RGB32F, L.FORMAT_RGBA16F])
@pytest.mark.parametrize("flags", [L.BATCH_FLAG_UNFUSED, L.BATCH_FLAG_FUSED])
def test_rcd_batch_bits(ctx, sizes, fmt, flags):
    prof = W.make_profile()
    space = L.CS_ACES_AP1 if fmt == L.FORMAT_RGBA16F else L.CS_BT2020
    ms = [W.synth_frame(w, h, 11 * i + w, rects=24, noise_a_dn=4.0, noise_b_dn=40.0) for i, (w, h) in enumerate(sizes)]
    fps = [L.frame_params(prof, denoise_strength=0.0 if i % 4 == 1 else 1.0, noise_override=W.noise_model(4, 40))
           for i in range(len(ms))]
    ups = [upload_mosaic(m) for m in ms]
    outs = [alloc_rgba(w, h, fmt) for w, h in sizes]
    bp = L.batch_params(1030, 360, max_frames=len(ms), debayer=L.DEBAYER_RCD, out_space=space, out_format=fmt,
                        flags=L.FLAG_DENOISE | flags)
    with L.Batch(ctx, bp) as b:
        b.record(torch.cuda.current_stream().cuda_stream, [u[1] for u in ups], [o[1] for o in outs], fps)
        torch.cuda.synchronize()
        tiles = sum(-(-w // 64) * -(-h // 32) for i, (w, h) in enumerate(sizes) if i % 4 != 1)
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        assert b.info()["denoise_shape"] == (1 if tiles > 2 * sms else 0)
    for (w, h), m, fp, (t, _) in zip(sizes, ms, fps, outs):
        pp = L.pipeline_params(w, h, debayer=L.DEBAYER_RCD, out_space=space, out_format=fmt, flags=L.FLAG_DENOISE)
        with L.Pipeline(ctx, pp) as pipe:
            want = develop(pipe, m, fp, fmt)
        assert np.array_equal(t.float().cpu().numpy(), want), (w, h)
