"""GPU: kernels launched before their predecessors on the stream have ended:
a clip's frames (denoise with history, develop, AWB), a frame through the
highlights, the exact rounding and the chroma denoise, recorded back to back
into the same buffers without a wait between, and the same captured into a
graph and replayed, against each recorded by itself."""
import numpy as np
import pytest
import torch

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from gpu_util import alloc_rgba, upload_mosaic

pytestmark = pytest.mark.gpu

W2, H2 = 1030, 410
CASES = {
    "clip": (L.DEBAYER_RCD, L.FLAG_DENOISE | L.FLAG_TEMPORAL_DENOISE, dict(denoise_temporal_strength=0.7), 0),
    "exact": (L.DEBAYER_RCD, L.FLAG_DENOISE, {}, 0),
    "exact_linear": (L.DEBAYER_MHC, L.FLAG_DENOISE, {}, 0),
    "chroma": (L.DEBAYER_MHC, L.FLAG_DENOISE | L.FLAG_CHROMA_DENOISE, dict(denoise_chroma_strength=0.6), 0),
    "highlights": (L.DEBAYER_RCD, L.FLAG_DENOISE | L.FLAG_HIGHLIGHT_RECONSTRUCTION, {},
                   L.FRAME_HIGHLIGHT_RECONSTRUCTION),
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("graph", [False, True])
def test_back_to_back(name, graph):
    deb, flags, kw, fflags = CASES[name]
    prof = W.make_profile()
    ms = [W.highlight_frame(W2, H2, 5 + i) for i in range(4)]
    srcs = [upload_mosaic(m) for m in ms]
    pp = L.pipeline_params(W2, H2, debayer=deb, out_space=L.CS_BT2020, out_format=L.FORMAT_RGBA32F, nb_awb_slots=4,
                           flags=flags | L.FLAG_AWB_HISTOGRAM)
    fp = L.frame_params(prof, denoise_strength=1.0, noise_override=W.noise_model(4, 40), flags=fflags, **kw)

    def frames(pipe, stream, outs, wait):
        for (_, src), (_, dst) in zip(srcs, outs):
            pipe.record(stream.cuda_stream, src, dst, fp)
            if wait:
                torch.cuda.synchronize()

    def results(pipe, outs):
        torch.cuda.synchronize()
        hist = [pipe.awb_histogram(3 - i) for i in range(4)]
        return [o.cpu().numpy() for o, _ in outs], [(h.count, h.weight, h.weight_bright) for h in hist]

    with L.Context(0) as ctx:
        outs = [alloc_rgba(W2, H2) for _ in ms]
        with L.Pipeline(ctx, pp) as pipe:
            frames(pipe, torch.cuda.current_stream(), outs, True)
            want, hist = results(pipe, outs)
        outs = [alloc_rgba(W2, H2) for _ in ms]
        s = torch.cuda.Stream()
        with L.Pipeline(ctx, pp) as pipe, torch.cuda.stream(s):
            if graph:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=s):
                    frames(pipe, s, outs, False)
                g.replay()
            else:
                frames(pipe, s, outs, False)
            got, got_hist = results(pipe, outs)
            assert pipe.kernel_errors() == 0
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
    for a, b in zip(hist, got_hist):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
