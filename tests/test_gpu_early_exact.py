"""GPU: frames with the exact rounding recorded back to back into the same
buffers without a wait between, and captured into a graph and replayed,
against each recorded by itself: the marking denoise, the kernels that settle
the marked codes in place, and the develop launched before the last of them
has ended. The statistics show that the rounding ran."""
import numpy as np
import pytest
import torch

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from gpu_util import alloc_rgba, upload_mosaic

pytestmark = pytest.mark.gpu

W2, H2, N = 1030, 410, 4


@pytest.fixture(autouse=True)
def _one_shape():
    """The marks are one denoise shape's: no timed choice between the two pipelines."""
    L.debug_force_denoise_shape(L.DN_SHAPES.index("2x8 f32x2"))
    yield
    L.debug_force_denoise_shape(-1)


@pytest.mark.parametrize("debayer", [L.DEBAYER_RCD, L.DEBAYER_MHC, L.DEBAYER_BILINEAR])
@pytest.mark.parametrize("graph", [False, True])
def test_back_to_back(debayer, graph):
    srcs = [upload_mosaic(W.highlight_frame(W2, H2, 5 + i)) for i in range(N)]
    pp = L.pipeline_params(W2, H2, debayer=debayer, out_space=L.CS_BT2020, out_format=L.FORMAT_RGBA32F, nb_awb_slots=N,
                           flags=L.FLAG_DENOISE | L.FLAG_EXACT_ROUNDING | L.FLAG_AWB_HISTOGRAM)
    fp = L.frame_params(W.make_profile(), denoise_strength=1.0, noise_override=W.noise_model(4, 40))

    def frames(pipe, stream, outs, wait):
        for (_, src), (_, dst) in zip(srcs, outs):
            pipe.record(stream.cuda_stream, src, dst, fp)
            if wait:
                torch.cuda.synchronize()

    def results(pipe, outs):
        torch.cuda.synchronize()
        hist = [pipe.awb_histogram(N - 1 - i) for i in range(N)]
        assert pipe.kernel_errors() == 0
        examined, changed, _, doubled = pipe.round_stats()
        return [o.cpu().numpy() for o, _ in outs], [(h.count, h.weight, h.weight_bright) for h in hist], \
            (examined, changed, doubled)

    with L.Context(0) as ctx:
        outs = [alloc_rgba(W2, H2) for _ in srcs]
        with L.Pipeline(ctx, pp) as pipe:
            frames(pipe, torch.cuda.current_stream(), outs, True)
            want, hist, settled = results(pipe, outs)
        outs = [alloc_rgba(W2, H2) for _ in srcs]
        s = torch.cuda.Stream()
        with L.Pipeline(ctx, pp) as pipe, torch.cuda.stream(s):
            if graph:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=s):
                    frames(pipe, s, outs, False)
                g.replay()
            else:
                frames(pipe, s, outs, False)
            got, got_hist, got_settled = results(pipe, outs)
    assert settled == got_settled and settled[0] > 0
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
    for a, b in zip(hist, got_hist):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
