"""GPU: a pipeline that finds no memory for its averaged planes, and a server
stream whose budget does not hold them, do without: the frames are the same
bit for bit."""
import numpy as np
import pytest
import torch

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from gpu_util import develop

pytestmark = pytest.mark.gpu

W2, H2 = 518, 262


@pytest.fixture(scope="module")
def ctx():
    c = L.Context(0)
    L.debug_force_denoise_shape(L.DN_SHAPES.index("2x8 f32x2"))
    yield c
    L.debug_force_denoise_shape(-1)
    L.debug_fail_alloc(0)
    c.close()


def params():
    return L.pipeline_params(W2, H2, debayer=L.DEBAYER_BILINEAR, out_space=L.CS_BT709, out_format=L.FORMAT_RGBA32F,
                             flags=L.FLAG_DENOISE | L.FLAG_TEMPORAL_DENOISE)


def frame_params():
    return L.frame_params(W.make_profile(), denoise_strength=1.0, denoise_temporal_strength=0.8,
                          noise_override=W.noise_model(4.0, 40.0))


def mosaics():
    return [W.synth_frame(W2, H2, 7, frame=f, rects=16, noise_a_dn=4.0, noise_b_dn=40.0, movers=[(3.0, 0.5)])
            for f in range(3)]


def clip(pipe):
    return [develop(pipe, m, frame_params()) for m in mosaics()]


def test_allocation_of_the_planes_fails(ctx):
    with L.Pipeline(ctx, params()) as pipe:
        want = clip(pipe)
    for k in range(1, 20):
        L.debug_fail_alloc(k)
        try:
            pipe = L.Pipeline(ctx, params())
        except L.CrawError as e:
            assert e.errno == 12
            continue
        break
    L.debug_fail_alloc(0)
    assert 5 < k < 12          # the allocations a frame cannot do without failed the creation
    with pipe:
        for a, b in zip(want, clip(pipe)):
            assert np.array_equal(a, b)


def test_stream_in_a_budget_without_planes(ctx):
    fp = frame_params()        # the server reads its profile as frames start

    def serve(srv):
        sid = srv.open(L.server_stream_params(params()))
        size = srv.stats().hbm_resident
        src = [torch.from_numpy(m.view(np.int16)).pin_memory() for m in mosaics()]
        dst = [torch.empty((H2, W2, 4)).pin_memory() for _ in src]
        for i, (s, d) in enumerate(zip(src, dst)):
            srv.submit(sid, s.data_ptr(), W2 * 2, d.data_ptr(), W2 * 16, fp, user=i)
        srv.drain()
        done = [r.status for r in srv.poll(8)]
        assert done == [0] * len(src)
        return size, [d.numpy().copy() for d in dst]

    with L.Server(ctx, L.server_params(hbm_budget=1 << 40)) as srv:
        size, want = serve(srv)
    with L.Server(ctx, L.server_params(hbm_budget=size - 1)) as srv:
        less, got = serve(srv)
    assert less < size
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
