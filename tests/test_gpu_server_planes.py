"""GPU: streams with a temporal history, whose pipelines hold averaged planes
that they can do without, in a budget that fits them only without: each is
admitted, idle or with frames in flight, and their frames are the same bit
for bit; one that fits neither way is refused and costs the others nothing."""
import numpy as np
import pytest
import torch

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W

pytestmark = pytest.mark.gpu

W2, H2, N = 1030, 518, 6


@pytest.fixture(scope="module")
def ctx():
    c = L.Context(0)
    L.debug_force_denoise_shape(L.DN_SHAPES.index("2x8 f32x2"))
    yield c
    L.debug_force_denoise_shape(-1)
    c.close()


def stream_params():
    return L.server_stream_params(L.pipeline_params(
        W2, H2, debayer=L.DEBAYER_BILINEAR, out_space=L.CS_BT709, out_format=L.FORMAT_RGBA32F,
        flags=L.FLAG_DENOISE | L.FLAG_TEMPORAL_DENOISE))


class Clip:
    """A stream's frames and where they go."""

    def __init__(self):
        self.fp = L.frame_params(W.make_profile(), denoise_strength=1.0, denoise_temporal_strength=0.8,
                                 noise_override=W.noise_model(4.0, 40.0))
        self.src = [torch.from_numpy(W.synth_frame(W2, H2, 7, frame=f, rects=16, noise_a_dn=4.0, noise_b_dn=40.0,
                                                   movers=[(3.0, 0.5)]).view(np.int16)).pin_memory() for f in range(N)]
        self.dst = [torch.empty((H2, W2, 4)).pin_memory() for _ in self.src]

    def submit(self, srv, sid, frames):
        for f in frames:
            srv.submit(sid, self.src[f].data_ptr(), W2 * 2, self.dst[f].data_ptr(), W2 * 16, self.fp, user=f)

    def frames(self):
        return [d.numpy() for d in self.dst]


@pytest.fixture(scope="module")
def known(ctx):
    """A stream's bytes with the planes and without, and its frames."""
    clip = Clip()
    with L.Server(ctx, L.server_params(hbm_budget=1 << 40)) as srv:
        sid = srv.open(stream_params())
        size = srv.stats().hbm_resident
        clip.submit(srv, sid, range(N))
        srv.drain()
        assert [r.status for r in srv.poll(2 * N)] == [0] * N
    with L.Server(ctx, L.server_params(hbm_budget=size - 1)) as srv:
        srv.open(stream_params())
        less = srv.stats().hbm_resident
    assert less < size
    return size, less, clip.frames()


@pytest.mark.parametrize("busy", [False, True])
@pytest.mark.parametrize("streams", [2, 3])
def test_streams_that_fit_without_planes(ctx, known, streams, busy):
    size, less, want = known
    clips = [Clip() for _ in range(streams)]
    with L.Server(ctx, L.server_params(hbm_budget=streams * less)) as srv:
        ids = []
        for c in clips:
            ids.append(srv.open(stream_params()))
            if busy:
                c.submit(srv, ids[-1], range(N // 2))
        st = srv.stats()
        assert st.hbm_resident <= st.hbm_budget
        for c, sid in zip(clips, ids):
            c.submit(srv, sid, range(N // 2 if busy else 0, N))
        srv.drain()
        assert [r.status for r in srv.poll(streams * N)] == [0] * (streams * N)
    for c in clips:
        for a, b in zip(want, c.frames()):
            assert np.array_equal(a, b)


def test_refused_stream_costs_nothing(ctx, known):
    size, less, _ = known
    room = (size - less) // 4          # what the planes give back does not reach
    with L.Server(ctx, L.server_params(hbm_budget=size + room)) as srv:
        srv.open(stream_params())
        before = srv.stats().hbm_resident
        with pytest.raises(L.CrawError) as e:
            srv.open(stream_params())
        assert e.value.errno == 11     # EAGAIN
        assert srv.stats().hbm_resident == before == size
