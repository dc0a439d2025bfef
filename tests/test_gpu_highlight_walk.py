"""GPU: the highlight reconstruction's walking warps where a strip or a
segment ends: planes one quad past 28 texels or 30 quads, an odd number of
quads, two rows of segments, mostly clipped and hardly clipped frames. Held
to the oracle by half-float steps, as tests/test_gpu_highlight.py explains."""
import pytest

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from test_gpu_highlight import MG, close_in_half_steps, orc, run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = L.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("w,h", [(58, 18), (60, 34), (62, 36), (110, 38), (112, 50), (114, 34), (122, 14), (226, 130),
                                 (2050, 258)])
@pytest.mark.parametrize("gain", [0.9, 2.5])
def test_rebuilt_mosaic_vs_oracle(ctx, w, h, gain):
    prof = MG.golden_profile()
    m = W.highlight_frame(w, h, 3 * w + h, gain=gain)
    _, rebuilt, _, _ = run(ctx, m, prof, deb=L.DEBAYER_BILINEAR)
    ok, st = close_in_half_steps(rebuilt, orc.highlights(m, prof, (2.0, 1.0, 1.5), "f32"))
    assert ok, st
