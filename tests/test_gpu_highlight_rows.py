"""GPU: the highlight reconstruction where its segments go over from 2 quad rows
to 4 and from 4 to 8 (21280 warps of either), and in frames of a few rows, with
heights that leave a segment short. Held to the oracle by half-float steps, as
tests/test_gpu_highlight.py explains."""
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


# Strips of 30 quads, so 50 across 3000 pixels: 425 segments of 2 rows are 21250
# warps; 80 across 4800: 266 of 4 are 21280.
@pytest.mark.parametrize("w,h", [(8, 8), (34, 10), (66, 12), (62, 22), (3000, 1700), (3000, 1702), (4800, 2128),
                                 (4800, 2130)])
def test_rebuilt_mosaic_vs_oracle(ctx, w, h):
    prof = MG.golden_profile()
    m = W.highlight_frame(w, h, 3 * w + h, gain=1.5)
    _, rebuilt, _, _ = run(ctx, m, prof, deb=L.DEBAYER_BILINEAR)
    ok, st = close_in_half_steps(rebuilt, orc.highlights(m, prof, (2.0, 1.0, 1.5), "f32"))
    assert ok, st
