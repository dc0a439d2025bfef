"""GPU: noise estimates whose used bins lie on either side of where the pairs'
costs are first bounded in floats (40), against the oracle."""
import pytest

import libcraw_gb300 as L
import test_gpu_noise_tiles as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,used", [(45, 39), (46, 40), (47, 41), (48, 42)])
def test_few_and_many_bins(nb, used):
    m = T.frame("ramp", 516, 260, 77)
    p = L.NoiseEstimateParams()
    p.nb_bins, p.min_bin_samples, p.max_level = nb, 10, 0.98
    ret, want = T.orc.noise_estimate(m, T.PROF, p)
    g, r = L.noise_estimate(m, T.PROF, p).as_tuple(), want.as_tuple()
    assert ret == 0 and r[2] == used
    assert (g[2], g[3]) == (r[2], r[3]), (g, r)
    assert all(abs(x - y) <= 1e-6 * max(abs(y), 1e-30) for x, y in zip(g[:2] + g[4:], r[:2] + r[4:])), (g, r)
