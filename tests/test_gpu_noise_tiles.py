"""GPU: the noise estimate where its kernels can go wrong: planes that end
one position past a tile or a strip, or inside a group of four; numbers of
bins on either side of the kept index's width and of the counters' windows;
frames whose high-pass is zero or whose means lie near zero. The bins hold
the reference's counts and medians exactly and their levels to the last
bits, so the fit agrees with the oracle's to 1e-6 relative."""
import numpy as np
import pytest

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from oracle import Oracle

pytestmark = pytest.mark.gpu
orc = Oracle()
PROF = W.make_profile()


def frame(kind, w, h, seed):
    if kind == "ramp":
        return W.noise_ramp(w, h, seed, lo=0.0)
    rng = np.random.default_rng(seed)
    black = 256
    if kind == "dark":          # means from below zero to a few 1e-3
        u = 16.0 * np.clip(np.arange(w)[None, :] / w - 0.2, 0, 1) + np.zeros((h, 1))
        return np.clip(black + u + rng.normal(0.0, 1.0, (h, w)) * np.sqrt(9 + 2 * u), 0, 65535).astype(np.uint16)
    if kind == "steps":         # flat steps, noise on every other one: half the high-pass zeros
        m = black + 40 + 240 * (np.arange(w)[None, :] // 64) + np.zeros((h, 1))
        n = rng.normal(0.0, 1.0, (h, w)) * 0.4 * np.sqrt(m - black) * ((np.arange(w)[None, :] // 32) & 1)
        return np.clip(m + n, 0, 65535).astype(np.uint16)
    assert kind == "loud"       # |high-pass| beyond every window, at steady means
    m = 1300 + 1700 * (np.arange(w)[None, :] / w) + np.zeros((h, 1))
    sign = 1 - 2.0 * ((np.arange(w)[None, :] // 2 + np.arange(h)[:, None] // 2) & 1)
    return np.clip(m + sign * np.sqrt(m) * (14 + rng.normal(0.0, 1.0, (h, w))), 0, 65535).astype(np.uint16)


@pytest.mark.parametrize("w,h,kind,nb,least", [
    (32, 32, "ramp", 8, 1), (34, 50, "ramp", 8, 1),
    (272, 80, "ramp", 64, 20), (274, 82, "ramp", 128, 20), (276, 84, "ramp", 129, 20),
    (256, 144, "ramp", 255, 10), (258, 146, "ramp", 256, 10), (262, 142, "ramp", 257, 10),
    (530, 278, "ramp", 512, 10),
    (394, 210, "dark", 300, 20), (394, 210, "dark", 512, 50),
    (770, 130, "steps", 64, 50), (1026, 258, "loud", 48, 50), (1026, 258, "loud", 300, 20),
])
def test_estimate_matches_oracle(w, h, kind, nb, least):
    m = frame(kind, w, h, 7 * w + h)
    p = L.NoiseEstimateParams()
    p.nb_bins, p.min_bin_samples, p.max_level = nb, least, 0.98
    ret, want = orc.noise_estimate(m, PROF, p)
    if ret < 0:
        with pytest.raises(L.CrawError) as e:
            L.noise_estimate(m, PROF, p)
        assert e.value.code == ret
        return
    g, r = L.noise_estimate(m, PROF, p).as_tuple(), want.as_tuple()
    assert (g[2], g[3]) == (r[2], r[3]), (g, r)
    assert all(abs(x - y) <= 1e-6 * max(abs(y), 1e-30) for x, y in zip(g[:2] + g[4:], r[:2] + r[4:])), (g, r)


@pytest.mark.parametrize("nb,least", [(54, 10), (55, 10), (56, 10)])
def test_few_and_many_bins(nb, least):
    """Numbers of used bins on either side of where the pairs' costs are
    first bounded in floats."""
    m = frame("ramp", 516, 260, 77)
    p = L.NoiseEstimateParams()
    p.nb_bins, p.min_bin_samples, p.max_level = nb, least, 0.98
    ret, want = orc.noise_estimate(m, PROF, p)
    assert ret == 0 and 46 <= want.as_tuple()[2] <= 50, want.as_tuple()
    g, r = L.noise_estimate(m, PROF, p).as_tuple(), want.as_tuple()
    assert (g[2], g[3]) == (r[2], r[3]), (g, r)
    assert all(abs(x - y) <= 1e-6 * max(abs(y), 1e-30) for x, y in zip(g[:2] + g[4:], r[:2] + r[4:])), (g, r)
