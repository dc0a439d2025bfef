"""GPU: device arithmetic that stands in for a division gives the division's
own rounding (tests/native/device_checks.cu, compiled with the kernels'
sources): no input differs in any bit."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from libcraw_gb300.build import NVCC, NVCC_FLAGS

pytestmark = pytest.mark.gpu

SRC = Path(__file__).resolve().parent / "native" / "device_checks.cu"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("checks") / "device_checks.so"
    subprocess.run([NVCC, *NVCC_FLAGS, "-fmad=false", "-shared", "-cudart", "static", str(SRC), "-o", str(so)],
                   check=True)
    lib = C.CDLL(str(so))
    for f in ("check_gamut_quotient", "check_clip_ramp", "check_noise_lut"):
        getattr(lib, f).restype = C.c_longlong
    return lib


# The three channels' scales of the reference gamut compression (lib/gamut.c:11-25).
@pytest.mark.parametrize("lim,thr", [(1.147, 0.815), (1.264, 0.803), (1.312, 0.880)])
def test_gamut_quotient(lib, lim, thr):
    r = ((1.0 - thr) / (lim - thr)) ** -1.2 - 1.0
    assert lib.check_gamut_quotient(C.c_float((lim - thr) / r ** (1.0 / 1.2))) == 0


def test_clip_ramp(lib):
    assert lib.check_clip_ramp() == 0


@pytest.mark.parametrize("seed", range(4))
def test_noise_lut(lib, seed):
    rng = np.random.default_rng(seed)
    black = rng.uniform(0.0, 0.1, 4).astype(np.float32)
    white = (black + rng.uniform(0.02, 1.0, 4)).astype(np.float32)
    if seed == 0:      # 12 bits with a black level, 16 bits without
        black = np.array([256, 256, 256, 0], np.float32) / np.float32(65535)
        white = np.array([4095, 4095, 65535, 65535], np.float32) / np.float32(65535)
    fp = C.POINTER(C.c_float)
    assert lib.check_noise_lut(black.ctypes.data_as(fp), white.ctypes.data_as(fp)) == 0
