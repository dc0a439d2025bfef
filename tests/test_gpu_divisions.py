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
    for f in ("check_reciprocal", "check_gamut_quotient", "check_gamut_compress", "check_clip_ramp", "check_noise_lut"):
        getattr(lib, f).restype = C.c_longlong
    return lib


def bits(x):
    return int(np.array(x, np.float32).view(np.uint32))


# The three channels of the reference gamut compression (lib/gamut.c:11-25).
THR, LIM, PWR = np.array([0.815, 0.803, 0.880]), np.array([1.147, 1.264, 1.312]), 1.2
SCL = (LIM - THR) / (((1.0 - THR) / (LIM - THR)) ** -PWR - 1.0) ** (1.0 / PWR)


def test_reciprocal(lib):
    """Every float above 2^-128 and below 1.34e38."""
    assert lib.check_reciprocal(C.c_uint32(bits(2.0 ** -128) + 1), C.c_uint32(bits(1.34e38))) == 0


@pytest.mark.parametrize("scl", SCL)
def test_gamut_quotient(lib, scl):
    assert lib.check_gamut_quotient(C.c_float(scl)) == 0


def test_gamut_compress(lib):
    """Pixels of every positive float up to 1e37 (those whose reciprocals are
    infinite among them), with zeros, infinities and NaN beside it."""
    thr, scl = THR.astype(np.float32), SCL.astype(np.float32)
    fp = C.POINTER(C.c_float)
    assert lib.check_gamut_compress(C.c_uint32(1), C.c_uint32(bits(1e37)), thr.ctypes.data_as(fp),
                                    scl.ctypes.data_as(fp), C.c_float(PWR)) == 0


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
