"""A pipeline's optional planes on failing calls (tests/native/planes_check.c):
only a lack of memory makes a pipeline go without them; another error is
returned, nothing stays allocated, and an error that is not the allocation's
stays the caller's to read."""
import ctypes as C
import errno
import subprocess
from pathlib import Path

import pytest

from libcraw_gb300.build import HOST_CFLAGS

SRC = Path(__file__).resolve().parent / "native" / "planes_check.c"
OOM, OTHER = 2, 1                  # cudaErrorMemoryAllocation, cudaErrorInvalidValue


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = tmp_path_factory.mktemp("planes") / "planes_check.so"
    subprocess.run(["gcc", *HOST_CFLAGS, "-w", "-shared", "-Wl,-z,lazy", str(SRC), "-o", str(so)], check=True)
    f = C.CDLL(str(so), mode=0x1).planes_check       # RTLD_LAZY

    def run(alloc, sync, error):
        out = (C.c_int * 4)()
        f(alloc, sync, error, out)
        return tuple(out)
    return run


@pytest.mark.parametrize("alloc,sync,error,want", [
    (0, 0, 0, (0, 1, 1, 0)),
    (-errno.ENOMEM, 0, OOM, (0, 0, 0, 0)),
    (-errno.ENOMEM, 0, OTHER, (0, 0, 0, OTHER)),
    (-errno.EIO, 0, OTHER, (-errno.EIO, 0, 0, OTHER)),
    (0, -errno.EIO, OTHER, (-errno.EIO, 0, 0, OTHER)),
])
def test_planes(check, alloc, sync, error, want):
    assert check(alloc, sync, error) == want
