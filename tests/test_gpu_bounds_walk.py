"""GPU: the bounds-checked build over the cases of bounds_walk_cases.py, in a
process of its own: no error bit set, and the product build's outputs bit for
bit."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import libcraw_gb300 as L

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent
BOUNDS = Path(L.__file__).resolve().parent / "_lib" / "libcraw_bounds.so"


def test_bounds_build_is_clean_and_equal(tmp_path):
    sys.path.insert(0, str(HERE))
    import bounds_walk_cases
    mine = bounds_walk_cases.run_cases()
    out = tmp_path / "bounds.npz"
    r = subprocess.run([sys.executable, str(HERE / "bounds_walk_cases.py"), str(out)],
                       env=dict(os.environ, CRAW_LIBRARY=str(BOUNDS)), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    theirs = dict(np.load(out))
    assert set(theirs) == set(mine)
    for key in sorted(mine):
        if key.endswith("/errors"):
            assert int(theirs[key][0]) == 0 and int(mine[key][0]) == 0, key
        else:
            assert np.array_equal(mine[key].view(np.uint8), theirs[key].view(np.uint8)), key
