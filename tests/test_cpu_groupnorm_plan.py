"""The host side of GroupNorm plans without dividing by the sample or row count (a child process: a division by zero would end it)."""
import subprocess
import sys

import pytest

from eridiffusion_b200.ops import _native as N

CODE = """
import ctypes, sys
lib = ctypes.CDLL(sys.argv[1])
lib.eri_gn_workspace.restype = ctypes.c_longlong
n, hw = int(sys.argv[2]), int(sys.argv[3])
assert lib.eri_gn_workspace(n, hw, 64, 8, 0) == 0 and lib.eri_gn_workspace(n, hw, 64, 8, 1) == 0
z, p = ctypes.c_int(0), ctypes.c_void_p(0)
assert lib.eri_gn_fwd(p, p, p, p, p, p, p, p, p, n, hw, 64, 8, ctypes.c_float(1e-5), 0, p) == -1
assert lib.eri_gn_bwd(p, p, p, p, p, p, p, p, p, p, p, p, p, p, n, hw, 64, 8, 0, 0, p) == -1
"""


@pytest.mark.parametrize("n,hw", [(0, 16), (2, 0), (0, 0)])
def test_no_samples_or_rows(n, hw):
    if not N._LIB_PATH.exists():
        pytest.skip("kernel library not built")
    r = subprocess.run([sys.executable, "-c", CODE, str(N._LIB_PATH), str(n), str(hw)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr)
