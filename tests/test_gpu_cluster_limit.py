"""The first ACA assembly of a process asks how large its clusters can be; the query must not take away the
error of a launch before it."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

SCRIPT = """
import sys, ctypes as C
sys.path.insert(0, "kernelmatrices.jl_gb300")
import numpy as np
import kmhodlr
from kmhodlr import _lib as L, hodlr as KH
from kmhodlr.data import uniform_points
lib = kmhodlr.load()
refused = lib._ZN2km14launch_glogdetEPKNS_9GNodeDescEiPdP11CUstream_st  # km::launch_glogdet of no nodes
refused.restype, refused.argtypes = None, [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
h = C.c_void_p()
cfg = L.KmConfig(device=0, precision=L.KM_PREC_FP64, hbm_budget_fraction=0.8, refine_max_iter=0, refine_tol=0.0)
assert lib.km_create(C.byref(cfg), C.byref(h)) == L.KM_OK
n = 600
pts, p = uniform_points(n, 1), np.array([1.0, 0.1, 1.0])
assemble = lambda: lib.km_assemble(h, KH._dp(pts), n, L.KM_KERNEL_MATERN32, KH._dp(p), 3, L.KM_METHOD_ACA, 1e-6, 0,
                                   L.KM_LEVEL_FIXED, 2)
refused(None, 0, None, None)  # an empty grid, which the runtime refuses
assert assemble() == L.KM_ERR_CUDA, "the refused launch went unnoticed"
assert assemble() == L.KM_OK, lib.km_last_error(h)
"""


def test_query_keeps_an_earlier_error(lib):
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
