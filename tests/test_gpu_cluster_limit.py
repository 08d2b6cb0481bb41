"""Cluster sizes of the ACA path.  The first ACA assembly of a process asks how large its clusters can be; the
query must not take away the error of a launch before it.  Smaller clusters give the same factor."""
import os
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


FACTOR = """
import sys
sys.path.insert(0, "kernelmatrices.jl_gb300")
import numpy as np
import kmhodlr as K
from kmhodlr.data import uniform_points
for n, lv, rank in ((3001, 1, 33), (3100, 3, 40), (13000, 4, 24)):  # top panels of 1500, 1550 and 6500 rows
    pts = uniform_points(n, 3)
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, np.array([1.0, 0.02 if n < 10000 else 0.005, 1.0]), K.Matern32()), 1e-13, rank, K.FixedLevel(lv))
    x = np.random.default_rng(4).standard_normal((n, 3))
    y = hk @ x
    K.symmetricfactorize(hk)
    close = lambda a, b: np.linalg.norm(a - b) < 1e-10 * np.linalg.norm(b)
    assert close(hk @ x, y) and close(hk.ldiv(y), x), (n, lv)
    assert close(hk.W.ldiv(hk.W @ x), x) and close(hk.W.T.ldiv(hk.W.T @ x), x), (n, lv)
    print(hk.logdet().hex())
"""


def test_smaller_clusters_give_the_same_factor(lib):
    """Where clusters of 16 are refused, ACA runs in clusters of 8 and panels that no cluster holds go to the kernels
    of all SMs: the identities of test_gpu_aca_factor.py to its 1e-10, and logdet to 1e-12 of the points."""
    got = {}
    for cap in ("16", "8", "2", "1"):
        r = subprocess.run([sys.executable, "-c", FACTOR], cwd=ROOT, env=dict(os.environ, KM_CLUSTER_MAX=cap),
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, (cap, r.stderr)
        got[cap] = [float.fromhex(v) for v in r.stdout.split()]
    for cap in ("8", "2", "1"):
        assert all(abs(a - b) < 1e-12 * n for a, b, n in zip(got[cap], got["16"], (3001, 3100, 13000))), (cap, got)
