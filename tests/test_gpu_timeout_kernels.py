"""Which kernel's bounded wait ran out (km_set_wait_limit(h, 0): every such wait gives up at its first poll).

The leaf QR comes before the nodes and gives up too, so the message names both where both did; a float-pair
root whose children are leaves has no wait in front of its Cholesky factor, so that only the leaves do.
Every form: FP64 and float pairs, one CTA a node and clusters.  The handle recovers."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent
LEAF = "a bounded wait of the leaf kernels ran out"
NODE = "a bounded wait inside the node factorisation ran out"

SCRIPT = """
import sys, json, ctypes as C
sys.path.insert(0, "kernelmatrices.jl_gb300")
import numpy as np
import kmhodlr
from kmhodlr import _lib as L, hodlr as KH
from kmhodlr.data import uniform_points
lib = kmhodlr.load()
out = []
for prec in (L.KM_PREC_FP64, L.KM_PREC_MIXED):
    for n, lv, r in ((4096, 4, 72), (1000, 2, 33), (600, 1, 40)):
        h = C.c_void_p()
        cfg = L.KmConfig(device=0, precision=prec, hbm_budget_fraction=0.8, refine_max_iter=0, refine_tol=0.0)
        assert lib.km_create(C.byref(cfg), C.byref(h)) == L.KM_OK
        pts, p = uniform_points(n, 31), np.array([1.0, 0.1, 1e-2])
        assemble = lambda: lib.km_assemble(h, KH._dp(pts), n, L.KM_KERNEL_MATERN32, KH._dp(p), 3, L.KM_METHOD_NYSTROM,
                                           0.0, r, L.KM_LEVEL_FIXED, lv)
        assert assemble() == L.KM_OK and lib.km_set_wait_limit(h, 0) == L.KM_OK
        assert lib.km_factorize(h) == L.KM_ERR_TIMEOUT
        out.append([prec == L.KM_PREC_MIXED, lv, lib.km_last_error(h).decode()])
        assert lib.km_set_wait_limit(h, -1) == L.KM_OK
        assert assemble() == L.KM_OK and lib.km_factorize(h) == L.KM_OK, lib.km_last_error(h)
        lib.km_destroy(h)
print(json.dumps(out))
"""


@pytest.mark.parametrize("cap", ["1", "2", "8"])
def test_message_names_the_kernels(lib, cap):
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, env=dict(os.environ, KM_NODE_CLUSTER=cap),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    got = json.loads(r.stdout.strip().splitlines()[-1])
    assert len(got) == 6
    for mixed, lv, message in got:
        leaves_only = mixed and lv == 1
        assert message == (LEAF if leaves_only else f"{LEAF}; {NODE}"), (mixed, lv, message)
