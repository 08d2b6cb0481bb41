"""Float-pair node factorisation (km_factor.cu): ranks around its panels of 4 columns, blocks of 8 rows
and chunks of 32 rows, on trees whose levels run with 1, 2, 4 and 8 CTAs a node.

Against the FP64 form, with the targets of the mixed form (test_gpu_mixed.py): logdet to 1e-6, solves to
1e-8 relative.  Cluster sizes: equal bits."""
import json
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("n,lv,r", [(900, 1, 2), (1000, 2, 3), (1100, 2, 7), (1100, 2, 31), (1101, 2, 33), (1300, 3, 64),
                                    (1303, 3, 66), (3000, 4, 79), (4000, 5, 80), (12345, 7, 37), (16000, 8, 40)])
def test_solve_and_logdet(lib, n, lv, r):
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    pts = uniform_points(n, 11)
    km = K.KernelMatrix(pts, pts, np.array([1.0, 0.1, 1e-2]), K.Matern32())
    b = np.random.default_rng(12).standard_normal((n, 2))
    h = [K.KernelHODLR(km, 0.0, r, K.FixedLevel(lv), nystrom=True, precision=p) for p in (K.KM_PREC_FP64, K.KM_PREC_MIXED)]
    for x in h:
        K.symmetricfactorize(x)
    want, got = (x.ldiv(b) for x in h)
    assert np.linalg.norm(got - want) < 1e-8 * np.linalg.norm(want)
    assert abs(h[1].logdet() - h[0].logdet()) < 1e-6


SCRIPT = """
import sys, json, hashlib
sys.path.insert(0, "kernelmatrices.jl_gb300")
import numpy as np
import kmhodlr as K
from kmhodlr.data import uniform_points
out = []
for n, lv, r in ((5000, 5, 71), (20000, 8, 33), (2600, 4, 80), (2000, 3, 5)):
    pts = uniform_points(n, 21)
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, np.array([1.0, 0.1, 1e-3]), K.Matern32()), 0.0, r, K.FixedLevel(lv),
                       nystrom=True, precision=K.KM_PREC_MIXED)
    K.symmetricfactorize(hk)
    z = np.random.default_rng(22).standard_normal((n, 3))
    for v in (hk.W @ z, hk.W.T.ldiv(z), np.array([hk.logdet()])):
        out.append(hashlib.sha256(np.ascontiguousarray(v).tobytes()).hexdigest())
print(json.dumps(out))
"""


def test_cluster_sizes_bit_identical(lib):
    got = []
    for cap in ("1", "2", "4", "8"):
        r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, env=dict(os.environ, KM_NODE_CLUSTER=cap),
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr
        got.append(json.loads(r.stdout.strip().splitlines()[-1]))
    assert all(g == got[0] for g in got)
