"""FP64 node factorisation (km_node64.cu): ranks around its 32-row chunks and the number of columns
a CTA or warp owns, on trees whose levels run with 1, 2, 4 and 8 CTAs a node.

Against the oracle: K^-1 b to 1e-9 relative and logdet to 1e-9 n, the tolerances of the FP64 Nystrom
parity tests (the matrices' condition number is below 1e6).  Cluster sizes: equal bits.
"""
import ctypes as C
import json
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("n,lv,r", [(900, 1, 2), (1100, 2, 31), (1100, 2, 32), (1101, 2, 33), (1300, 3, 64), (1303, 3, 65),
                                    (3000, 5, 72), (5000, 5, 80), (12345, 7, 79), (20000, 8, 40)])
def test_solve_and_logdet(lib, n, lv, r):
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    from oracle import hodlr_oracle as O
    pts = uniform_points(n, 11)
    p = np.array([1.0, 0.1, 1e-2])
    b = np.random.default_rng(12).standard_normal((n, 2))
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, p, K.Matern32()), 0.0, r, K.FixedLevel(lv), nystrom=True)
    K.symmetricfactorize(hk)
    ok = O.build_hodlr(O.KernelMatrix(pts, pts, p, O.KERNEL_MATERN32), 0.0, r, O.FixedLevel(lv), nystrom=True)
    O.symmetricfactorize(ok)
    want = O.hodlr_ldiv(ok, b)
    assert np.linalg.norm(hk.ldiv(b) - want) < 1e-9 * np.linalg.norm(want)
    assert abs(hk.logdet() - O.hodlr_logdet(ok)) < 1e-9 * n
    z = np.random.default_rng(13).standard_normal((n, 2))
    back = hk.W.ldiv(hk.W @ z)
    assert np.linalg.norm(back - z) < 1e-9 * np.linalg.norm(z)


SCRIPT = """
import sys, json, hashlib
sys.path.insert(0, "kernelmatrices.jl_gb300")
import numpy as np
import kmhodlr as K
from kmhodlr.data import uniform_points
out = []
for n, lv, r in ((5000, 5, 72), (20000, 8, 33), (2600, 4, 80)):
    pts = uniform_points(n, 21)
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, np.array([1.0, 0.1, 1e-3]), K.Matern32()), 0.0, r, K.FixedLevel(lv),
                       nystrom=True)
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


@pytest.mark.parametrize("r", [33, 72])
def test_wait_runs_out_then_the_handle_recovers(lib, r):
    """km_set_wait_limit(h, 0) makes every bounded wait of the node kernel give up."""
    from kmhodlr import _lib as L, hodlr as KH
    from kmhodlr.data import uniform_points
    n = 4096
    pts = uniform_points(n, 31)
    p = np.array([1.0, 0.1, 1e-3])
    b = np.asfortranarray(np.random.default_rng(32).standard_normal((n, 2)))

    def make():
        h = C.c_void_p()
        cfg = L.KmConfig(device=0, precision=L.KM_PREC_FP64, hbm_budget_fraction=0.8, refine_max_iter=0, refine_tol=0.0)
        assert lib.km_create(C.byref(cfg), C.byref(h)) == L.KM_OK
        return h

    def assemble(h):
        assert lib.km_assemble(h, KH._dp(pts), n, L.KM_KERNEL_MATERN32, KH._dp(p), 3, L.KM_METHOD_NYSTROM, 0.0, r,
                               L.KM_LEVEL_FIXED, 4) == L.KM_OK

    def solve(h):
        x = np.empty_like(b, order="F")
        assert lib.km_factorize(h) == L.KM_OK, lib.km_last_error(h)
        assert lib.km_solve(h, KH._dp(b), KH._dp(x), 2) == L.KM_OK
        return x

    h, fresh = make(), make()
    assemble(h)
    assert lib.km_set_wait_limit(h, 0) == L.KM_OK
    assert lib.km_factorize(h) == L.KM_ERR_TIMEOUT
    assert b"bounded wait" in lib.km_last_error(h)
    assert lib.km_set_wait_limit(h, -1) == L.KM_OK
    assemble(h)
    assemble(fresh)
    assert np.array_equal(solve(h), solve(fresh))
    lib.km_destroy(h)
    lib.km_destroy(fresh)


@pytest.mark.parametrize("n,lv,r", [(160, 3, 2), (331, 4, 3), (332, 3, 4), (500, 4, 5), (700, 4, 6), (701, 3, 7),
                                    (333, 3, 8), (400, 3, 9)])
def test_ranks_below_the_cluster_size(lib, n, lv, r):
    """With 8 CTAs a node and fewer columns than that, some CTAs own no column.  The factor's
    identities to 1e-12 times the condition number (below 1e3 with a nugget of 1), and the oracle."""
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    from oracle import hodlr_oracle as O
    pts = uniform_points(n, 11)
    p = np.array([1.0, 0.05, 1.0])
    b = np.random.default_rng(12).standard_normal((n, 3))
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, p, K.Matern32()), 0.0, r, K.FixedLevel(lv), nystrom=True)
    y = hk @ b
    K.symmetricfactorize(hk)
    ok = O.build_hodlr(O.KernelMatrix(pts, pts, p, O.KERNEL_MATERN32), 0.0, r, O.FixedLevel(lv), nystrom=True)
    O.symmetricfactorize(ok)
    close = lambda a, c: np.linalg.norm(a - c) < 1e-9 * np.linalg.norm(c)  # noqa: E731
    assert close(hk.ldiv(b), O.hodlr_ldiv(ok, b))
    assert close(hk.ldiv(y), b) and close(hk @ b, y)
    assert close(hk.W.ldiv(hk.W @ b), b) and close(hk.W.T.ldiv(hk.W.T @ b), b)
    assert abs(hk.logdet() - O.hodlr_logdet(ok)) < 1e-9 * n
