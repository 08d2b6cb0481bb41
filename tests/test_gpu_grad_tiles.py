"""Gradient contractions at the edges of their tiles: last leaf tiles of 1, 8, 9, 16, 17, 31 and 32 rows (the
short ones change sides), odd and even column counts around the chunk of 32 and the CTA of 40.

Against the oracle with the same probes, to the 1e-6 of test_gpu_gradient.py (FP64) and 1e-5 of
test_gpu_hessian.py (float pairs)."""
import numpy as np
import pytest

from oracle import hodlr_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf,p", [(65, 24), (72, 31), (73, 32), (80, 33), (81, 39), (95, 40), (96, 41), (129, 73)])
@pytest.mark.parametrize("mixed", [False, True])
def test_gradient(lib, leaf, p, mixed):
    import kmhodlr as K
    from kmhodlr.data import rademacher, uniform_points
    n, rank, level = 4 * leaf, 24, 2
    pts = uniform_points(n, n + 5)
    params = (1.0, 0.1, 1e-2)
    y = np.random.default_rng(n).standard_normal(n)
    V = rademacher(n, p, n + 7)
    ok = O.KernelMatrix(pts, pts, np.array(params), O.KERNEL_MATERN32)
    ohk = O.build_hodlr(ok, 0.0, rank, O.FixedLevel(level), nystrom=True)
    O.symmetricfactorize(ohk)
    g0 = O.stoch_gradient(ok, ohk, y, 3, [V[:, c] for c in range(p)])
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, params, K.Matern32()), 0.0, rank, K.FixedLevel(level), nystrom=True,
                       precision=K.KM_PREC_MIXED if mixed else K.KM_PREC_FP64)
    K.symmetricfactorize(hk)
    g = K.stoch_gradient(hk, y, V)
    assert np.all(np.abs(g - g0) <= (1e-5 if mixed else 1e-6) * np.max(np.abs(g0)))
