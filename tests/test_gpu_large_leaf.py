"""Product with a matrix of the largest leaves that the leaf product holds: 8 columns of points and landmarks
together with its 32 KB of partial sums fill the shared memory of a CTA (227 KB), 3120 rows and landmarks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf,r", [(3112, 8), (3090, 30)])
def test_matvec(lib, leaf, r):
    """Against the oracle; sums of 6000 terms of either sign in FP64, 1e-12 of the largest as the other products."""
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    from oracle import hodlr_oracle as O
    n = 2 * leaf
    pts = uniform_points(n, 5)
    p = np.array([1.0, 0.1, 1e-2])
    x = np.random.default_rng(6).standard_normal((n, 3))
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, p, K.Matern32()), 0.0, r, K.FixedLevel(1), nystrom=True)
    ok = O.build_hodlr(O.KernelMatrix(pts, pts, p, O.KERNEL_MATERN32), 0.0, r, O.FixedLevel(1), nystrom=True)
    want = O.hodlr_mul(ok, x)
    assert np.max(np.abs(hk @ x - want)) < 1e-12 * np.max(np.abs(want))
