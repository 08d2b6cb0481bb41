"""FP64 leaf Cholesky (km_chol.cu): one leaf holding the whole matrix, so W is the leaf factor.

Sizes around the block width (32 columns, 16 above 743 points, 8 above 1497) and the tile (32 rows).
The factor of a matrix of condition number about 10 (unit diagonal plus a nugget of 1) has a relative
error of at most about m eps; 1e-12 leaves room for m = 1600.
"""
import numpy as np
import pytest
import scipy.linalg as sla

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 31, 32, 33, 64, 65, 500, 743, 744, 1600])
def test_single_leaf_factor(lib, n):
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    from oracle import hodlr_oracle as O
    pts = uniform_points(n, 7)
    p = np.array([1.0, 0.05, 1.0 + n / 100.0])
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, p, K.Matern32()), 0.0, 2, K.FixedLevel(0), nystrom=True)
    K.symmetricfactorize(hk)
    A = O.kernel_block(O.KERNEL_MATERN32, pts, pts, p)
    Lc = sla.cholesky(A, lower=True)
    z = np.random.default_rng(8).standard_normal((n, 3))
    for got, want in ((hk.W @ z, Lc @ z), (hk.W.T @ z, Lc.T @ z), (hk.ldiv(z), sla.cho_solve((Lc, True), z))):
        assert np.linalg.norm(got - want) < 1e-12 * np.linalg.norm(want)
    assert abs(hk.logdet() - 2 * np.log(np.diag(Lc)).sum()) < 1e-12 * n


def test_not_positive_definite_pivot(lib):
    """Two equal points without a nugget: unit diagonal and unit coupling, so the second one's pivot is
    exactly 1 - 1 = 0 (every other entry is below 1e-3 and their squares cancel alike)."""
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    pts = uniform_points(400, 9)
    pts[300] = pts[40]
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, np.array([1.0, 1e-3, 0.0]), K.Matern32()), 0.0, 2, K.FixedLevel(0),
                       nystrom=True)
    with pytest.raises(K.PosDefException, match=r"leaf 0 is not positive definite \(pivot 301\)"):
        K.symmetricfactorize(hk)
