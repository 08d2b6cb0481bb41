"""Sweep kernels that start before the kernel in front of them has ended (km_apply.cu): trees of 1 to 9
levels, staged and unstaged launches (few and many columns), solves and products back to back.

W W^{-1} b = b to 1e-9 relative; the same call again gives the same bits (a vector read too early would
still hold the previous call's values)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["KM_PREC_FP64", "KM_PREC_MIXED"])
@pytest.mark.parametrize("n,lv,r,k", [(400, 1, 33, 1), (1000, 2, 72, 3), (9000, 6, 40, 1), (40000, 9, 24, 1), (40000, 9, 72, 2),
                                      (20000, 7, 80, 33)])
def test_back_to_back(lib, n, lv, r, k, prec):
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    pts = uniform_points(n, 51)
    if n // 2**lv < r + 2:
        n = (r + 2) * 2**lv
        pts = uniform_points(n, 51)
    km = K.KernelMatrix(pts, pts, np.array([1.0, 0.1, 1e-2]), K.Matern32())
    hk = K.KernelHODLR(km, 0.0, r, K.FixedLevel(lv), nystrom=True, precision=getattr(K, prec))
    K.symmetricfactorize(hk)
    b = [np.random.default_rng(52 + i).standard_normal((n, k)) for i in range(2)]
    first = [hk.ldiv(x) for x in b]
    for _ in range(3):
        for x, want in zip(b, first):
            assert np.array_equal(hk.ldiv(x), want)
    for x in b:
        assert np.linalg.norm(hk.W @ hk.W.ldiv(x) - x) < 1e-9 * np.linalg.norm(x)
        assert np.linalg.norm(hk.W.T @ hk.W.T.ldiv(x) - x) < 1e-9 * np.linalg.norm(x)
