"""Float-pair leaf kernels: the explicit Q of a leaf panel with its columns in registers (8, 16 or 32 rows a
lane: leaves up to 256, 512 and 1024 points, in place beyond) and the leaf solves of 32 and more right-hand
sides (64 x 64 tiles, 12 columns a CTA).

Against the FP64 form, with the targets of the mixed form (test_gpu_mixed.py): solves to 1e-8 relative,
logdet to 1e-6; W W^{-1} z = z, which needs an orthonormal Q, to 1e-9."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lv,r,k", [(140, 1, 32, 33), (300, 1, 64, 36), (510, 1, 3, 32), (513, 1, 33, 37), (514, 1, 80, 72),
                                      (1024, 1, 72, 48), (1027, 1, 31, 35), (2048, 1, 65, 33), (2052, 1, 40, 34),
                                      (3001, 4, 72, 73), (4500, 3, 17, 64), (140, 1, 32, 1), (513, 1, 33, 2), (514, 1, 60, 4),
                                      (1280, 1, 40, 5), (1000, 2, 72, 13), (2045, 1, 80, 3), (2048, 1, 20, 16)])
def test_solve(lib, n, lv, r, k):
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    pts = uniform_points(n, 41)
    km = K.KernelMatrix(pts, pts, np.array([1.0, 0.1, 1e-2]), K.Matern32())
    b = np.random.default_rng(42).standard_normal((n, k))
    h = [K.KernelHODLR(km, 0.0, r, K.FixedLevel(lv), nystrom=True, precision=p) for p in (K.KM_PREC_FP64, K.KM_PREC_MIXED)]
    for x in h:
        K.symmetricfactorize(x)
    want, got = (x.ldiv(b) for x in h)
    assert np.linalg.norm(got - want) < 1e-8 * np.linalg.norm(want)
    assert abs(h[1].logdet() - h[0].logdet()) < 1e-6
    z = h[1].W @ h[1].W.ldiv(b)
    assert np.linalg.norm(z - b) < 1e-9 * np.linalg.norm(b)


@pytest.mark.parametrize("n,lv,r,k", [(16 * 512, 9, 8, 20), (37 * 512, 9, 16, 16), (38 * 512, 9, 16, 20), (65 * 256, 8, 24, 33),
                                      (66 * 256 + 7, 8, 24, 48), (67 * 128, 7, 24, 100), (1024, 0, 2, 33), (1000, 0, 2, 9)])
def test_small_leaves_and_few_ctas(lib, n, lv, r, k):
    """Both sides of the rules that send many leaves with ill-filled tiles to the substitution and the chunks of few
    leaves to the kernel of 4 columns.  Tolerances as above."""
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    pts = uniform_points(n, 41)
    km = K.KernelMatrix(pts, pts, np.array([1.0, 0.1, 1e-1]), K.Matern32())
    b = np.random.default_rng(42).standard_normal((n, k))
    h = [K.KernelHODLR(km, 0.0, r, K.FixedLevel(lv), nystrom=True, precision=p) for p in (K.KM_PREC_FP64, K.KM_PREC_MIXED)]
    for x in h:
        K.symmetricfactorize(x)
    want, got = (x.ldiv(b) for x in h)
    assert np.linalg.norm(got - want) < 1e-8 * np.linalg.norm(want)
    z = h[1].W.T @ h[1].W.T.ldiv(b)
    assert np.linalg.norm(z - b) < 1e-9 * np.linalg.norm(b)
