"""Leaf solves, projections and expansions at the edges of their blocks: 32-row blocks and their
inverses, column chunks of 1, 2, 4, 8 and 16, row chunks of 128, basis columns split over CTAs.

Against the oracle's solves and factor products, FP64 to 1e-9 and mixed to 1e-7 relative (the
tolerances of the parity tests; condition numbers below 1e6).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(0, 1e-9), (1, 1e-7)])
@pytest.mark.parametrize("n,lv,r,k", [(66, 1, 2, 1), (130, 1, 31, 2), (1000, 1, 32, 25), (1027, 3, 40, 3), (1029, 2, 72, 17),
                                      (3001, 4, 64, 73), (9000, 5, 80, 33), (20001, 7, 50, 9)])
def test_solves_and_projections(lib, precision, tol, n, lv, r, k):
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    from oracle import hodlr_oracle as O
    pts = uniform_points(n, 41)
    p = np.array([1.0, 0.1, 1e-2])
    b = np.random.default_rng(42).standard_normal((n, k))
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, p, K.Matern32()), 0.0, r, K.FixedLevel(lv), nystrom=True,
                       precision=precision)
    K.symmetricfactorize(hk)
    ok = O.build_hodlr(O.KernelMatrix(pts, pts, p, O.KERNEL_MATERN32), 0.0, r, O.FixedLevel(lv), nystrom=True)
    O.symmetricfactorize(ok)
    close = lambda a, c: np.linalg.norm(a - c) < tol * np.linalg.norm(c)  # noqa: E731
    assert close(hk.ldiv(b), O.hodlr_ldiv(ok, b))
    assert close(hk.W.ldiv(hk.W @ b), b)
    assert close(hk.W.T.ldiv(hk.W.T @ b), b)
    z = O.rademacher_probes(n, k, 43)
    nll, g = hk.nll_grad_seeded(b[:, 0], k, 43)
    assert abs(nll - O.negloglik(ok, b[:, 0])) < tol * abs(nll)
    # the estimator depends on the factor's basis in the null directions of the leaf panels
    want = O.stoch_gradient(O.KernelMatrix(pts, pts, p, O.KERNEL_MATERN32), ok, b[:, 0], 3, [z[:, j] for j in range(k)])
    assert np.linalg.norm(g - want) < 1e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("n,lv,k", [(16 * 768 + 15, 4, 20), (16 * 769, 4, 19), (16 * 800 + 3, 4, 40), (16 * 1057, 4, 33),
                                    (32 * 900 + 1, 5, 9), (8 * 1120, 3, 80)])
def test_backward_solves_of_large_leaves(lib, n, lv, k):
    """Leaves above 768 points with more CTAs than SMs turn the factor's entries round in shared memory: last blocks
    of 1 to 32 rows, chunks of 2 and 4 columns, ragged ones too.  A column alone takes the direct form; both
    against W' to 1e-12 (unit diagonal plus a nugget of 1, condition number below 1e3)."""
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    pts = uniform_points(n, 41)
    b = np.random.default_rng(42).standard_normal((n, k))
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, np.array([1.0, 0.02, 1.0]), K.Matern32()), 0.0, 16, K.FixedLevel(lv),
                       nystrom=True)
    K.symmetricfactorize(hk)
    x = hk.W.T.ldiv(b)
    assert np.linalg.norm(hk.W.T @ x - b) < 1e-12 * np.linalg.norm(b)
    for c in (0, k // 2, k - 1):
        one = hk.W.T.ldiv(b[:, c])
        assert np.linalg.norm(one - x[:, c]) < 1e-12 * np.linalg.norm(one)
