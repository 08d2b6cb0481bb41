"""General (ACA) factorisation at ranks and sizes around its tiles: 32-column reflector blocks,
32 x 32 tiles, right-hand sides 8 (4, 2, 1) at a time, row chunks of 128 to 512.

Every check is an identity of the matrix that the engine itself multiplies by before factorising:
W (W' x) = K x, K (K^-1 b) = b, W^-1 and W'^-1 against W and W'.  The matrices have a unit diagonal
plus a nugget of 1, condition number below 1e5, so 1e-10 relative is well above rounding.  (With a
longer range the rank-limited matrix of 25000 points is not positive definite.)
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lv,rank,k", [(300, 1, 2, 1), (300, 1, 31, 2), (517, 2, 32, 3), (517, 2, 33, 8), (1000, 2, 64, 9),
                                        (1003, 1, 65, 17), (2500, 3, 97, 5), (4100, 2, 40, 33), (6000, 2, 130, 8),
                                        (25000, 5, 24, 4)])
def test_factor_identities(lib, n, lv, rank, k):
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    pts = uniform_points(n, 3)
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, np.array([1.0, 0.02 if n < 10000 else 0.005, 1.0]), K.Matern32()), 1e-13, rank,
                       K.FixedLevel(lv))
    x = np.random.default_rng(4).standard_normal((n, k))
    y = hk @ x
    K.symmetricfactorize(hk)
    close = lambda a, b: np.linalg.norm(a - b) < 1e-10 * np.linalg.norm(b)  # noqa: E731
    assert close(hk @ x, y)
    assert close(hk.ldiv(y), x)
    assert close(hk.W.ldiv(hk.W @ x), x)
    assert close(hk.W.T.ldiv(hk.W.T @ x), x)
    one = hk.ldiv(y[:, :1].copy())
    assert close(one, x[:, :1])


def test_unsorted_points_full_rank(lib):
    """Unsorted points: the top block's rank comes close to its size (the README example's case)."""
    import kmhodlr as K
    from kmhodlr.data import normal_points
    from oracle import hodlr_oracle as O
    n = 600
    pts = normal_points(n, 5)
    p = np.array([1.0, 1.0, 1.0])
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, p, K.RatQuad()), 1e-12, 0, K.FixedLevel(1))
    A = O.kernel_block(O.KERNEL_RQ, pts, pts, p)
    b = np.random.default_rng(6).standard_normal(n)
    K.symmetricfactorize(hk)
    want = np.linalg.solve(A, b)
    assert np.linalg.norm(hk.ldiv(b) - want) < 1e-9 * np.linalg.norm(want)
    assert abs(hk.logdet() - np.linalg.slogdet(A)[1]) < 1e-8 * n


def test_solve_at_the_memory_budget(lib):
    """Where the scratch of the split does not fit, the node applications run without it: the same solution to
    1e-12 (only the order of the sums over the rows differs; condition number below 1e2)."""
    import ctypes as C
    import torch
    from kmhodlr import _lib as L, hodlr as KH
    from kmhodlr.data import uniform_points
    n, k = 4100, 512
    pts, p = uniform_points(n, 3), np.array([1.0, 0.005, 1.0])
    b = np.asfortranarray(np.random.default_rng(4).standard_normal((n, k)))

    def solve(fraction):
        h = C.c_void_p()
        cfg = L.KmConfig(device=0, precision=L.KM_PREC_FP64, hbm_budget_fraction=fraction, refine_max_iter=0, refine_tol=0.0)
        assert lib.km_create(C.byref(cfg), C.byref(h)) == L.KM_OK
        assert lib.km_assemble(h, KH._dp(pts), n, L.KM_KERNEL_MATERN32, KH._dp(p), 3, L.KM_METHOD_ACA, 1e-13, 40,
                               L.KM_LEVEL_FIXED, 2) == L.KM_OK, lib.km_last_error(h)
        assert lib.km_factorize(h) == L.KM_OK, lib.km_last_error(h)
        x, st = np.empty_like(b, order="F"), L.KmStats()
        assert lib.km_solve(h, KH._dp(b), KH._dp(x), k) == L.KM_OK, lib.km_last_error(h)
        assert lib.km_get_stats(h, C.byref(st)) == L.KM_OK
        lib.km_destroy(h)
        return x, st.device_bytes

    want, used = solve(0.8)
    got, less = solve((used - 4096) / torch.cuda.mem_get_info()[1])
    assert less < used - 4096
    assert np.linalg.norm(got - want) < 1e-12 * np.linalg.norm(want)


@pytest.mark.parametrize("n,lv,k", [(40000, 5, 17), (70000, 6, 300)])
def test_tall_sides(lib, n, lv, k):
    """Sides of 20000 and 35000 rows: row chunks above the 512 rows that a projection stages at a time."""
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    pts = uniform_points(n, 3)
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, np.array([1.0, 0.003, 1.0]), K.Matern32()), 1e-13, 24, K.FixedLevel(lv))
    x = np.random.default_rng(4).standard_normal((n, k))
    y = hk @ x
    K.symmetricfactorize(hk)
    close = lambda a, b: np.linalg.norm(a - b) < 1e-10 * np.linalg.norm(b)  # noqa: E731
    assert close(hk @ x, y)
    assert close(hk.ldiv(y), x)
    assert close(hk.W.ldiv(hk.W @ x), x)


@pytest.mark.parametrize("n,lv", [(24575, 4), (24576, 4), (24577, 4), (24578, 4)])
def test_panels_at_the_cluster_limit(lib, n, lv):
    """Top panels of 12287 to 12289 rows: 12288 is what 16 CTAs hold, one more goes to the kernels of all SMs, and
    at 24577 points the two panels of one level go different ways."""
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    pts = uniform_points(n, 3)
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, np.array([1.0, 0.005, 1.0]), K.Matern32()), 1e-13, 33, K.FixedLevel(lv))
    x = np.random.default_rng(4).standard_normal((n, 2))
    y = hk @ x
    K.symmetricfactorize(hk)
    close = lambda a, b: np.linalg.norm(a - b) < 1e-10 * np.linalg.norm(b)  # noqa: E731
    assert close(hk @ x, y)
    assert close(hk.ldiv(y), x)
    assert close(hk.W.ldiv(hk.W @ x), x)
    assert close(hk.W.T.ldiv(hk.W.T @ x), x)
