"""Product with the derivative of a Nystrom HODLR in FP64 (the landmark coefficients solved once per leaf and
column, leaf rows in items of four columns): leaves around the block of 128 items, 1 to 9 columns a chunk.

K_j x against the dense derivative blocks is covered by the gradient and Fisher tests; here the Fisher matrix
against the oracle to 1e-6 of its largest entry, the tolerance of the Hessian tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lv,r,p", [(200, 1, 7, 1), (258, 1, 33, 3), (514, 2, 40, 4), (600, 2, 64, 7), (1040, 3, 16, 8),
                                      (1030, 2, 48, 15)])
def test_fisher(lib, n, lv, r, p):
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    from oracle import hodlr_oracle as O
    pts = uniform_points(n, 61)
    params = (1.0, 0.1, 1e-2)
    y = np.random.default_rng(62).standard_normal(n)
    V = O.rademacher_probes(n, p, 63)
    ok = O.KernelMatrix(pts, pts, np.array(params), O.KERNEL_MATERN32)
    ohk = O.build_hodlr(ok, 0.0, r, O.FixedLevel(lv), nystrom=True)
    O.symmetricfactorize(ohk)
    want = O.stoch_fisher(ok, ohk, [O.derivative_hodlr(ok, j, ohk) for j in range(3)], [V[:, c] for c in range(p)])
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, params, K.Matern32()), 0.0, r, K.FixedLevel(lv), nystrom=True)
    K.symmetricfactorize(hk)
    got = K.grad_and_fisher(hk, y, V)[-1]
    assert np.max(np.abs(got - want)) < 1e-6 * np.max(np.abs(want))
