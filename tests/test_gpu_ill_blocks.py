"""Leaf solves of matrices with points closer to each other than the nugget hides, next to each other in the leaf.

The solves multiply by the inverses of the factor's diagonal blocks, which loses up to a block's condition number
against a substitution; blocks with an ill-conditioned inverse are substituted.  One leaf holds the whole matrix,
so W @ I is its Cholesky factor L (products with zeros and ones), and the errors against substitutions with L
in extended precision are compared with those of the same substitutions in FP64 (numpy): at most 16 times as
large in FP64 (another order of the sums), 2^12 as large in float pairs (rounding errors up to 2^-43 an
operation, 1024 times FP64's, and the factor of 4 for the order again).  Products with the inverses are off by 100 to
10000 times as much."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _forward(L, b):
    x = b.astype(L.dtype)
    for i in range(len(L)):
        x[i] /= L[i, i]
        x[i + 1:] -= np.outer(L[i + 1:, i], x[i])
    return x


def _backward(L, b):
    x = b.astype(L.dtype)
    for i in range(len(L) - 1, -1, -1):
        x[i] /= L[i, i]
        x[:i] -= np.outer(L[i, :i], x[i])
    return x


@pytest.mark.parametrize("m", [64, 200, 333])
@pytest.mark.parametrize("nugget", [1e-6, 1e-8, 1e-10])
@pytest.mark.parametrize("precision,k", [(0, 1), (0, 2), (0, 6), (1, 33), (1, 90)])
def test_against_substitution(lib, m, nugget, precision, k):
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    rng = np.random.default_rng(m)
    q = uniform_points(m, 3)
    q[1::2] = q[0:m - 1:2][:len(q[1::2])] + 1e-5 * rng.standard_normal((len(q[1::2]), 2))
    hk = K.KernelHODLR(K.KernelMatrix(q, q, np.array([1.0, 0.3, nugget]), K.Matern32()), 0.0, 2, K.FixedLevel(0),
                       nystrom=True, precision=precision)
    K.symmetricfactorize(hk)
    L = np.tril(hk.W @ np.eye(m))
    Lx = L.astype(np.longdouble)
    smooth = np.sin(np.outer(np.arange(m) / 7.0, 1.0 + np.arange(k) / 5.0))
    factor = 16.0 if precision == 0 else 4096.0
    err = lambda a, r: np.max(np.linalg.norm((a - r).astype(float), axis=0) / np.linalg.norm(r.astype(float), axis=0))  # noqa: E731
    for b, engine, sub in ((L @ rng.standard_normal((m, k)), hk.W.ldiv, _forward),
                           (rng.standard_normal((m, k)), hk.W.T.ldiv, _backward),
                           (L @ (L.T @ smooth), hk.ldiv, lambda A, v: _backward(A, _forward(A, v)))):
        want = sub(Lx, b)
        assert err(engine(b), want) <= factor * max(err(sub(L, b), want), 2.0**-52)
