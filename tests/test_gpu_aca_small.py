"""ACA of many small blocks: clusters of 2 CTAs for sides up to 40, of 4 up to 130, from 64 blocks on, beside the
clusters of 16 of the others.  Ranks and pivots exactly the oracle's (rational quadratic: every entry is formed alike),
the blocks to 1e-12 relative, as in test_gpu_aca.py."""
import numpy as np
import pytest

from oracle import hodlr_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lv,rank,tol", [(640, 6, 0, 1e-8), (2560, 7, 0, 1e-6), (2625, 6, 12, 1e-10), (5300, 7, 10, 1e-8),
                                           (8321, 7, 8, 1e-8), (4100, 8, 5, 1e-12)])
def test_ranks_and_pivots(lib, n, lv, rank, tol):
    import kmhodlr as K
    from kmhodlr.data import uniform_points
    pts = uniform_points(n, n + 3)
    p = np.array([1.0, 0.2, 1.0])
    ohk = O.build_hodlr(O.KernelMatrix(pts, pts, p, O.KERNEL_RQ), tol, rank, O.FixedLevel(lv), nystrom=False)
    hk = K.KernelHODLR(K.KernelMatrix(pts, pts, p, K.RatQuad()), tol, rank, K.FixedLevel(lv), nystrom=False)
    assert list(hk.block_ranks()) == [u.shape[1] for level in ohk.U for u in level]
    q = 0
    for level in range(len(ohk.U)):
        for k in range(len(ohk.U[level])):
            rows, cols = hk.aca_pivots(q)
            assert (list(rows), list(cols)) == tuple(map(list, ohk.pivots[level][k])), (level, k)
            if k < 2:
                U, V = hk.block_factors(q)
                want = ohk.U[level][k] @ ohk.V[level][k].T
                assert np.linalg.norm(U @ V.T - want) < 1e-12 * np.linalg.norm(want)
            q += 1
