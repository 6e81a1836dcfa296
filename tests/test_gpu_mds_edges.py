"""The MDS and outlier kernels at the edges of their tiles, against FP64 numpy.

Full-matrix MDS: the iteration ends when the eigenvalues change by less than
1e-14, so an eigenvector's residual |B v - lambda v| (whose square over the gap
bounds the eigenvalue's error) stays below 1e-6 of the largest eigenvalue and
the eigenvalues agree to 1e-9 of it, whatever the gaps.  Outlier scores: FP64
sums rounded to float32, 1e-4 as in the test of rank 16."""
import numpy as np
import pytest

from rfx_b200 import synth

pytestmark = pytest.mark.gpu


def _load(n, T, nodesize=1):
    from rfx_b200 import abi

    X, y = synth.gaussian_classes(n, 13, 3, seed=n, mean_scale=1.0)
    f = abi.grow_forest(X, y, T, 3, nodesize, nclass=3)
    ctx = abi.Context(0)
    ctx.load(f, X, y)
    return ctx


# 64 rows make a partial Gram matrix; a warp adds 32 of them at a time (n = 2,048)
@pytest.mark.parametrize("n", [40, 64, 65, 1985, 2048, 2049])
def test_full_matrix_mds(built, n):
    ctx = _load(n, 80)
    _, nout, _ = ctx.route_oob()
    P = ctx.finishprox(ctx.proximity_upper(), full=True)
    C, ev = ctx.mds3d_full(P)
    ctx.close()
    Q = P.astype(np.float64)
    Q = np.where(nout[:, None] > 0, Q / np.maximum(nout, 1)[:, None], Q)
    Q = 0.5 * (Q + Q.T)
    np.fill_diagonal(Q, 1.0)
    D2 = (Q.max() - Q) ** 2
    np.fill_diagonal(D2, 0.0)
    m = D2.mean(1)
    B = -0.5 * (D2 - m[:, None] - m[None, :] + m.mean())
    w = np.linalg.eigvalsh(B)[::-1][:3]
    assert np.abs(ev - w).max() <= 1e-9 * w[0]
    V = C / np.sqrt(ev)
    assert np.abs(V.T @ V - np.eye(3)).max() <= 1e-6
    assert np.linalg.norm(B @ V - V * ev, axis=0).max() <= 1e-6 * w[0]


@pytest.mark.parametrize("k", [1, 7, 63, 64, 65, 95, 97, 104])
def test_outlier_scores(built, k):
    n = 701  # the last CTA takes 29 of its 32 rows
    ctx = _load(n, 40, nodesize=5)
    A, _ = ctx.lowrank(k, oversample=16, power_iters=1, precision=0)
    got = ctx.outlier_scores()
    ctx.close()
    G = A.astype(np.float64) @ A.astype(np.float64).T
    np.fill_diagonal(G, 0.0)
    raw = 1.0 / (1.0 + (G ** 2).sum(1))
    assert np.allclose(got, raw / np.sort(raw)[n // 2], rtol=1e-4)
