"""finishprox at the edges of its tiles (64 x 64 below n = 4,096, 64 x 128 from
there on), full and packed, INT32 and FP64 sums, against the oracle (exact: the
FP64 operations run in the reference's order)."""
import numpy as np
import pytest

from rfx_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 129, 4095, 4096, 4161, 4225])
def test_finishprox_matches_oracle(built, n):
    from oracle import oracle as orc
    from rfx_b200 import abi

    m = max(n, 40)
    X, y = synth.gaussian_classes(m, 5, 3, seed=m, mean_scale=1.0)
    f = abi.grow_forest(X[:n], y[:n], 3, 2, 1, nclass=3)
    ctx = abi.Context(0)
    ctx.load(f, X[:n], y[:n])
    _, nout, _ = ctx.route_oob()
    S = np.random.default_rng(n).integers(0, 9, n * (n + 1) // 2).astype(np.int32)
    i = np.arange(n, dtype=np.int64)
    S[i * n - i * (i - 1) // 2] = 0  # the diagonal
    for full in (True, False):
        want = orc.finishprox(S, nout, full=full)
        assert np.array_equal(ctx.finishprox(S, full=full), want)
        assert np.array_equal(ctx.finishprox_f64(S.astype(np.float64), full=full), want)
    ctx.close()
