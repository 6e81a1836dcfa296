"""Case-wise weighting and RF-GAP at the edges of the row kernel's tiles, against
the oracle: sizes around the column window (1,024), tree counts around a step
(32 trees), leaves with hundreds of members, one-tree and tiny forests.  Every
sum runs in the reference's order, so all comparisons are exact."""
import numpy as np
import pytest

from rfx_b200 import synth

pytestmark = pytest.mark.gpu

CASES = [("gauss", 17, 3, 1), ("gauss", 33, 1, 1), ("gauss", 511, 257, 1), ("cover", 1025, 33, 1),
         ("gauss", 1024, 256, 5), ("gauss", 2049, 12, 900), ("cover", 4097, 6, 300), ("gauss", 8193, 4, 1)]


@pytest.mark.parametrize("data,n,T,nodesize", CASES)
def test_weighted_matches_oracle(built, data, n, T, nodesize):
    from oracle import oracle as orc
    from rfx_b200 import abi

    X, y = synth.mixed_cover(n, seed=n) if data == "cover" else synth.gaussian_classes(n, 9, 3, seed=n, mean_scale=1.0)
    cat = synth.detect_categorical(X) if data == "cover" else None
    c = int(y.max()) + 1
    f = abi.grow_forest(X, y, T, 3, nodesize, nclass=c, cat=cat)
    O = orc.analyse(X, y, f, casewise=True, want_cw=True, want_leaf=True)
    ctx = abi.Context(0, use_casewise=True)
    ctx.load(f, X, y)
    q, nout = ctx.casewise_votes()
    assert np.array_equal(q, O["q_raw"]) and np.array_equal(nout, O["nout"])
    S = ctx.proximity_upper_f64()
    assert np.array_equal(S, O["Sd"])
    assert np.array_equal(ctx.finishprox_f64(S), orc.finishprox_f64(O["Sd"], O["nout"]))
    avimp, sqsd, qimp, qimpm = ctx.varimp(True)
    for got, want in ((avimp, "avimp"), (sqsd, "sqsd"), (qimp, "qimp"), (qimpm, "qimpm")):
        assert np.array_equal(got, O[want], equal_nan=True), want
    a2, s2, _, _ = ctx.varimp(False)
    assert np.array_equal(a2, avimp, equal_nan=True) and np.array_equal(s2, sqsd, equal_nan=True)
    ctx.close()
    ctx = abi.Context(0)
    ctx.load(f, X, y)
    P = ctx.proximity_rfgap()
    assert np.array_equal(P, orc.rfgap(f.nin, O["leaf"])[np.triu_indices(n)])
    assert np.array_equal(ctx.proximity_upper_f64(), ctx.proximity_upper().astype(np.float64))
    ctx.close()
