"""The forms of case-wise weighting and RF-GAP that only large forests or scarce
memory reach by themselves, forced at small sizes, against the oracle: the range
table in several blocks of rows, the importance in several chunks of trees (the
last one partial), weights formed per pair; and the importance walk's widths
(1, 2 and 4 words of features, more than one block of 256) and votes of many
classes.  Every sum runs in the reference's order, so all comparisons are
exact."""
import numpy as np
import pytest

from rfx_b200 import synth

pytestmark = pytest.mark.gpu


def _same(ctx, O, f, n, names=("avimp", "sqsd", "qimp", "qimpm")):
    q, nout = ctx.casewise_votes()
    assert np.array_equal(q, O["q_raw"]) and np.array_equal(nout, O["nout"])
    assert np.array_equal(ctx.proximity_upper_f64(), O["Sd"])
    got = ctx.varimp(True)
    for g, want in zip(got, names):
        assert np.array_equal(g, O[want], equal_nan=True), want
    short = ctx.varimp(False)
    assert np.array_equal(short[0], got[0], equal_nan=True) and np.array_equal(short[1], got[1], equal_nan=True)
    assert np.array_equal(ctx.proximity_rfgap(), orc_rfgap(f, O)[np.triu_indices(n)])


def orc_rfgap(f, O):
    from oracle import oracle as orc

    return orc.rfgap(f.nin, O["leaf"])


def _case(n, p, c, T, nodesize=1):
    from oracle import oracle as orc
    from rfx_b200 import abi

    X, y = synth.gaussian_classes(n, p, c, seed=n + p, mean_scale=1.0)
    f = abi.grow_forest(X, y, T, max(1, int(p ** 0.5)), nodesize, nclass=c)
    return X, y, f, orc.analyse(X, y, f, casewise=True, want_cw=True, want_leaf=True)


# 1 MB of ranges: 16 bytes x 97 trees a row, 675 rows a block (four blocks,
# the last of 24 rows); of importance values: 4 x 2,049 x 10 bytes a tree,
# 12 trees a chunk (nine chunks, the last of one tree)
@pytest.mark.parametrize("weights", ["1", "0"])
def test_pieces(built, monkeypatch, weights):
    from rfx_b200 import abi

    n, T = 2049, 97
    X, y, f, O = _case(n, 9, 3, T)
    monkeypatch.setenv("RFX_CW_MB", "1")
    monkeypatch.setenv("RFX_CW_WEIGHTS", weights)
    ctx = abi.Context(0, use_casewise=True)
    ctx.load(f, X, y)
    _same(ctx, O, f, n)
    ctx.close()
    ctx = abi.Context(0)  # unweighted sums
    ctx.load(f, X, y)
    assert np.array_equal(ctx.proximity_upper_f64(), ctx.proximity_upper().astype(np.float64))
    ctx.close()


@pytest.mark.parametrize("p,c", [(64, 8), (65, 9), (128, 17), (129, 33), (256, 64), (257, 2), (600, 64)])
def test_features_and_classes(built, p, c):
    from rfx_b200 import abi

    n = 300
    X, y, f, O = _case(n, p, c, 21)
    ctx = abi.Context(0, use_casewise=True)
    ctx.load(f, X, y)
    _same(ctx, O, f, n)
    ctx.close()
