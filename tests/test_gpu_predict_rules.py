"""Test-set votes on both sides of every line of the rule that picks the
prediction kernel's form (rows, trees, features, classes, categorical features,
go-left table, tree size), against the oracle (exact votes)."""
import dataclasses

import numpy as np
import pytest

from rfx_b200 import synth

pytestmark = pytest.mark.gpu


def _check(X, y, T, c, rows, cat=None, table=False):
    from oracle import oracle as orc
    from rfx_b200 import abi

    n = X.shape[0] - max(rows)
    f = abi.grow_forest(X[:n], y[:n], T, 3, 1, nclass=c, cat=cat)
    if table:
        rng = np.random.default_rng(5)
        f = dataclasses.replace(f, catgoleft=rng.integers(0, 2, int(f.offs[-1]) * f.maxcat).astype(np.int32))
    ctx = abi.Context(0)
    ctx.load(f, X[:n], y[:n])
    want = orc.predict(X[n:], f)[0]
    for m in rows:
        assert np.array_equal(ctx.predict_votes(X[n: n + m]), want[:m]), m
    ctx.close()


@pytest.mark.parametrize("T,rows", [(639, [32, 33, 255, 1500, 4096]), (640, [31, 32, 33, 255, 256, 1499, 1500, 4095, 4096]),
                                    (480, [4096, 4167, 4700])])
@pytest.mark.parametrize("table", [False, True])
def test_categorical(built, T, rows, table):
    n = 300
    X, y = synth.mixed_cover(n + max(rows), seed=T)
    X[n::17, 2] = np.nan
    X[n::7, 20] = np.float32(0.49999997)
    X[n::13, 13] = -3.0
    _check(X, y, T, 7, rows, cat=synth.detect_categorical(X[:n]), table=table)


def test_categorical_large_with_table(built):
    n = 300
    X, y = synth.mixed_cover(n + 9376, seed=2)
    _check(X, y, 640, 7, [9374, 9375, 9376], cat=synth.detect_categorical(X[:n]), table=True)  # 6,000,000 walks


@pytest.mark.parametrize("p,c,T,n,rows", [
    (39, 10, 20, 300, [61, 1500, 4096]), (40, 10, 20, 300, [1, 32, 33, 255, 256, 1499, 1500, 4097]),
    (40, 11, 20, 300, [61, 1500]), (40, 16, 20, 300, [1500]), (40, 17, 20, 300, [1500]),
    (12, 3, 479, 300, [61]), (12, 3, 480, 300, [1, 33, 255, 256]), (12, 11, 480, 300, [61]),
    (12, 5, 12, 1500, [32767, 32768, 33000]), (12, 6, 12, 1500, [32768]), (12, 5, 12, 200, [32768]),
    (40, 10, 12, 1500, [32767, 32768]), (80, 10, 12, 1500, [32767, 32768]), (80, 17, 12, 1500, [32768])])
def test_numeric(built, p, c, T, n, rows):
    X, y = synth.gaussian_classes(n + max(rows), p, c, seed=p + c, mean_scale=0.3)
    _check(X, y, T, c, rows)
