"""Test-set votes at the edges of the prediction kernel's tiles (32 samples
below 256 rows, one tree per CTA below 1,500, 128 and from 4,096 rows on 512
samples) and its class limits (counts in
shared memory, an atomic per walk beyond), with and without a go-left table, on
numeric and mixed-type tables with values outside the levels, against the oracle
(exact votes)."""
import dataclasses

import numpy as np
import pytest

from rfx_b200 import synth

pytestmark = pytest.mark.gpu


def _check(X, y, Xt, T, c, cat=None, table=False):
    from oracle import oracle as orc
    from rfx_b200 import abi

    f = abi.grow_forest(X, y, T, 3, 1, nclass=c, cat=cat)
    if table:
        rng = np.random.default_rng(5)
        f = dataclasses.replace(f, catgoleft=rng.integers(0, 2, int(f.offs[-1]) * f.maxcat).astype(np.int32))
    ctx = abi.Context(0)
    ctx.load(f, X, y)
    got = ctx.predict_votes(Xt)
    ctx.close()
    assert np.array_equal(got, orc.predict(Xt, f)[0])


@pytest.mark.parametrize("m", [1, 31, 33, 255, 256, 1499, 1500, 4095, 4096, 4609])
@pytest.mark.parametrize("table", [False, True])
def test_predict_rows(built, m, table):
    X, y = synth.mixed_cover(900 + m, seed=m)
    X, y, Xt = X[:900], y[:900], X[900:].copy()
    Xt[::7, 20] = np.float32(0.49999997)
    Xt[::11, 12] = 1.5
    Xt[::13, 13] = -3.0
    Xt[::17, 2] = np.nan
    Xt[::19, 15] = 1e30
    _check(X, y, Xt, 23, 7, cat=synth.detect_categorical(X), table=table)


@pytest.mark.parametrize("c,m", [(40, 4200), (60, 5000), (700, 70), (800, 70), (800, 4100)])
def test_predict_classes(built, c, m):
    X, _ = synth.gaussian_classes(1700 + m, 6, 3, seed=c)
    y = (np.arange(1700) % c).astype(np.int32)
    _check(X[:1700], y, X[1700:], 3, c)
