"""Launch shapes are chosen per form of the kernels: a forest without a go-left
table and one of the same sizes with a table do not share a choice."""
import dataclasses

import numpy as np
import pytest

from rfx_b200 import synth

pytestmark = pytest.mark.gpu


def test_forms_are_tuned_apart(built, monkeypatch):
    from rfx_b200 import abi

    for name in ("RFX_AUTOTUNE", "RFX_TUNE_ROUTE", "RFX_TUNE_ROUTE_LEAF", "RFX_TUNE_VWALK"):
        monkeypatch.delenv(name, raising=False)
    X, y = synth.gaussian_classes(600, 130, 3, seed=1, mean_scale=1.0)
    f = abi.grow_forest(X, y, 70, 5, 1, nclass=3)
    table = dataclasses.replace(f, catgoleft=np.zeros(int(f.offs[-1]) * f.maxcat, np.int32))
    got = []
    for forest in (f, table):
        ctx = abi.Context(0)
        ctx.load(forest, X, y)
        S = ctx.proximity_upper()  # routing in natural order
        q, _, _ = ctx.route_oob()  # and in leaf order
        got.append([S, q, *ctx.varimp(True)])
        ctx.close()
    assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(*got))
    stages = [r["stage"] for r in abi.tuned_shapes() if (r["log2_n"], r["log2_ntree"], r["log2_p"]) == (9, 6, 7)]
    for stage in ("route", "route_leaf_order", "varimp_walk"):
        assert stages.count(stage) == 2, stages
