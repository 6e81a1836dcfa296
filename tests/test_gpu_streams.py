"""A context's own stream beside other streams' work, against the oracle."""
import numpy as np
import pytest

from rfx_b200 import synth

pytestmark = pytest.mark.gpu


def _forest(n=700, T=23):
    from rfx_b200 import abi

    X, y = synth.gaussian_classes(n, 6, 3, seed=n, mean_scale=1.0)
    return X, y, abi.grow_forest(X, y, T, 3, 1, nclass=3)


def test_new_context_while_the_default_stream_is_busy(built):
    """The first summaries of a context count from zero, whatever the default
    stream still holds when it is created."""
    import torch

    from oracle import oracle as orc
    from rfx_b200 import abi

    X, y, f = _forest()
    O = orc.analyse(X, y, f)
    want = orc.oob_summary(O["q_raw"], O["nout"], y)
    torch.cuda._sleep(100_000_000)  # about 50 ms
    ctx = abi.Context(0)
    ctx.load(f, X, y)
    ctx.route_oob()
    for _ in range(2):
        err, pred, proba = ctx.oob_summary()
        assert np.float32(err) == want[0]
        assert np.array_equal(pred, want[1]) and np.array_equal(proba, want[2])
    ctx.close()
