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


@pytest.mark.parametrize("casewise", [False, True])
def test_calls_complete_on_return(built, casewise):
    """Results in device memory are there when these calls return: nothing is
    left on the context's stream, and a stream that does not wait for it reads
    the oracle's values."""
    import torch

    from oracle import oracle as orc
    from rfx_b200 import abi

    n = 1500
    X, y, f = _forest(n, 60)
    O = orc.analyse(X, y, f, casewise=casewise, want_cw=casewise, want_leaf=True)
    ctx = abi.Context(0, use_casewise=casewise)
    ctx.load(f, X, y)
    own = torch.cuda.ExternalStream(ctx.stream)
    L = n * (n + 1) // 2
    new = lambda k, t: torch.full((k,), -1, dtype=t, device="cuda")
    err, pred, proba = new(1, torch.float32), new(n, torch.int32), new(3 * n, torch.float32)
    S, P, q, nout = new(L, torch.float64), new(L, torch.float64), new(3 * n, torch.float32), new(n, torch.int32)
    torch.cuda.synchronize()
    want = orc.oob_summary(O["q_raw"], O["nout"], y)
    ctx.oob_summary(err, pred, proba)
    assert own.query()
    assert np.array_equal(pred.cpu().numpy(), want[1]) and np.array_equal(proba.cpu().numpy(), want[2].ravel())
    ctx.proximity_upper_f64(S)
    assert own.query()
    assert np.array_equal(S.cpu().numpy(), O["Sd"] if casewise else O["S"].astype(np.float64))
    ctx.proximity_rfgap(P)
    assert own.query()
    assert np.array_equal(P.cpu().numpy(), orc.rfgap(f.nin, O["leaf"])[np.triu_indices(n)])
    if casewise:
        ctx.casewise_votes(q, nout)
        assert own.query()
        assert np.array_equal(q.cpu().numpy().reshape(n, 3), O["q_raw"])
        assert np.array_equal(nout.cpu().numpy(), O["nout"])
    ctx.close()
