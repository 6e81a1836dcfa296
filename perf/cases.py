"""Timed cases of the post-growth analysis path.

Each case is a dict of plain values; ``kind`` names the entry points it calls:

votes        OOB routing, votes, error, predictions and probabilities
analysis     everything a small fit reports: votes, pair counts, proximity,
             importance (overall and local) and the 3-D MDS of the proximity
counts       exact INT32 pair counts, packed upper triangle
importance   permutation importance, overall and local
predict      votes of new rows
finishprox   normalised proximity from pair counts
casewise     case-wise weighted votes, FP64 pair sums, proximity, importance
rfgap        RF-GAP proximity
product      one product M V of the low-rank operator (M = P - I)
factors      low-rank factors, their quantised form, MDS and outlier scores
batch        several uneven forests replayed as one captured CUDA graph

A user's program holds a loaded forest before these calls, so `prepare` grows
one on seeded synthetic data and loads it.  A few dozen trees are grown; larger
forests repeat them, every copy with a bootstrap sample of its own.
"""
import ctypes
import dataclasses

import numpy as np
import torch

from rfx_b200 import abi, synth

GROWN = 1_600_000  # rows x trees grown on the host; further trees are copies with their own bags


def listed():
    return [
        # the smallest call: a toy forest, where launches and latency count
        dict(name="votes_n300_t60", kind="votes", data="gauss", n=300, p=8, c=3, trees=60, mtry=3, nodesize=1),
        # everything a fit on a small table reports
        dict(name="analysis_n2000_t500", kind="analysis", data="gauss", n=2000, p=13, c=3, trees=500, mtry=3,
             nodesize=1),
        # the pair counts of a large mixed-type table: the dominant stage of an exact analysis
        dict(name="counts_n50000_t1000", kind="counts", data="cover", n=50000, p=54, c=7, trees=1000, mtry=7,
             nodesize=1),
        # its permutation importance, overall and local
        dict(name="importance_n50000_t1000", kind="importance", data="cover", n=50000, p=54, c=7, trees=1000, mtry=7,
             nodesize=1),
        # serving: a few rows through a forest
        dict(name="predict_m61_t1000", kind="predict", data="cover", n=20000, p=54, c=7, trees=1000, mtry=7,
             nodesize=1, m=61),
        # scoring a whole test set
        dict(name="predict_m50000_t1000", kind="predict", data="cover", n=20000, p=54, c=7, trees=1000, mtry=7,
             nodesize=1, m=50000),
        # the full float32 proximity matrix of an odd number of rows
        dict(name="finishprox_n30001", kind="finishprox", data="gauss", n=30001, p=8, c=3, trees=200, mtry=3,
             nodesize=5, full=True),
        # case-wise weighting: weighted votes, FP64 pair sums, proximity and importance
        dict(name="casewise_n3001_t300", kind="casewise", data="gauss", n=3001, p=20, c=4, trees=300, mtry=4,
             nodesize=1),
        # RF-GAP proximity
        dict(name="rfgap_n5000_t500", kind="rfgap", data="gauss", n=5000, p=16, c=4, trees=500, mtry=4, nodesize=1),
        # one FP32 product of the low-rank operator, the step that a user's own solver repeats
        dict(name="product_n100000_t500", kind="product", data="gauss", n=100000, p=32, c=4, trees=500, mtry=5,
             nodesize=5, width=48, precision=0),
        # rank-64 factors of a mixed-type table in the BF16 form, INT8 storage, MDS and outlier scores
        dict(name="factors_n50000_t1000", kind="factors", data="cover", n=50000, p=54, c=7, trees=1000, mtry=7,
             nodesize=1, rank=64, precision=1, fmt=1),
        # several uneven forests at once
        dict(name="batch_6x20000", kind="batch", data="gauss", n=20000, p=40, c=8, trees=300, mtry=6, nodesize=1,
             forests=6),
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread over the logarithm."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["votes", "analysis", "counts", "importance", "predict", "finishprox", "casewise", "rfgap",
                       "product", "factors", "batch"])
    data = "cover" if kind in ("counts", "importance", "predict", "factors", "votes") and rng.random() < 0.5 \
        else "gauss"
    lo, hi = {"votes": (200, 50000), "analysis": (300, 3000), "counts": (700, 50000), "importance": (700, 50000),
              "predict": (500, 20000), "finishprox": (400, 30000), "casewise": (300, 3000), "rfgap": (300, 5000),
              "product": (3000, 100000), "factors": (2000, 50000), "batch": (1500, 20000)}[kind]
    most = {"analysis": 500, "casewise": 300, "rfgap": 500, "product": 500, "batch": 300, "finishprox": 200}
    p = 54 if data == "cover" else _log(rng, 4, 40 if kind in ("casewise", "analysis", "batch") else 100)
    case = dict(kind=kind, data=data, n=_log(rng, lo, hi), p=p, c=7 if data == "cover" else rng.randint(2, 10),
                trees=_log(rng, 40, most.get(kind, 1000)), mtry=max(1, int(p ** 0.5)),
                nodesize=5 if kind in ("product", "finishprox") else rng.choice([1, 1, 5]))
    if kind == "predict":
        case["m"] = _log(rng, 1, 50000)
    if kind == "finishprox":
        case["full"] = rng.random() < 0.7
    if kind == "product":
        case.update(width=8 * rng.randint(1, 10), precision=rng.choice([0, 0, 1, 3]))
    if kind == "factors":
        case.update(rank=rng.choice([16, 32, 32, 64, 64]), precision=rng.choice([0, 1, 3]),
                    fmt=rng.choice([1, 2, 3, 4]))
    if kind == "batch":
        case["forests"] = rng.randint(2, 6)
    return case


# --- inputs -----------------------------------------------------------------


def _table(case, n, seed):
    if case["data"] == "cover":
        return synth.mixed_cover(n, seed=seed)
    return synth.gaussian_classes(n, case["p"], case["c"], seed=seed, mean_scale=1.0)


def _forest(case, seed):
    """Data and forest: (rows to predict, forest with its node counts, device arrays in the padded layout, maxnode)."""
    n, T = case["n"], case["trees"]
    X, y = _table(case, n + case.get("m", 0), seed)
    X, y, new = X[:n], y[:n], X[n:]
    cat = synth.detect_categorical(X) if case["data"] == "cover" else None
    grown = min(T, max(16, GROWN // n))
    f = abi.grow_forest(X, y, grown, case["mtry"], case["nodesize"], iseed=seed % 100000 + 1, nclass=case["c"],
                        cat=cat)
    most = int(f.nnode.max())
    tree = np.arange(T) % grown

    def padded(a, k=1):
        out = np.zeros((grown, k * most), a.dtype)
        for t in range(grown):
            out[t, : k * f.nnode[t]] = a[k * f.offs[t]: k * f.offs[t + 1]]
        return torch.from_numpy(out).cuda()[torch.from_numpy(tree).cuda()].contiguous()

    dev = {k: padded(getattr(f, k)) for k in ("nodestatus", "bestvar", "xbestsplit", "nodeclass")}
    dev["treemap"] = padded(f.treemap, 2)
    if grown == T:
        dev["nin"] = torch.from_numpy(f.nin).cuda()
    else:
        g = torch.Generator(device="cuda").manual_seed(seed)
        at = torch.randint(n, (T, n), generator=g, device="cuda")
        at += torch.arange(T, device="cuda")[:, None] * n
        dev["nin"] = torch.bincount(at.view(-1), minlength=T * n).view(T, n).to(torch.int32)
    dev.update(X=torch.from_numpy(X).cuda(), y=torch.from_numpy(y).cuda(), cat=torch.from_numpy(f.cat).cuda())
    return new, dataclasses.replace(f, nnode=f.nnode[tree]), dev, most


def _load(case, seed, casewise=False):
    new, f, dev, most = _forest(case, seed)
    ctx = abi.Context(0, use_casewise=casewise)
    torch.cuda.synchronize()  # the context works on a stream of its own
    ctx.load_device(f, dev, most)
    return ctx, new


def _new(*shape, dtype=torch.float32):
    return torch.zeros(shape, dtype=dtype, device="cuda")


def _counts(case, seed):
    """Pair counts as a finishprox caller has them: mostly 0, a few, some large; zero diagonal."""
    n = case["n"]
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    S = torch.rand(n * (n + 1) // 2, generator=g, device="cuda")
    S = (S ** 8 * case["trees"]).to(torch.int32)
    i = torch.arange(n, device="cuda")
    S[i * n - i * (i - 1) // 2] = 0
    return S


def _uneven(case):
    """The batch's forests: sizes falling from the case's."""
    for q in range(case["forests"]):
        yield dict(case, n=max(200, int(case["n"] / (1 + 0.45 * q))), p=max(2, case["p"] - 5 * q),
                   mtry=max(1, case["mtry"] - q // 2), c=max(2, case["c"] - q))


def prepare(case, seed):
    kind, n, p, c = case["kind"], case["n"], case["p"], case["c"]
    if kind == "batch":
        items = []
        for q, sub in enumerate(_uneven(case)):
            m, k = sub["n"], sub["p"]
            items.append(dict(ctx=_load(sub, seed + 1000 * q)[0], impn=True, votes=_new(m, sub["c"], dtype=torch.int32),
                              nout=_new(m, dtype=torch.int32), oob_error=_new(1), oob_pred=_new(m, dtype=torch.int32),
                              S=_new(m * (m + 1) // 2, dtype=torch.int32), avimp=_new(k), sqsd=_new(k), qimp=_new(m),
                              qimpm=_new(m * k)))
        torch.cuda.synchronize()
        return dict(kind=kind, items=items, graph=abi.BatchGraph(items))
    ctx, new = _load(case, seed, casewise=kind == "casewise")
    s = dict(kind=kind, ctx=ctx)
    upper = n * (n + 1) // 2
    if kind in ("votes", "analysis", "casewise"):
        s.update(q=_new(n, c, dtype=torch.float32 if kind == "casewise" else torch.int32),
                 nout=_new(n, dtype=torch.int32), err=_new(1), pred=_new(n, dtype=torch.int32), proba=_new(n, c))
    if kind in ("analysis", "counts"):
        s["S"] = _new(upper, dtype=torch.int32)
    if kind in ("casewise", "rfgap"):
        s["S"] = _new(upper, dtype=torch.float64)
    if kind in ("analysis", "casewise"):
        s["P"] = _new(n, n)
    if kind in ("analysis", "casewise", "importance"):
        s.update(avimp=_new(p), sqsd=_new(p), qimp=_new(n), qimpm=_new(n * p), local=_new(n, p))
    if kind == "analysis":
        s["coords"] = _new(n, 3, dtype=torch.float64)
    if kind == "finishprox":
        s.update(S=_counts(case, seed), full=case["full"], P=_new(n, n) if case["full"] else _new(upper))
    if kind == "predict":
        s.update(X=torch.from_numpy(np.ascontiguousarray(new)).cuda(), votes=_new(case["m"], c, dtype=torch.int32))
    if kind == "product":
        g = torch.Generator(device="cuda").manual_seed(seed + 2)
        s.update(V=torch.randn(n, case["width"], generator=g, device="cuda"), MV=_new(n, case["width"]),
                 width=case["width"], precision=case["precision"])
    if kind == "factors":
        s.update(A=_new(n, case["rank"]), rank=case["rank"], precision=case["precision"], fmt=case["fmt"])
    torch.cuda.synchronize()
    return s


# --- one pass ---------------------------------------------------------------


def _importance(ctx, s):
    ctx.varimp(True, s["avimp"], s["sqsd"], s["qimp"], s["qimpm"])
    ctx.localimp(s["qimp"], s["qimpm"], s["local"])
    return {k: s[k] for k in ("avimp", "sqsd", "qimp", "qimpm", "local")}


def _summary(ctx, s):
    ctx.oob_summary(s["err"], s["pred"], s["proba"])
    return {k: s[k] for k in ("q", "nout", "err", "pred", "proba")}


def run(s):
    kind = s["kind"]
    if kind == "batch":
        s["graph"].launch()
        return [{k: v for k, v in it.items() if k not in ("ctx", "impn")} for it in s["items"]]
    ctx = s["ctx"]
    if kind == "votes":
        ctx.route_oob(s["q"], s["nout"])
        return _summary(ctx, s)
    if kind == "analysis":
        ctx.route_oob(s["q"], s["nout"])
        out = _summary(ctx, s)
        ctx.proximity_upper(s["S"])
        ctx.finishprox(s["S"], s["P"], full=True)
        out.update(_importance(ctx, s), S=s["S"], P=s["P"])
        out["coords"], out["evals"] = ctx.mds3d_full(s["P"], s["coords"])
        return out
    if kind == "counts":
        return ctx.proximity_upper(s["S"])
    if kind == "importance":
        return _importance(ctx, s)
    if kind == "predict":
        return ctx.predict_votes(s["X"], s["votes"])
    if kind == "finishprox":
        return ctx.finishprox(s["S"], s["P"], full=s["full"])
    if kind == "casewise":
        ctx.casewise_votes(s["q"], s["nout"])
        out = _summary(ctx, s)
        ctx.proximity_upper_f64(s["S"])
        ctx.finishprox_f64(s["S"], s["P"], full=True)
        out.update(_importance(ctx, s), S=s["S"], P=s["P"])
        return out
    if kind == "rfgap":
        return ctx.proximity_rfgap(s["S"])
    if kind == "product":
        V, MV = ctypes.c_void_p(s["V"].data_ptr()), ctypes.c_void_p(s["MV"].data_ptr())
        status = abi.lib().rfx_lowrank_operator(ctx._h, s["width"], s["precision"], V, MV)
        if status != abi.RFX_OK:
            raise abi.RfxError(status, abi.lib().rfx_last_error().decode())
        return s["MV"]
    A, evals = ctx.lowrank(s["rank"], precision=s["precision"], A=s["A"])
    codes, scales = ctx.lowrank_quantize(s["fmt"])
    coords, ev = ctx.mds_from_factors(3, use_quantized=True, precision=s["precision"])
    return dict(A=A, evals=evals, codes=codes, scales=scales, coords=coords, mds_evals=ev,
                scores=ctx.outlier_scores(use_quantized=True))


# --- what a pass cannot do without --------------------------------------------


def work(case):
    if case["kind"] == "batch":
        parts = [work(dict(sub, kind=k)) for sub in _uneven(case) for k in ("counts", "importance")]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    kind, n, p, T, c = case["kind"], case["n"], case["p"], case["trees"], case["c"]
    nodes = T * max(1.0, 0.35 * n / case["nodesize"])  # about what these tables grow
    base = 4.0 * n * p + 16 * nodes + T * n  # the rows, the trees and the bag flags, once
    upper = n * (n + 1) / 2
    votes = 4.0 * n * (2 * c + 2)
    importance = 4.0 * (n + 2 * n * p + 2 * p)
    b, fl = base, 0.0
    if kind == "votes":
        b += votes
    elif kind == "analysis":
        b += votes + importance + 2 * 4 * upper + 2 * 4.0 * n * n + 8 * 3 * n
        fl = 2.0 * n * n * 3
    elif kind == "counts":
        b += 4 * upper
    elif kind == "importance":
        b += importance
    elif kind == "predict":
        b = 4.0 * case["m"] * (p + c) + 16 * min(nodes, case["m"] * T * 16.0)  # a walk passes some 16 nodes
    elif kind == "finishprox":
        b = 4 * upper + 4.0 * (n * n if case["full"] else upper)
    elif kind == "casewise":
        b += 3.0 * T * n + votes + importance + 2 * 8 * upper + 4.0 * n * n
    elif kind == "rfgap":
        b += 3.0 * T * n + 8 * upper
    else:
        w = case["width"] if kind == "product" else case["rank"] + 16
        b += 3 * 4.0 * n * w + 4.0 * T * n
        # every (tree, row) adds its 2w values to a leaf's sum and one leaf's sum to its own
        fl = 4.0 * T * n * w * (1 if kind == "product" else 3)
        if kind == "factors":
            b += (4 + 1) * n * case["rank"] + 8 * 3 * n + 4 * n
    return {"bytes": float(b), "flops": float(fl)}


# --- 64-bit values --------------------------------------------------------------


def _leaves(dev):
    """Node that every (tree, row) ends on, numeric splits: (T, n).  An out-of-bag walk gives up after 999 splits
    and counts as the root's (large tables grow a few chains that deep)."""
    T, n = dev["nin"].shape
    most = dev["nodestatus"].shape[1]
    flat = {k: dev[k].reshape(-1) for k in ("nodestatus", "bestvar", "xbestsplit")}
    kids = dev["treemap"].reshape(-1, 2)
    node = (torch.arange(T, device="cuda")[:, None] * most).expand(T, n).reshape(-1).clone()
    oob = (dev["nin"] == 0).view(-1)
    live = torch.arange(T * n, device="cuda")
    step = 0
    while True:
        live = live[flat["nodestatus"][node[live]] == 1]
        if not live.numel():
            break
        at = node[live]
        step += 1
        if step >= 1000:
            node[live] = torch.where(oob[live], at // most * most, at)
            live = live[~oob[live]]
            at = node[live]
        x = dev["X"][live % n, flat["bestvar"][at].long()]
        node[live] = at // most * most + kids[at, (x > flat["xbestsplit"][at]).long()]
    return node.view(T, n) - torch.arange(T, device="cuda")[:, None] * most


def _exact_votes(case, dev, node, weight=None):
    """Votes of the out-of-bag trees and their summary; weight: (T, nodes) or None."""
    n, c = case["n"], case["c"]
    q = torch.zeros(n * c, dtype=torch.float64, device="cuda")
    row = torch.arange(n, device="cuda")
    for t in range(node.shape[0]):
        oob = dev["nin"][t] == 0
        w = torch.ones(n, dtype=torch.float64, device="cuda") if weight is None else weight[t][node[t]]
        q.index_add_(0, (row * c + dev["nodeclass"][t][node[t]])[oob], w[oob])
    q = q.view(n, c)
    some = (dev["nin"] == 0).any(0)
    total = q.sum(1, keepdim=True)
    pred = c - 1 - q.flip(1).argmax(1)
    right = ((pred == dev["y"]) & some).sum().double()
    err = (1 - right / some.sum().double()).view(1)
    proba = torch.where(total > 0, q / total.clamp(min=1e-300), torch.full_like(q, 1.0 / c))
    return q, err, proba


def _pair_sums(dev, node, pair):
    """Sum over trees of pair(t): weights of the out-of-bag rows (n) and of the in-bag columns (n) that
    share a leaf; the whole n x n matrix."""
    T, n = node.shape
    C = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    for t in range(T):
        leaf = dev["nodestatus"][t][node[t]] == -1
        rows = (leaf & (dev["nin"][t] == 0)).nonzero().view(-1)
        cols = (leaf & (dev["nin"][t] > 0)).nonzero().view(-1)
        same = node[t][rows][:, None] == node[t][cols][None, :]
        i, j = same.nonzero(as_tuple=True)
        C.view(-1).index_add_(0, rows[i] * n + cols[j], pair(t)[cols[j]])
    return C


def _leaf_mass(dev, node, t, values):
    mass = torch.zeros(dev["nodestatus"].shape[1], dtype=torch.float64, device="cuda")
    return mass.index_add_(0, node[t], values)


def _shares(dev, node):
    """t -> bootstrap multiplicity over its leaf's total, per row."""
    def share(t):
        m = dev["nin"][t].double()
        return m / _leaf_mass(dev, node, t, m)[node[t]].clamp(min=1e-300)
    return share


def _proximity(S, nout):
    inv = torch.where(nout > 0, 1.0 / nout.clamp(min=1).double(), torch.ones_like(nout, dtype=torch.float64))
    P = 0.5 * (S / 2 * inv[:, None] + S / 2 * inv[None, :])
    P.fill_diagonal_(1.0)
    return P


def _packed(M):
    n = M.shape[0]
    return M[torch.ones(n, n, dtype=torch.bool, device="cuda").triu()]


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if case["data"] == "cover" or kind not in ("votes", "analysis", "finishprox", "casewise", "rfgap", "product"):
        return None  # whole numbers, or values that take too long (importance) or hang on a random sketch (factors)
    _, _, dev, _ = _forest(case, seed)
    nout = 2 * (dev["nin"] == 0).sum(0)
    if kind == "finishprox":
        S = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        S[torch.ones(n, n, dtype=torch.bool, device="cuda").triu()] = _counts(case, seed).double()
        P = _proximity(S + S.t(), nout)
        return P if case["full"] else _packed(P)
    node = _leaves(dev)
    if kind == "votes":
        _, err, proba = _exact_votes(case, dev, node)
        return dict(q=None, nout=None, err=err, pred=None, proba=proba)
    if kind == "rfgap":
        C = _pair_sums(dev, node, _shares(dev, node))
        oob = (nout / 2).double()
        C = torch.where(oob[:, None] > 0, C / oob.clamp(min=1)[:, None], C)
        P = (C + C.t()) / 2
        P.diagonal().copy_((nout == 0).double())
        return _packed(P)
    if kind == "product":
        inv = torch.where(nout > 0, 1.0 / nout.clamp(min=1).double(), torch.ones(n, dtype=torch.float64, device="cuda"))
        g = torch.Generator(device="cuda").manual_seed(seed + 2)
        V = torch.randn(n, case["width"], generator=g, device="cuda").double()
        Z = torch.cat([V, V * inv[:, None]], 1)
        Y = torch.zeros_like(Z)
        for t in range(case["trees"]):
            key = 2 * node[t] + (dev["nin"][t] > 0)
            G = torch.zeros(2 * dev["nodestatus"].shape[1], Z.shape[1], dtype=torch.float64, device="cuda")
            keep = dev["nodestatus"][t][node[t]] == -1
            G.index_add_(0, key[keep], Z[keep])
            Y[keep] += G[(key ^ 1)[keep]]
        return 0.25 * (inv[:, None] * Y[:, : case["width"]] + Y[:, case["width"]:])
    out = dict.fromkeys(("q", "nout", "err", "pred", "proba", "avimp", "sqsd", "qimp", "qimpm", "local", "S", "P"))
    if kind == "analysis":
        out.update(coords=None, evals=None)
        _, out["err"], out["proba"] = _exact_votes(case, dev, node)
        ones = torch.ones(n, dtype=torch.float64, device="cuda")
        C = _pair_sums(dev, node, lambda t: ones)
        out["P"] = _proximity(C + C.t(), nout)
        return out
    weight = torch.stack([_leaf_mass(dev, node, t, dev["nin"][t].double()) /
                          _leaf_mass(dev, node, t, (dev["nin"][t] > 0).double()).clamp(min=1)
                          for t in range(case["trees"])])
    out["q"], out["err"], out["proba"] = _exact_votes(case, dev, node, weight)
    C = _pair_sums(dev, node, _shares(dev, node))
    out["P"] = _proximity(C + C.t(), nout)
    out["S"] = _packed((C + C.t()).fill_diagonal_(0.0))
    return out
