"""The leaf-list kernel at the edges of its batches (256 samples per warp, 2,048
per round), with one key shared by most lanes, few keys, and many, and left-out
samples, through the allocation-free entry point against the oracle (exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 255, 256, 257, 2047, 2048, 2049, 4100])
@pytest.mark.parametrize("leaves", ["one", "few", "many"])
def test_leaf_lists(built, n, leaves):
    import torch

    from oracle import oracle as orc
    from rfx_b200 import abi

    rng = np.random.default_rng(n)
    T = 3
    most = {"one": 1, "few": min(n, 5), "many": n}[leaves]
    leaf = rng.integers(0, most, (T, n)).astype(np.int32)
    leaf[0, rng.random(n) < 0.5] = -1
    leaf[1, rng.random(n) < 0.6] = most - 1
    inbag = (rng.random((T, n)) < 0.63).astype(np.uint8)
    want, bad = orc.pairs_from_leaves(leaf, inbag, most)
    assert bad == 0
    S = torch.zeros(n * (n + 1) // 2, dtype=torch.int32, device="cuda")
    abi.pair_counts_noalloc(torch.from_numpy(leaf).cuda(), torch.from_numpy(inbag).cuda(), n, T, most, S)
    assert np.array_equal(S.cpu().numpy(), want)
