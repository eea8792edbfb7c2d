"""Batches whose units are shared out by weight against single searches: base sets
that end around the sixteenth tile, query sets that leave one or two tiles in their
last group, empty sets, and lists just below and above the size from which shares
are weighted (8 units per worker). Exact equality."""
import numpy as np
import pytest

import matching_sift_b200 as ms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na,nb,copies", [
    ((1, 256, 257, 512, 769), (1, 128, 2047, 2048, 2049), 1),   # below the rule
    ((700, 256, 300, 0, 1025), (2048, 2049, 4500, 700, 0), 12),
    ((513, 2000), (5000, 2176), 20),
])
def test_weighted_batch_equals_single_searches(cuda_device, na, nb, copies):
    import torch

    rng = np.random.default_rng(len(na) + copies)
    na, nb = np.tile(na, copies), np.tile(nb, copies)
    rng.shuffle(na)
    rng.shuffle(nb)
    q = torch.from_numpy(rng.integers(0, 200, (int(na.sum()), 128), dtype=np.uint8)).to(cuda_device)
    r = torch.from_numpy(rng.integers(0, 200, (int(nb.sum()), 128), dtype=np.uint8)).to(cuda_device)
    off = np.concatenate([[0], np.cumsum(nb)[:-1]])
    got = ms.match_batch(q, r, np.stack([na, nb, off], 1))
    qa = np.concatenate([[0], np.cumsum(na)])
    for p in range(len(na)):
        if not na[p]:
            continue
        want = ms.match(q[qa[p]:qa[p + 1]], r[off[p]:off[p] + nb[p]])
        for key in ("nn_idx", "nn_dist"):
            assert torch.equal(got[key][qa[p]:qa[p + 1]], want[key]), (p, na[p], nb[p], key)
