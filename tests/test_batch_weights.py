"""How a batch's units are shared out by weight (no GPU): a restatement of the rule
over random lists -- every unit has one owner, no worker of a range is without a
unit, the owner of a unit follows from its weight position -- and the library's
list count per group (partial lists that the merge reads) against it."""
import numpy as np
import pytest

import matching_sift_b200 as ms

BN, DENSE_TILES = 128, 16


def _weights(na, nb, group):
    """Weights of a problem's units in order: 6 in the first 16 tiles, 5 after, one less where at most
    256 rows of a group of 512 are left."""
    t = -(-nb // BN)
    full = np.where(np.arange(t) < DENSE_TILES, 6, 5)
    out = []
    for g in range(-(-na // group)):
        out.append(full - (1 if group > 256 and na - g * group <= 256 else 0))
    return out


@pytest.mark.parametrize("qpt", [1, 2])
@pytest.mark.parametrize("workers", [1, 7, 74])
@pytest.mark.parametrize("hi", [700, 9000])
def test_weighted_shares(qpt, workers, hi):
    rng = np.random.default_rng(workers + hi)
    for _ in range(8):
        n = int(rng.integers(1, 90))
        na, nb = rng.integers(0, hi, n), rng.integers(0, hi, n)
        na[rng.random(n) < 0.2] = rng.choice([256, 257, 512, 768, 769])
        nb[rng.random(n) < 0.2] = rng.choice([1, 2047, 2048, 2049])
        nb[rng.random(n) < 0.1] = 0
        pairs = np.stack([na, nb, np.concatenate([[0], np.cumsum(nb)[:-1]])], 1)
        got = ms.batch_describe(pairs, int(nb.sum()), qpt=qpt, workers=workers)
        groups = [g for a, b in zip(na, nb) for g in _weights(int(a), int(b), 256 * qpt) if len(g)]
        units = sum(len(g) for g in groups)
        grid = min(workers, units)
        assert got["units"] == units and got["grid"] == grid
        if not grid:
            continue
        w = np.concatenate(groups)
        if units < 8 * grid:
            w = np.ones_like(w)
        begin = np.concatenate([[0], np.cumsum(w)]).astype(int)
        total = int(begin[-1])
        edges = [c * total // grid for c in range(grid + 1)]
        owner = np.searchsorted(edges, begin[:-1], side="right") - 1
        assert set(owner) == set(range(grid)) and (np.diff(owner) >= 0).all()
        assert (owner == ((begin[:-1] + 1) * grid - 1) // total).all()
        ends = np.cumsum([len(g) for g in groups])
        lists = owner[ends - 1] - owner[ends - [len(g) for g in groups]] + 1
        assert got["max_splits"] == lists.max()
