"""The packed top-2 of batches at the ends of its range: the largest keys of
either sign (all-255 and all-0 rows), ties within and across tiles, base sets
that end on every kind of chunk edge, stray rows of the next problem past a
set's end. Integers against the oracle: bit-exact."""
import numpy as np
import pytest

import matching_sift_b200 as ms
import oracle

pytestmark = pytest.mark.gpu


def _check(cuda_device, sets_q, sets_r, shape):
    import torch

    q, r = np.concatenate(sets_q), np.concatenate(sets_r)
    pairs, off = [], 0
    for a, b in zip(sets_q, sets_r):
        pairs.append([len(a), len(b), off])
        off += len(b)
    qd, rd = torch.from_numpy(q).to(cuda_device), torch.from_numpy(r).to(cuda_device)
    plan = ms.BatchPlan(qd, rd, pairs, tune=False, shape=shape)
    for out in (plan.run(), ms.match_batch(qd, rd, pairs)):
        idx, dist = out["nn_idx"].cpu().numpy(), out["nn_dist"].cpu().numpy()
        at = 0
        for a, b in zip(sets_q, sets_r):
            d, i = oracle.brute_2nn_u8(a, b)
            np.testing.assert_array_equal(idx[at:at + len(a)], i)
            np.testing.assert_array_equal(dist[at:at + len(a)][i >= 0].astype(np.int64), d[i >= 0])
            at += len(a)


@pytest.mark.parametrize("shape", [0, 1, 2])
def test_extreme_keys_and_ties(cuda_device, shape):
    rng = np.random.default_rng(shape)
    ends = np.zeros((300, 128), np.uint8)
    ends[::3] = 255
    ends[1::7, :64] = 255
    q = np.concatenate([ends[:5], rng.integers(0, 2, (40, 128)).astype(np.uint8) * 255])
    flat = np.full((257, 128), 255, np.uint8)
    _check(cuda_device, [q, q[:1], q, q[5:]], [ends, flat, flat[:2], np.zeros((130, 128), np.uint8)], shape)


@pytest.mark.parametrize("shape", [0, 2])
def test_base_set_ends(cuda_device, shape):
    rng = np.random.default_rng(7)
    sizes = [1, 2, 15, 16, 17, 31, 33, 112, 113, 127, 128, 129, 255, 257, 640, 1025, 2047, 2049, 2190]
    sets_r = [rng.integers(0, 6, (n, 128)).astype(np.uint8) for n in sizes]
    # Queries equal rows of the NEXT base set: what lies past a set's end must not be found.
    sets_q = [np.concatenate([sets_r[(k + 1) % len(sizes)][:3], sets_r[k][-1:], rng.integers(0, 6, (1 + 60 * k, 128))]).astype(np.uint8)
              for k in range(len(sizes))]
    _check(cuda_device, sets_q, sets_r, shape)
