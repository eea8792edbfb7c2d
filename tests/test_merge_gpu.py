"""The merge of partial top-2 lists at every number of threads per query row:
2 lists (one thread), 6 (8 threads), 34 and 148 (32 threads), row counts on
both sides of a block's 32 rows, ties across lists. Integers: bit-exact."""
import numpy as np
import pytest

import matching_sift_b200 as ms
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q_n,r_n", [(1, 1), (31, 100), (257, 128), (33, 300), (100, 17 * 128 - 5), (1, 74 * 128 + 1),
                                     (65, 74 * 128), (545, 40 * 128 + 3)])
def test_merge_lanes_equal_oracle(cuda_device, q_n, r_n):
    import torch

    rng = np.random.default_rng([q_n, r_n])
    r = rng.integers(0, 4, (r_n, 128)).astype(np.uint8)
    half = r_n // 2
    r[r_n - half:] = r[:half]  # rows twice: ties between lists of different workers
    q = rng.integers(0, 4, (q_n, 128)).astype(np.uint8)
    q[0] = r[-1]
    out = ms.match(torch.from_numpy(q).to(cuda_device), torch.from_numpy(r).to(cuda_device), threshold=0.9)
    dist, idx = oracle.brute_2nn_u8(q, r)
    np.testing.assert_array_equal(out["nn_idx"].cpu().numpy(), idx)
    present = idx >= 0
    got = out["nn_dist"].cpu().numpy()
    np.testing.assert_array_equal(got[present].astype(np.int64), dist[present])
    assert (got[~present] == np.finfo(np.float32).max).all()
