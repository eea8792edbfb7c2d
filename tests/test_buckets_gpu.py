"""Bucket tables at the edges of their launches (chunks of 8,192 points, blocks
of 1,024 bins): one point, full and partial chunks, every point in one bin, one
bit, codes longer than the bucket bits. Compared as sets with a numpy grouping."""
import numpy as np
import pytest

import matching_sift_b200 as ms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,k,kind", [(1, 1, 16, "spread"), (8191, 2, 1, "spread"), (8192, 1, 10, "spread"),
                                        (8193, 3, 12, "crowd"), (20000, 2, 16, "one"), (100003, 1, 20, "crowd"),
                                        (3000000, 1, 16, "crowd"), (4097, 8, 32, "spread")])
def test_bucket_tables(cuda_device, n, L, k, kind):
    import torch

    rng = np.random.default_rng([n, k])
    codes = rng.integers(0, 1 << k, (L, n), dtype=np.uint64).astype(np.uint32)
    if kind == "one":
        codes[:] = (1 << k) - 1
    elif kind == "crowd":
        codes[:, rng.random(n) < 0.6] = 5 << max(0, k - 16)
    start, order, ocode = (x.cpu().numpy() for x in ms.lsh_buckets(
        torch.from_numpy(codes.view(np.int32)).to(cuda_device), k))
    assert ms.stream_status() == ms.SIFT_OK
    top = min(k, 16)
    for t in range(L):
        bins = (codes[t] >> (k - top)).astype(np.int64)
        np.testing.assert_array_equal(start[t], np.concatenate([[0], np.cumsum(np.bincount(bins, minlength=1 << top))]))
        np.testing.assert_array_equal(np.sort(order[t]), np.arange(n))
        np.testing.assert_array_equal(ocode[t].view(np.uint32), codes[t][order[t]])
        np.testing.assert_array_equal(bins[order[t]], np.repeat(np.arange(1 << top), np.diff(start[t])))
