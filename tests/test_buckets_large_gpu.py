"""Bucket tables of 2^31 - 1 points, the most that the entry point takes (26 GB of
codes, ids and grouped codes)."""
import pytest

import matching_sift_b200 as ms

pytestmark = pytest.mark.gpu


def test_largest_table(cuda_device):
    import torch

    if torch.cuda.mem_get_info(cuda_device)[0] < 60 << 30:
        pytest.skip("needs 60 GB of free device memory")
    n, k, step = (1 << 31) - 1, 8, 1 << 27
    codes = torch.empty((1, n), dtype=torch.int32, device=cuda_device).random_(0, 1 << k)
    start, order, ocode = ms.lsh_buckets(codes, k)
    assert ms.stream_status() == ms.SIFT_OK
    counts = torch.zeros(1 << k, dtype=torch.int64, device=cuda_device)
    seen = torch.zeros(n, dtype=torch.bool, device=cuda_device)
    for a in range(0, n, step):
        b = min(n, a + step)
        counts += torch.bincount(codes[0, a:b], minlength=1 << k)
        ids = order[0, a:b].long()
        assert torch.equal(codes[0][ids], ocode[0, a:b])
        seen[ids] = True
        e = min(n, b + 1)
        assert bool((ocode[0, a + 1:e] >= ocode[0, a:e - 1]).all())
    assert bool(seen.all())
    assert torch.equal(start[0].long(), torch.cat([counts.new_zeros(1), counts.cumsum(0)]))
