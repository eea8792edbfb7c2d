"""The first units of an FP16 search (packed exact keys from float accumulators)
where they can go wrong: base sets that end inside a chunk, a tile and past the
first units, extreme keys, ties, scaled values, plain dot products. The same
integers as u8 rows are the oracle: equal indices, distances equal up to the
power-of-two scale, both exactly."""
import pytest

import matching_sift_b200 as ms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r_n", [1, 15, 16, 17, 127, 129, 1023, 1025, 74 * 128 * 3 + 5, 74 * 128 * 9 + 100])
@pytest.mark.parametrize("metric", [ms.METRIC_L2, ms.METRIC_DOT])
def test_equals_u8(cuda_device, r_n, metric):
    import torch

    g = torch.Generator(device=cuda_device).manual_seed(r_n)
    q = torch.randint(0, 256, (130, 128), generator=g, device=cuda_device, dtype=torch.uint8)
    r = torch.randint(0, 256, (r_n, 128), generator=g, device=cuda_device, dtype=torch.uint8)
    q[0], q[1] = 0, 255
    r[0] = 255                       # the largest norm and product
    r[r_n // 2] = 0
    r[r_n - 1] = q[2]                # an exact match in the last row
    if r_n > 40:
        r[33:37] = r[5]              # ties within and across chunks
    want = ms.match(q, r, metric=metric)
    for scale in (1.0, 2.0 ** -9):
        got = ms.match(q.half() * scale, r.half() * scale, metric=metric)
        assert torch.equal(got["nn_idx"], want["nn_idx"])
        d = want["nn_dist"].clone()
        d[d < 3e38] *= scale * scale
        assert torch.equal(got["nn_dist"], d)
