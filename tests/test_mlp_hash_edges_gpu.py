"""Learned-hash inference at the edges of its tile pipeline: one row, partial
tiles, one, two, three and more tiles per block, 1 to 32 bits. z against FP64
within the inference test's 5e-3 (BF16 hidden values), codes equal wherever |z|
exceeds that, and a row's result independent of how many rows are hashed."""
import numpy as np
import pytest

import matching_sift_b200 as ms
from matching_sift_b200 import datagen
from oracle import learned_hash as lh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 7, 32])
def test_hash_at_tile_edges(cuda_device, k):
    import torch

    p = lh.init_params(k, seed=k)
    model = ms.MlpHash.from_params(torch.from_numpy(p).to(cuda_device), k)
    x = datagen.make_base(148 * 128 * 3 + 77, seed=k)
    xd = torch.from_numpy(x).to(cuda_device)
    all_codes, all_z = model.hash(xd, with_z=True)
    _, z = lh.forward(p, x[:3000], k)
    got = all_z[:3000].cpu().numpy().astype(np.float64)
    tol = 5e-3 * max(1.0, np.abs(z).max())
    assert np.abs(got - z).max() < tol
    bits = (all_codes[:3000].cpu().numpy().view(np.uint32)[:, None] >> np.arange(k)) & 1
    sure = np.abs(z) > tol
    np.testing.assert_array_equal(bits[sure], (z > 0)[sure])
    for n in (1, 127, 128, 129, 148 * 128, 148 * 128 + 1, 148 * 256 + 5):
        codes, zn = model.hash(xd[:n], with_z=True)
        assert torch.equal(codes, all_codes[:n]) and torch.equal(zn, all_z[:n])
        assert torch.equal(model.hash(xd[:n]), all_codes[:n])
    assert ms.stream_status() == ms.SIFT_OK
