"""One training step of the learned hash at the edges of its launches (48 rows
per forward block, 32 pairs per backward pass, 36 chunks of pairs) against FP64.

Tolerances: FP32 sums of at most 256 terms (h, dz) and 3 x 4,099 rows give
relative errors near 1e-6; a hidden value that rounds to the other BF16
neighbour changes by 2^-8 of itself, at most a few of a row's 256, so 2e-3 of a
block's norm bounds both."""
import numpy as np
import pytest

import matching_sift_b200 as ms
from matching_sift_b200 import datagen
from oracle import learned_hash as lh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,k", [(1, 1), (5, 32), (15, 3), (16, 16), (17, 16), (100, 24), (1152, 8), (4099, 17)])
def test_step_gradients_at_edges(cuda_device, B, k):
    import torch

    rng = np.random.default_rng(B)
    base = datagen.make_base(B + 50, seed=B)
    near = base[rng.integers(0, len(base), B)]
    q = np.clip(near.astype(int) + rng.integers(-9, 10, near.shape), 0, 255).astype(np.uint8)
    x = np.concatenate([q, near, base[rng.integers(0, len(base), B)]])
    p = lh.init_params(k, seed=B + k)
    loss, g = ms.mlp_loss_grad(torch.from_numpy(x).to(cuda_device), B, k, torch.from_numpy(p).to(cuda_device), 0.7, 0.9)
    want_loss, want = lh.loss_grad(p, x, B, k, 0.7, 0.9)
    np.testing.assert_allclose(loss, want_loss, rtol=2e-3, atol=1e-5)
    g = g.cpu().numpy().astype(np.float64)
    cuts = np.cumsum([0, lh.HID * lh.IN, lh.HID, lh.OUT_ROWS * lh.HID, lh.OUT_ROWS])
    for a, b in zip(cuts[:-1], cuts[1:]):
        assert np.linalg.norm(g[a:b] - want[a:b]) <= 2e-3 * np.linalg.norm(want[a:b])
    again = ms.mlp_loss_grad(torch.from_numpy(x).to(cuda_device), B, k, torch.from_numpy(p).to(cuda_device), 0.7, 0.9)
    np.testing.assert_array_equal(again[1].cpu().numpy(), g.astype(np.float32))  # fixed-order sums
