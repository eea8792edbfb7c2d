"""One training step at the edges of its launches (48 rows per forward block, 32
pairs per backward pass, at least 8 and at most 36 chunks of pairs) where the
hidden layer is exact: weights are a few bits of 2^-5, so every sum of layer 1 is an
integer below 2^24 times 2^-11 and rounds to the BF16 value that FP64 gives.

Tolerance, derived before the first run: the outputs are FP32 sums of 256 terms
(relative error near sqrt(256) 2^-24 = 1e-6), tanh adds two units in the last place,
dz a factor of up to 10 where its terms cancel, and the rounding errors of different
rows are independent like the rows' own shares, so a block's error stays below 2e-5
of its norm. A pair left out or counted twice is at least 1 / sqrt(3 x 4,099) = 1e-2
of it."""
import numpy as np
import pytest

import matching_sift_b200 as ms
from oracle import learned_hash as lh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,k", [(1, 1), (7, 5), (8, 16), (16, 17), (31, 4), (33, 32), (97, 16), (287, 24), (289, 7),
                                 (1151, 32), (1153, 16), (2048, 16), (4099, 17)])
def test_step_gradients_with_exact_hidden_layer(cuda_device, B, k):
    import torch

    rng = np.random.default_rng([B, k])
    x = rng.integers(0, 256, (3 * B, 128)).astype(np.uint8)
    x[B:2 * B] = np.clip(x[:B].astype(int) + rng.integers(-9, 10, (B, 128)), 0, 255)
    w2, b2 = np.zeros((lh.OUT_ROWS, lh.HID)), np.zeros(lh.OUT_ROWS)
    w2[:k] = rng.integers(-8, 9, (k, lh.HID)) / 128
    b2[:k] = rng.integers(-8, 9, k) / 64
    p = lh.pack(rng.integers(-2, 3, (lh.HID, lh.IN)) / 32, rng.integers(-8, 9, lh.HID) / 16, w2, b2)
    loss, g = ms.mlp_loss_grad(torch.from_numpy(x).to(cuda_device), B, k, torch.from_numpy(p).to(cuda_device), 0.7, 0.9)
    want_loss, want = lh.loss_grad(p, x, B, k, 0.7, 0.9)
    np.testing.assert_allclose(loss, want_loss, rtol=2e-5, atol=2e-6)
    g = g.cpu().numpy().astype(np.float64)
    cuts = np.cumsum([0, lh.HID * lh.IN, lh.HID, lh.OUT_ROWS * lh.HID, lh.OUT_ROWS])
    for a, b in zip(cuts[:-1], cuts[1:]):
        assert np.linalg.norm(g[a:b] - want[a:b]) <= 2e-5 * np.linalg.norm(want[a:b])
