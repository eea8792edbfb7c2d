"""Gradients of one training step where the row halves of the backward, the row
pairs of a forward warp and the two output ranges (up to 16, above) end, against
FP64; and the place of the loss.

Tolerance as for the other edges of the step: FP32 sums give relative errors near
1e-6, a hidden value that rounds to the other BF16 neighbour changes by 2^-8 of
itself and at most a few of a row's 256 do, so 2e-3 of a block's norm bounds both."""
import ctypes

import numpy as np
import pytest

import matching_sift_b200 as ms
from matching_sift_b200 import datagen
from oracle import learned_hash as lh

pytestmark = pytest.mark.gpu


def _rows(B, seed):
    rng = np.random.default_rng(seed)
    base = datagen.make_base(B + 50, seed=seed)
    near = base[rng.integers(0, len(base), B)]
    q = np.clip(near.astype(int) + rng.integers(-9, 10, near.shape), 0, 255).astype(np.uint8)
    return np.concatenate([q, near, base[rng.integers(0, len(base), B)]])


@pytest.mark.parametrize("B,k", [(2, 4), (33, 15), (47, 31), (65, 1), (288, 16), (1185, 20)])
def test_gradients_at_row_halves(cuda_device, B, k):
    import torch

    x = _rows(B, B + k)
    p = lh.init_params(k, seed=B)
    loss, g = ms.mlp_loss_grad(torch.from_numpy(x).to(cuda_device), B, k, torch.from_numpy(p).to(cuda_device), 0.7, 0.9)
    want_loss, want = lh.loss_grad(p, x, B, k, 0.7, 0.9)
    np.testing.assert_allclose(loss, want_loss, rtol=2e-3, atol=1e-5)
    g = g.cpu().numpy().astype(np.float64)
    cuts = np.cumsum([0, lh.HID * lh.IN, lh.HID, lh.OUT_ROWS * lh.HID, lh.OUT_ROWS])
    for a, b in zip(cuts[:-1], cuts[1:]):
        assert np.linalg.norm(g[a:b] - want[a:b]) <= 2e-3 * np.linalg.norm(want[a:b])
    w2 = g[cuts[2]:cuts[3]].reshape(lh.OUT_ROWS, lh.HID)
    assert not w2[k:].any() and not g[cuts[3] + k:].any()  # outputs past k have no gradient


def test_loss_lands_in_any_memory(cuda_device):
    import torch

    x = torch.from_numpy(_rows(4, 1)).to(cuda_device)
    p = torch.from_numpy(lh.init_params(8, seed=1)).to(cuda_device)
    g = torch.empty_like(p)
    loss = torch.zeros(4, device=cuda_device)
    fn = ms.lib().sift_mlp_loss_grad
    pinned, pageable = torch.zeros(4).pin_memory(), torch.zeros(4)
    for out in (loss, pinned, pageable):
        assert fn(x.data_ptr(), 4, 8, p.data_ptr(), 0.7, 0.9, g.data_ptr(),
                  ctypes.cast(out.data_ptr(), fn.argtypes[-1])) == ms.SIFT_OK
    assert pageable[0] > 0 and torch.equal(pinned, pageable) and torch.equal(loss.cpu(), pageable)
