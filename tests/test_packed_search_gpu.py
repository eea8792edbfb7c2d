"""Single searches on both sides of the rule that takes small ones to the packed
epilogue (64 units of 512 queries x 128 base rows per CTA pair), its key range,
the DOT metric and half inputs that stay off it: every kernel variant gives the
same bit-exact result."""
import numpy as np
import pytest

import matching_sift_b200 as ms
import oracle

pytestmark = pytest.mark.gpu


def _all(q, r, metric, dev):
    import torch

    qd, rd = torch.from_numpy(q).to(dev), torch.from_numpy(r).to(dev)
    out = []
    for variant in (0, 3):
        ms.lib().sift_set_kernel_variant(variant)
        try:
            o = ms.match(qd, rd, metric=metric, outputs=("matches", "nn_idx", "nn_dist", "sorted"))
            out.append({k: v.cpu().numpy() for k, v in o.items()})
        finally:
            ms.lib().sift_set_kernel_variant(0)
    for k in out[0]:
        np.testing.assert_array_equal(out[0][k], out[1][k], err_msg=k)
    return out[0]


@pytest.mark.parametrize("metric", [ms.METRIC_L2, ms.METRIC_DOT])
@pytest.mark.parametrize("q_n,r_n", [(1, 1), (513, 255), (129, 4097), (40, 64 * 74 * 128), (40, 64 * 74 * 128 + 1)])
def test_both_sides_of_the_rule(cuda_device, metric, q_n, r_n):
    rng = np.random.default_rng([q_n, r_n])
    r = rng.integers(0, 9, (r_n, 128)).astype(np.uint8)
    q = rng.integers(0, 9, (q_n, 128)).astype(np.uint8)
    q[0] = r[-1]
    got = _all(q, r, metric, cuda_device)
    d, i = oracle.brute_2nn_u8(q[:16], r, metric=metric)
    np.testing.assert_array_equal(got["nn_idx"][:16], i)
    np.testing.assert_array_equal(got["nn_dist"][:16][i >= 0].astype(np.int64), d[i >= 0])


def test_extreme_keys(cuda_device):
    rng = np.random.default_rng(1)
    r = (rng.integers(0, 2, (700, 128)) * 255).astype(np.uint8)
    r[::5] = 255
    r[1::5] = 0
    q = np.concatenate([np.full((2, 128), 255), np.zeros((2, 128)), r[7:40]]).astype(np.uint8)
    got = _all(q, r, ms.METRIC_L2, cuda_device)
    d, i = oracle.brute_2nn_u8(q, r)
    np.testing.assert_array_equal(got["nn_idx"], i)
    np.testing.assert_array_equal(got["nn_dist"].astype(np.int64), d)
