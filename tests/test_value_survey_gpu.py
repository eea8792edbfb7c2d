"""Float and half inputs at the edges of the value survey: the finest multiples,
the largest values, negative zero, one stray value that decides the path, scales
that differ between the two sets. Integers times one power of two are searched
exactly (bit-exact distances against FP64); anything else within
2^-16 (|q|^2 + |r|^2), the float path's stated bound."""
import numpy as np
import pytest

import matching_sift_b200 as ms
import oracle

pytestmark = pytest.mark.gpu

# (name, scale of the query set, scale of the base set, stray value put into the base, searched exactly)
CASES = [("plain", 1, 1, None, True), ("neg_zero", 1, 1, -0.0, True), ("largest", 1, 1, 255.0, True),
         ("256", 1, 1, 256.0, False), ("half_step", 1, 1, 2.5, True), ("fine_with_255", 1, 1, 2.0 ** -10, False),
         ("negative", 1, 1, -1.0, False), ("scaled", 2.0 ** -9, 2.0 ** -9, None, True),
         ("mixed_scales", 2.0 ** -9, 2.0 ** -4, None, True), ("finest", 2.0 ** -24, 2.0 ** -24, None, True),
         ("third", 1, 1, 1.0 / 3.0, False)]


@pytest.mark.parametrize("dtype", ["float32", "float16"])
@pytest.mark.parametrize("name,sq,sr,stray,exact", CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize("q_n,r_n", [(1, 3), (130, 1025)])
def test_value_survey(cuda_device, dtype, name, sq, sr, stray, exact, q_n, r_n):
    import torch

    rng = np.random.default_rng([q_n, len(name)])
    # Small integers, so that sets of different scales fit one scale (values <= 7 at 2^-4 and 2^-9: up to 7 * 32).
    top = 8 if name in ("mixed_scales", "half_step") else 200
    q = (rng.integers(0, top, (q_n, 128)) * sq).astype(dtype)
    r = (rng.integers(0, top, (r_n, 128)) * sr).astype(dtype)
    if name == "fine_with_255":
        r[0, 0] = 255.0
    if stray is not None:
        r[r_n - 1, 127] = stray
    qd, rd = torch.from_numpy(q).to(cuda_device), torch.from_numpy(r).to(cuda_device)
    out = ms.match(qd, rd, outputs=("nn_idx", "nn_dist"))
    d, i = oracle.brute_2nn_f64(q.astype(np.float32), r.astype(np.float32))
    got = out["nn_dist"].cpu().numpy().astype(np.float64)
    if exact:
        np.testing.assert_array_equal(out["nn_idx"].cpu().numpy(), i)
        np.testing.assert_array_equal(got, d)  # integers below 2^24 times a power of two: exact in float32
    else:
        slack = 2.0 ** -16 * ((q.astype(np.float64) ** 2).sum(1).max() + (r.astype(np.float64) ** 2).sum(1).max())
        assert np.abs(got - d).max() <= slack


@pytest.mark.parametrize("dtype", ["float32", "float16"])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_not_finite_is_refused(cuda_device, dtype, value):
    import torch

    q = torch.ones((5, 128), dtype=getattr(torch, dtype), device=cuda_device)
    r = torch.ones((300, 128), dtype=getattr(torch, dtype), device=cuda_device)
    r[299, 127] = float(value)
    with pytest.raises(ms.SiftError):
        ms.match(q, r)
    with pytest.raises(ms.SiftError):
        ms.match(r, q)
