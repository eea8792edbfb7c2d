"""Multi-probe with margins that are not numbers (a learned hash with NaN weights,
float rows whose projections overflow to inf - inf): the probes are those of the
serial selection below, the query's own code first, so a query that is a base row
finds itself. Codes and counts are integers: exact."""
import numpy as np
import pytest

import matching_sift_b200 as ms

pytestmark = pytest.mark.gpu


def _probes(code, z, probes):
    """Bits kept by insertion in bit order, then the first lightest subset left, in float32."""
    k = len(z)
    flip, mag, bit = min(6, k), [], []
    for j, a in enumerate(np.abs(z.astype(np.float32))):
        if len(mag) == flip:
            if not a < mag[-1]:
                continue
            mag.pop(), bit.pop()
        p = len(mag)
        while p > 0 and mag[p - 1] > a:
            p -= 1
        mag.insert(p, a), bit.insert(p, j)
    out, left = [], list(range(1 << flip))
    while left and len(out) < probes:
        sums = {}
        for s in left:
            sums[s] = np.float32(0)
            for b in range(flip):
                if s >> b & 1:
                    sums[s] = np.float32(sums[s] + mag[b])
        best = left[0]
        for s in left[1:]:
            if sums[s] < sums[best]:
                best = s
        left.remove(best)
        out.append(int(code) ^ sum(1 << bit[b] for b in range(flip) if best >> b & 1))
    return out


@pytest.mark.parametrize("k,nan_bits,probes", [(8, (1,), 8), (12, (0, 7, 11), 16), (3, (2,), 8), (16, (4,), 64)])
def test_learned_hash_with_nan_outputs(cuda_device, k, nan_bits, probes):
    import torch

    rng = np.random.default_rng(k)
    r = torch.from_numpy(rng.integers(0, 200, (900, 128)).astype(np.uint8)).to(cuda_device)
    q = r[100:165].contiguous()  # past one block of 32 queries
    g = torch.Generator().manual_seed(k)
    params = 0.1 * torch.randn(256 * 128 + 256 + 32 * 256 + 32, generator=g)
    for j in nan_bits:
        params[256 * 128 + 256 + 32 * 256 + j] = float("nan")
    model = ms.MlpHash.from_params(params.to(cuda_device), k)
    out = model.match(q, r, n_probes=probes)
    codes, z = (x.cpu().numpy() for x in model.hash(q, with_z=True))
    base = np.asarray(model.hash(r).cpu().numpy()).astype(np.int64) & 0xFFFFFFFF
    assert np.isnan(z).sum() == len(nan_bits) * len(z)
    count = np.bincount(base, minlength=1 << k)
    want = [int(sum(count[c] for c in set(_probes(codes.astype(np.int64)[i], z[i], probes)))) for i in range(len(z))]
    np.testing.assert_array_equal(out["candidates"].cpu().numpy().astype(np.int64), want)
    np.testing.assert_array_equal(out["nn_dist"].cpu().numpy()[:, 0], 0)


def test_float_rows_that_overflow(cuda_device):
    import torch

    rng = np.random.default_rng(9)
    r = rng.standard_normal((300, 128)).astype(np.float32)
    r[:40, ::2] = 2.9e38  # dot products with both signs: inf - inf
    r = torch.from_numpy(r).to(cuda_device)
    planes = torch.from_numpy(rng.integers(-90, 91, (2, 10, 128)).astype(np.int8)).to(cuda_device)
    one = ms.lsh_match(r[40:], r[40:], planes, probes=1, candidates=True)
    out = ms.lsh_match(r, r, planes, probes=4, candidates=True)
    torch.cuda.synchronize()
    assert (out["candidates"][:40].cpu().numpy().astype(np.int64) >= 1).all()  # the own bucket is among the probes
    assert (out["nn_dist"][40:, 0] == 0).all()
    assert (out["candidates"][40:].cpu().numpy().astype(np.int64) >= one["candidates"].cpu().numpy().astype(np.int64)).all()
