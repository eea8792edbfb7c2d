"""Probe codes and the candidate scan at the edges of their launches: one
query, rows on both sides of a 32-query block, fewer bits than can be flipped,
every probe of a table, codes longer than the bucket bits, many probes with
skewed buckets. Integers against the oracle: bit-exact."""
import numpy as np
import pytest

import matching_sift_b200 as ms
import oracle

pytestmark = pytest.mark.gpu


def _probes(codes, dots, k, probes):
    flip = min(6, k)
    out = np.empty((probes, len(codes)), np.uint32)
    for i, c in enumerate(codes):
        mag = np.abs(dots[i, :k])
        kept = sorted(range(k), key=lambda j: (mag[j], j))[:flip]
        order = sorted(range(1 << flip), key=lambda s: (sum(mag[kept[b]] for b in range(flip) if s >> b & 1), s))
        for p in range(probes):
            out[p, i] = int(c) ^ sum(1 << kept[b] for b in range(flip) if order[p] >> b & 1)
    return out


@pytest.mark.parametrize("q_n,r_n,L,k,probes", [(1, 40, 1, 3, 8), (33, 1000, 2, 1, 2), (31, 129, 3, 6, 64),
                                                (65, 3000, 4, 20, 16), (129, 5000, 8, 16, 32), (40, 20000, 8, 8, 16),
                                                (7, 1, 2, 5, 4)])
def test_probe_scan_equals_oracle(cuda_device, q_n, r_n, L, k, probes):
    import torch

    rng = np.random.default_rng([q_n, r_n, k])
    r = rng.integers(0, 40, (r_n, 128)).astype(np.uint8)
    r[r_n // 2:] = np.clip(r[0].astype(int) + rng.integers(-3, 4, (r_n - r_n // 2, 128)), 0, 255)  # one crowded region
    q = rng.integers(0, 40, (q_n, 128)).astype(np.uint8)
    q[q_n // 2:] = r[rng.integers(0, r_n, q_n - q_n // 2)]
    planes = rng.integers(-3, 4, (L, k, 128)).astype(np.int8)  # small values: margins tie
    out = ms.lsh_match(*(torch.from_numpy(x).to(cuda_device) for x in (q, r, planes)), probes=probes, candidates=True)
    qcodes, rcodes, cand = [], [], np.zeros(q_n, np.int64)
    for t in range(L):
        qc, dots = oracle.lsh_codes(q, planes[t].astype(np.float32))
        rc, _ = oracle.lsh_codes(r, planes[t].astype(np.float32))
        pc = _probes(qc, dots, k, probes)
        cand += (pc[:, :, None] == rc[None, None, :]).any(0).sum(1)
        qcodes.append(pc)
        rcodes.extend([rc] * probes)
    d, i = oracle.lsh_scan(q, r, np.concatenate(qcodes), np.stack(rcodes))
    np.testing.assert_array_equal(out["nn_idx"].cpu().numpy().astype(np.int64), i)
    np.testing.assert_array_equal(out["nn_dist"].cpu().numpy()[i >= 0].astype(np.int64), d[i >= 0])
    np.testing.assert_array_equal(out["candidates"].cpu().numpy().astype(np.int64), cand)


def test_learned_probes_past_the_subsets(cuda_device):
    """k = 3 bits and 64 probes: 8 distinct codes, the rest repeat the query's own and add no candidates."""
    import torch

    rng = np.random.default_rng(4)
    q, r = (torch.from_numpy(rng.integers(0, 200, (n, 128)).astype(np.uint8)).to(cuda_device) for n in (37, 700))
    g = torch.Generator().manual_seed(3)
    params = 0.1 * torch.randn(256 * 128 + 256 + 32 * 256 + 32, generator=g)
    out = ms.MlpHash.from_params(params.to(cuda_device), 3).match(q, r, n_probes=64)
    d, i = oracle.brute_2nn_u8(q.cpu().numpy(), r.cpu().numpy())
    np.testing.assert_array_equal(out["nn_idx"].cpu().numpy(), i)
    assert (out["candidates"].cpu().numpy() == 700).all()
