"""The search with folded norms at sizes that take it (more than 64 units of 512
queries x 128 base rows per CTA pair; smaller L2 searches take the packed kernel):
norms around and above the largest half-norm that the digits hold, ties in every
tile, ragged ends, and its chain of overlapped launches back to back and in a
captured graph, between calls of the packed kernel. Integers against the oracle and
the single-CTA kernel: bit-exact."""
import numpy as np
import pytest

import matching_sift_b200 as ms
import oracle
from matching_sift_b200 import datagen

pytestmark = pytest.mark.gpu


def _rows(n_q, extra, dev):
    """The fewest whole base tiles that n_q queries leave to the folded kernel, plus `extra` rows."""
    import torch

    limit = 64 * (torch.cuda.get_device_properties(dev).multi_processor_count // 2)
    return (limit // -(-n_q // 512) + 1) * 128 + extra


def _check(q, r, dev):
    import torch

    out = []
    for variant in (0, 1):
        ms.lib().sift_set_kernel_variant(variant)
        try:
            o = ms.match(torch.from_numpy(q).to(dev), torch.from_numpy(r).to(dev))
            out.append({k: v.cpu().numpy() for k, v in o.items()})
        finally:
            ms.lib().sift_set_kernel_variant(0)
    assert ms.stream_status() == ms.SIFT_OK
    for k in out[0]:
        np.testing.assert_array_equal(out[0][k], out[1][k], err_msg=k)
    n = min(len(q), 96)
    sel = np.unique(np.concatenate([np.arange(n // 2), len(q) - 1 - np.arange(n // 2)]))
    d, i = oracle.brute_2nn_u8(q[sel], r)
    np.testing.assert_array_equal(out[0]["nn_idx"][sel].astype(np.int64), i)
    np.testing.assert_array_equal(out[0]["nn_dist"][sel].astype(np.int64), d)
    np.testing.assert_array_equal(out[0]["matches"][sel].astype(np.uint32), oracle.ratio_match(d, i, 0.8))


@pytest.mark.parametrize("q_n,extra", [(1, 1), (512, -1), (513, 0), (600, 127), (1025, 1)])
def test_ragged_sizes(cuda_device, q_n, extra):
    r_n = _rows(q_n, extra, cuda_device)
    rng = np.random.default_rng(q_n)
    r = rng.integers(0, 60, (r_n, 128)).astype(np.uint8)
    q = rng.integers(0, 60, (q_n, 128)).astype(np.uint8)
    q[0] = r[-1]  # the nearest row is the last one
    q[-1] = r[-min(r_n, 130)]
    _check(q, r, cuda_device)


@pytest.mark.parametrize("lo,hi", [(118, 131), (0, 256), (230, 256)])
def test_norms_past_the_digits(cuda_device, lo, hi):
    """Half-norms of up to 979,454 are folded; rows of 124s have 984,064, rows of 255s 4.2 M (large residuals)."""
    r_n = _rows(600, 5, cuda_device)
    rng = np.random.default_rng(hi)
    r = rng.integers(lo, hi, (r_n, 128)).astype(np.uint8)
    r[::7] = 255 - r[::7] // 3  # large rows among all others
    r[1::11] //= 4              # small ones
    r[3] = 0
    r[r_n // 2] = 255
    q = rng.integers(lo, hi, (600, 128)).astype(np.uint8)
    q[1::4] = r[rng.integers(0, r_n, len(q[1::4]))]
    q[2], q[6] = 0, 255
    _check(q, r, cuda_device)


def test_ties_in_every_tile(cuda_device):
    r_n = _rows(600, 64, cuda_device)
    few = np.concatenate([datagen.make_base(40, seed=1), np.full((2, 128), 255, np.uint8), np.zeros((1, 128), np.uint8)])
    r = np.tile(few, (-(-r_n // len(few)), 1))[:r_n]
    q = np.concatenate([few, datagen.make_base(600 - len(few), seed=2)])
    _check(q, r, cuda_device)


def test_overlapped_launches(cuda_device):
    """Folded and packed searches of several sizes over one workspace, enqueued back to back and captured."""
    import torch

    g = torch.Generator(device=cuda_device).manual_seed(5)
    sizes = [(700, _rows(700, 3, cuda_device)), (300, 900), (2000, 200000), (40, 5000), (513, _rows(513, 0, cuda_device))]
    calls = [[torch.randint(0, 180, (n, 128), generator=g, device=cuda_device, dtype=torch.uint8) for n in s] for s in sizes]
    want = []
    for q, r in calls:
        want.append(ms.match(q, r))
        torch.cuda.synchronize()
    for _ in range(3):
        got = [ms.match(q, r) for q, r in calls]
        torch.cuda.synchronize()
        for w, o in zip(want, got):
            assert torch.equal(w["nn_idx"], o["nn_idx"]) and torch.equal(w["nn_dist"], o["nn_dist"])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [ms.match(q, r)["nn_idx"] for _ in range(2) for q, r in calls]
    for _ in range(3):
        for o in got:
            o.fill_(-7)
        graph.replay()
        torch.cuda.synchronize()
        for w, o in zip(want + want, got):
            assert torch.equal(w["nn_idx"], o)
