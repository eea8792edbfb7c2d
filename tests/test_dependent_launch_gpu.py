"""Searches whose kernels start while the kernel before still runs: calls enqueued
back to back over the same scratch, with sizes, types and paths that alternate,
return what each returns with a synchronisation around it. Exact equality: the
kernels are deterministic."""
import pytest

import matching_sift_b200 as ms

pytestmark = pytest.mark.gpu

# (queries, base rows, dtype): packed, folded, FP16 and general float searches,
# 4, 32 and more partial lists per row.
CALLS = [(517, 733, "u8"), (3, 70001, "u8"), (1400, 1, "f16"), (300, 30000, "f16"), (130, 9000, "f32"), (64, 128, "u8"),
         (1000, 10000, "f32"), (9000, 640, "u8")]


def _inputs(cuda_device):
    import torch

    g = torch.Generator(device=cuda_device).manual_seed(3)
    out = []
    for q, r, kind in CALLS:
        rows = [torch.randint(0, 180, (n, 128), generator=g, device=cuda_device, dtype=torch.uint8) for n in (q, r)]
        if kind == "f16":
            rows = [x.half() for x in rows]
        elif kind == "f32":
            rows = [x.float() + 0.3 * torch.rand(x.shape, generator=g, device=cuda_device) for x in rows]
        out.append(rows)
    return out


def test_back_to_back_calls(cuda_device):
    import torch

    inputs = _inputs(cuda_device)
    want = []
    for q, r in inputs:
        want.append(ms.match(q, r))
        torch.cuda.synchronize()
    for _ in range(3):
        got = [ms.match(q, r) for q, r in inputs]
        torch.cuda.synchronize()
        for w, g in zip(want, got):
            assert torch.equal(w["nn_idx"], g["nn_idx"]) and torch.equal(w["nn_dist"], g["nn_dist"])


def test_captured_calls(cuda_device):
    import torch

    pairs = [p for p, c in zip(_inputs(cuda_device), CALLS) if c[2] == "u8"]
    want = [ms.match(q, r)["nn_idx"] for q, r in pairs]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [ms.match(q, r)["nn_idx"] for _ in range(2) for q, r in pairs]
    for _ in range(3):
        for g in got:
            g.fill_(-7)
        graph.replay()
        torch.cuda.synchronize()
        for w, g in zip(want + want, got):
            assert torch.equal(w, g)
