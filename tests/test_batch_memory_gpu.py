"""Device memory of a batch plan: per query row a norm, one bound and the partial
lists (two of 16 bytes per worker that shares the row's group), nothing else."""
import numpy as np
import pytest

import matching_sift_b200 as ms

pytestmark = pytest.mark.gpu


def test_plan_memory_per_query_row(cuda_device):
    import torch

    rows = 4 << 20
    q = torch.zeros((rows, 128), dtype=torch.uint8, device=cuda_device)
    r = torch.zeros((100, 128), dtype=torch.uint8, device=cuda_device)
    pairs = np.array([[rows, 100, 0]], np.uint32)
    ms.BatchPlan(q[:1000], r, np.array([[1000, 100, 0]], np.uint32), tune=False, shape=0).close()  # contexts, modules
    out = [torch.empty((rows, n), dtype=torch.int32, device=cuda_device) for n in (1, 2, 2)]  # the plan's outputs, warm
    del out
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info(cuda_device)[0]
    plan = ms.BatchPlan(q, r, pairs, tune=False, shape=0)
    used = free - torch.cuda.mem_get_info(cuda_device)[0]
    # One unit per query group, so one worker per row: 4 + 4 + 2 x 16 bytes. 8 MiB for the
    # allocator's granularity and the graph; a second bound would add 16 MiB.
    assert used <= rows * (4 + 4 + 2 * 16) + (8 << 20)
    idx = plan.run()["nn_idx"]
    assert int(idx[:, 0].abs().max()) == 0 and int(idx[:, 1].min()) == 1 and int(idx[:, 1].max()) == 1
    plan.close()
