"""The reproducible sparse push at the edges of its 64-occurrence blocks, against the host restatement of its order."""
import numpy as np
import pytest
import torch

from parameter_server_b200 import SparseTable

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,hot", [(16, [64, 65, 63]), (128, [128, 129, 2]), (64, [64 * 17, 64 * 17 + 1, 64 * 16 + 63]), (100, [20000, 1]), (256, [64 * 33 + 5])])
def test_ordered_sum_at_the_edges_of_its_blocks(dim, hot):
    from blocked_sum import blocked_segment_sum
    keys = torch.cat([torch.full((h,), 77 * (i + 1), dtype=torch.int64) for i, h in enumerate(hot)] + [torch.arange(200) * 5 + 100000])
    keys = keys[torch.randperm(keys.numel(), generator=torch.Generator().manual_seed(dim))]
    n = keys.numel()
    t = SparseTable(dim, "sum", device="cuda", capacity=1 << 12, max_keys=n)
    t.set_deterministic(True)
    c = SparseTable(dim, "sum", device="cpu")
    grads = torch.randn(n, dim, generator=torch.Generator().manual_seed(1))
    for _ in range(2):
        t.pull(keys.cuda()); c.pull(keys)
        t.push(grads.cuda())
        uk, agg = blocked_segment_sum(keys.numpy(), grads.numpy())
        c.push(torch.from_numpy(agg), keys=torch.from_numpy(np.ascontiguousarray(uk)))
    t.check()
    uk = torch.unique(keys)
    assert torch.equal(t.get_rows(uk.cuda())[0].cpu(), c.get_rows(uk)[0])
