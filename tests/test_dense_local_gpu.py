"""The dense push of one rank against the host table's update of the same coordinates, bit for bit."""
import pytest
import torch

from parameter_server_b200 import DenseTable, SparseTable

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opt,kw", [("adamw", dict(lr=3e-3, weight_decay=0.1)), ("adagrad", dict(lr=0.05)), ("sgd", dict(lr=0.1, weight_decay=0.01)),
                                    ("ftrl", dict(alpha=0.05, beta=1.0, l1=0.001, l2=0.01)), ("sum", {})])
@pytest.mark.parametrize("numel,grad16,sms", [(1, False, 0), (65, True, 0), (148 * 1024 * 4 - 8, False, 0), (148 * 1024 * 8 + 72, True, 0), (70003, False, 3)])
def test_dense_push_is_the_host_update(opt, kw, numel, grad16, sms):
    t = DenseTable({"w": (numel,)}, opt, dict(kw), grad_dtype=torch.bfloat16 if grad16 else torch.float32, device="cuda")
    t.set_sm_budget(sms)
    g = torch.Generator().manual_seed(numel)
    w = torch.randn(numel, generator=g)
    t.load({"w": w})
    pad = -numel % 64
    host = SparseTable(64, opt, dict(kw), device="cpu")
    keys = torch.arange((numel + pad) // 64)
    slots = host.table.stride() // 64
    rows = torch.zeros(keys.numel(), slots * 64)
    rows[:, :64] = torch.nn.functional.pad(w, (0, pad)).view(-1, 64)
    host.set_rows(keys, rows)
    for step in range(3):
        grad = torch.randn(numel, generator=g) * 1e-2
        t.zero_grads()
        t.grads["w"].copy_(grad)
        t.push()
        host.push(torch.nn.functional.pad(t.grads["w"].float().cpu(), (0, pad)).view(-1, 64), keys=keys)
    t.check()
    want = host.get_rows(keys)[0].reshape(-1)[:numel]
    assert torch.equal(t.master_slice().cpu()[:numel], want)
    assert torch.equal(t.params["w"].cpu(), want.bfloat16())
