"""Calls that are refused on the device, and the push that follows before anybody has asked for the status: the error is
reported at the next check, the table is as it was, and the engine works again after a reset."""
import pytest
import torch

from parameter_server_b200 import SparseTable, StatusCode

pytestmark = pytest.mark.gpu

RESERVED = (-(1 << 63), -(1 << 63) + 1)


def tables(dim=16, max_keys=4096, **kw):
    g = SparseTable(dim, "adagrad", dict(lr=0.05, init_accumulator=0.1), device="cuda", capacity=1 << 14, max_keys=max_keys, **kw)
    c = SparseTable(dim, "adagrad", dict(lr=0.05, init_accumulator=0.1), device="cpu")
    return g, c


def whole(rows, dim, seed=1):
    """Small whole numbers over 64: their sums are exact in any order."""
    return torch.randint(-8, 9, (rows, dim), generator=torch.Generator().manual_seed(seed)).float() / 64


def step(g, c, keys, bag=1):
    grads = whole(keys.numel() // bag, g.dim, keys.numel())
    assert torch.equal(g.pull(keys.cuda(), bag).cpu(), c.pull(keys, bag))
    g.push(grads.cuda()); c.push(grads)
    g.check()


def same(g, c, keys):
    u = torch.unique(keys)
    a, fa = g.get_rows(u.cuda(), emb_only=False)
    b, fb = c.get_rows(u, emb_only=False)
    assert fa.all() and fb.all() and torch.equal(a.cpu(), b) and g.size() == c.size()


@pytest.mark.parametrize("reserved", RESERVED)
@pytest.mark.parametrize("how", ["after_a_plain_pull", "fewer_keys_than_before", "switched_on_behind_it"])
def test_reproducible_push_behind_a_refused_pull(how, reserved):
    g, c = tables()
    keys = torch.arange(1000) % 800 * 31 + 5          # 200 keys occur twice
    hot = torch.cat([keys, torch.full((500,), 5, dtype=torch.int64)])
    if how == "fewer_keys_than_before":
        g.set_deterministic(True)
    step(g, c, hot)
    bad = keys[:100].clone()
    bad[3] = reserved
    if how == "after_a_plain_pull":
        g.set_deterministic(True)
    g.pull(bad.cuda())
    if how == "switched_on_behind_it":                # two pulls: the second finds the status and leaves at its top
        g.pull(bad.cuda())
        g.set_deterministic(True)
    g.push(torch.ones(100, 16, device="cuda"))
    st = g.status()
    assert st.code() == StatusCode.ERROR and "reserved" in st.msg()
    same(g, c, hot)
    g.reset()
    for on in (True, False):
        g.set_deterministic(on)
        step(g, c, hot)
        step(g, c, keys[:100])
    same(g, c, hot)


def test_pair_capacity_below_the_batch_on_one_gpu():
    """Exact up to ``pair_capacity`` distinct keys whatever the batch's length, an error status beyond."""
    g, c = tables(pair_capacity=1000)
    keys = torch.arange(4096) % 1000 * 7 + 3
    few = torch.arange(1000) * 7 + 10                 # short enough for a plan with an entry per position
    for k in (keys, few, keys.flip(0)):
        step(g, c, k)
        assert torch.equal(g.pull(k.cuda(), insert=False, for_push=False).cpu(), c.pull(k))
    step(g, c, keys, bag=4)
    grads = whole(4096, 16)
    g.pull(keys.cuda(), insert=False, for_push=False); c.pull(keys)
    g.push(grads.cuda()); c.push(grads)
    g.check()
    same(g, c, torch.cat([keys, few]))
    g.pull((torch.arange(1001) * 7 + 3).cuda())
    st = g.status()
    assert st.code() == StatusCode.ERROR and "pair_capacity" in st.msg()
    g.reset()
    step(g, c, keys)
