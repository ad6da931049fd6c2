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


@pytest.mark.parametrize("n,at,sms,bag", [(1, 0, 0, 1), (300, 299, 0, 1), (9000, 8999, 1, 1), (9000, 4500, 3, 3), (70000, 69999, 0, 1), (70000, 0, 5, 7), (70000, 35000, 1, 70000)])
@pytest.mark.parametrize("call", ["pull", "plan"])
def test_a_refused_batch_leaves_the_table_alone(n, at, sms, bag, call):
    """A reserved key anywhere (one tile or several per CTA): none of the batch's other keys is inserted."""
    g, c = tables(max_keys=70000)
    if sms:
        g.set_sm_budget(sms, sms)
    old = torch.arange(500) * 13 + 1
    step(g, c, old)
    fresh = torch.arange(n) * 13 + 2
    bad = fresh.clone()
    bad[at] = RESERVED[n % 2]
    getattr(g, call)(bad.cuda(), bag)
    g.push(torch.ones(n // bag, 16, device="cuda"))
    st = g.status()
    assert st.code() == StatusCode.ERROR and "reserved" in st.msg()
    assert g.size() == 500 and not g.get_rows(fresh.cuda())[1].any()
    same(g, c, old)
    g.reset()
    step(g, c, fresh, bag)
    step(g, c, old)
    same(g, c, torch.cat([old, fresh]))


@pytest.mark.parametrize("n,at,sms,bag", [(1, 0, 0, 1), (300, 299, 0, 1), (9000, 8999, 1, 1), (9000, 4500, 3, 3), (70000, 69999, 0, 1), (70000, 0, 5, 7), (70000, 35000, 1, 70000)])
@pytest.mark.parametrize("call", ["pull", "plan"])
def test_a_refused_batch_leaves_the_table_alone(n, at, sms, bag, call):
    """A reserved key anywhere (one tile or several per CTA): none of the batch's other keys stays in the table."""
    g, c = tables(max_keys=70000)
    if sms:
        g.set_sm_budget(sms, sms)
    old = torch.arange(500) * 13 + 1
    step(g, c, old)
    fresh = torch.arange(n) * 13 + 2
    bad = torch.cat([fresh, fresh[:n // 3]])[-n:]       # some keys twice
    bad[at] = RESERVED[n % 2]
    getattr(g, call)(bad.cuda(), bag)
    g.push(torch.ones(n // bag, 16, device="cuda"))
    st = g.status()
    assert st.code() == StatusCode.ERROR and "reserved" in st.msg()
    assert g.size() == 500 and not g.get_rows(fresh.cuda())[1].any()
    same(g, c, old)
    g.reset()
    step(g, c, fresh, bag)
    step(g, c, old)
    same(g, c, torch.cat([old, fresh]))


def test_a_refused_batch_gives_back_the_rows_of_an_exhausted_pool():
    g, c = tables(max_keys=4096, slab_shift=11)
    old = torch.arange(500) * 13 + 1
    g.reserve(500, exact=True)
    g.set_rows(old.cuda(), torch.ones(500, 32).cuda()); c.set_rows(old, torch.ones(500, 32))
    g.table.set_limits(1, 1)                            # no further slab: 2048 rows
    bad = torch.arange(4000) * 13 + 2
    bad[17] = RESERVED[0]
    g.pull(bad.cuda())
    assert g.status().code() == StatusCode.ERROR and g.size() == 500
    g.reset()
    same(g, c, old)
    step(g, c, torch.arange(1548) * 13 + 2)             # all rows that are left, check() included
    same(g, c, torch.cat([old, torch.arange(1548) * 13 + 2]))
