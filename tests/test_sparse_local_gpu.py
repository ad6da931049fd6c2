"""The single-GPU pull / push / lookup kernels at the sizes where they can go wrong, against the host table.

Gradients are small whole numbers times a power of two, so every order of adding them gives the same fp32 sum and the
tables can be compared bit for bit whatever the kernels' order is.
"""
import pytest
import torch

from parameter_server_b200 import SparseTable, StatusCode

pytestmark = pytest.mark.gpu

OPTS = {"sgd": dict(lr=0.5, weight_decay=0.1), "adagrad": dict(lr=0.05, init_accumulator=0.1), "ftrl": dict(alpha=0.05, beta=1.0, l1=0.001, l2=0.01),
        "adam": dict(lr=0.01), "sum": {}}


def pair(dim, opt, max_keys, **kw):
    g = SparseTable(dim, opt, dict(OPTS[opt]), device="cuda", capacity=1 << 16, max_keys=max_keys, **kw)
    c = SparseTable(dim, opt, dict(OPTS[opt]), device="cpu", sync=kw.get("sync", False))
    return g, c


def whole(rows, dim, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randint(-8, 9, (rows, dim), generator=g).float() / 64


def same_tables(g, c, keys):
    g.check()
    u = torch.unique(keys)
    a, fa = g.get_rows(u.cuda(), emb_only=False)
    b, fb = c.get_rows(u, emb_only=False)
    assert fa.all() and fb.all() and torch.equal(a.cpu(), b)
    assert g.size() == c.size()


def batch(n, hot, seed):
    """n keys; the first ``len(hot)`` keys occur hot[i] times each (as far as there is room), the rest once, shuffled."""
    k = torch.cat([torch.full((h,), 1000003 * (i + 1), dtype=torch.int64) for i, h in enumerate(hot)] + [torch.arange(n) * 7919 + 5])[:n]
    return k[torch.randperm(n, generator=torch.Generator().manual_seed(seed))]


# below 2^18 keys a work item of a lane group holds 16 occurrences and a key of more than 1024 goes to CTA items of 256; a tile
# holds 1024 (2048) keys; lane groups of 1 .. 32 lanes
@pytest.mark.parametrize("dim,opt,n,hot", [
    (4, "sum", 1, []), (4, "sgd", 31, [2]), (8, "adagrad", 33, [31, 2]), (16, "adagrad", 257, [32, 33]), (64, "adagrad", 1025, [64, 65, 2, 3]),
    (64, "ftrl", 4099, [33, 1000]), (100, "adam", 3001, [2, 2, 2, 500]), (32, "sum", 9001, [1025, 1024, 2048, 2049, 3]), (128, "adagrad", 70001, [40000, 97, 32, 31]), (256, "sgd", 2049, [1500, 2]),
    (260, "adagrad", 999, [100, 5])])
@pytest.mark.parametrize("sms", [0, 5])
def test_step_is_the_host_tables_step(dim, opt, n, hot, sms):
    g, c = pair(dim, opt, n + 3)
    if sms:
        g.set_sm_budget(sms, sms)      # the 1024-thread shape
    for step in range(3):
        keys = batch(n, hot, step)
        a, b = g.pull(keys.cuda()), c.pull(keys)
        assert torch.equal(a.cpu(), b)
        assert g.engine.last_unique(0) == torch.unique(keys).numel()
        grads = whole(n, dim, step)
        g.push(grads.cuda()); c.push(grads)
    same_tables(g, c, keys)
    assert torch.equal(g.pull(keys.cuda(), insert=False).cpu(), c.pull(keys))
    if dim % 8 == 0:
        assert torch.equal(g.pull(keys.cuda(), insert=False, out_dtype=torch.bfloat16).cpu(), c.pull(keys).bfloat16())


# once-only keys of wide rows, from one position per block to thirty-two (148 SMs hold 4736 warps, a budget of 5 holds 160)
@pytest.mark.parametrize("dim,opt,n", [(256, "ftrl", 4735), (256, "adagrad", 9473), (128, "adam", 13312), (128, "sgd", 37889), (100, "ftrl", 75777), (256, "sum", 151553)])
@pytest.mark.parametrize("sms", [0, 5])
def test_keys_that_occur_once_at_every_block_length(dim, opt, n, sms):
    g, c = pair(dim, opt, n)
    if sms:
        g.set_sm_budget(sms, sms)
    keys = batch(n, [2], n)
    grads = whole(n, dim, 5)
    for _ in range(2):
        g.pull(keys.cuda()); c.pull(keys)
        g.push(grads.cuda()); c.push(grads)
    same_tables(g, c, keys)


# The three ways a batch's repeated keys are cut into work items: lane-group items of 16 occurrences and CTA items of 256 above 1024
# (below 2^18 keys), 32 and 512 above 2048 (below 2^21), 32 and 1024 above 2048. 700 001 keys are several tiles per CTA.
CUTS = {(1 << 18) - 1: [15, 16, 17, 31, 32, 33, 255, 256, 257, 1023, 1024, 1025, 1279, 1280, 1281, 5000],
        1 << 18: [15, 17, 31, 32, 33, 63, 64, 65, 1025, 2047, 2048, 2049, 2559, 2560, 2561, 20000],
        700001: [32, 33, 2048, 2049, 4607, 4608, 4609, 150000],
        (1 << 21) - 1: [33, 2048, 2049, 3071, 3072, 3073, 200000],
        1 << 21: [32, 33, 64, 65, 2048, 2049, 3071, 3072, 3073, 4097, 300000]}


@pytest.mark.parametrize("dim,opt,n,sms", [(4, "sum", (1 << 18) - 1, 0), (4, "sum", 1 << 18, 0), (64, "adagrad", (1 << 18) - 1, 0), (64, "adagrad", 1 << 18, 7), (16, "ftrl", 1 << 18, 0),
                                           (4, "sum", 700001, 0), (16, "adagrad", 700001, 0), (4, "sum", (1 << 21) - 1, 0), (4, "sum", 1 << 21, 0), (8, "adagrad", 1 << 21, 148)])
def test_step_of_large_batches_at_the_edges_of_their_work_items(dim, opt, n, sms):
    g, c = pair(dim, opt, n)
    if sms:
        g.set_sm_budget(sms, sms)
    keys = batch(n, CUTS[n], n)
    grads = whole(n, dim, 1)
    for _ in range(2):
        g.pull(keys.cuda()); c.pull(keys)
        g.push(grads.cuda()); c.push(grads)
    same_tables(g, c, keys)
    assert torch.equal(g.pull(keys.cuda()).cpu(), c.pull(keys))


@pytest.mark.parametrize("bag,mean", [(2, False), (4, True), (8, True)])
def test_pooled_step(bag, mean):
    g, c = pair(32, "sgd", 4096)
    keys = batch(4000, [300, 40, 2], 1)
    a, b = g.pull(keys.cuda(), bag_size=bag, mean=mean), c.pull(keys, bag_size=bag, mean=mean)
    assert torch.equal(a.cpu(), b)
    grads = whole(4000 // bag, 32, 2)
    g.push(grads.cuda()); c.push(grads)
    same_tables(g, c, keys)
    assert torch.equal(g.pull(keys.cuda(), bag, mean, insert=False).cpu(), c.pull(keys, bag, mean))


def test_sync_push_of_repeated_keys_and_a_plan_pushed_twice():
    g, c = pair(16, "adagrad", 4096, sync=True)
    keys = batch(3000, [200, 33, 2], 3)
    grads = whole(3000, 16, 4)
    g.pull(keys.cuda()); c.pull(keys)
    for _ in range(2):
        g.push(grads.cuda(), sync=True); c.push(grads, sync=True)
    g.store(); c.store()
    g.push(grads.cuda()); c.push(grads)
    same_tables(g, c, keys)


@pytest.mark.parametrize("how", ["deterministic_on", "lookup_first", "lookup_then_deterministic"])
def test_a_plan_of_another_kind_is_remade_for_the_push(how):
    """The pull's plan and the push's needs may differ: reproducible sums switched on in between, or a read-only pull."""
    g, c = pair(64, "adagrad", 4096)
    keys = batch(3000, [200, 33, 2], 5)
    g.pull(keys.cuda()); c.pull(keys)
    kd = keys.cuda()
    if how != "deterministic_on":
        g.pull(kd, insert=False, for_push=False)
        kd.zero_()                       # the plan is of the keys as they were pulled
        assert how != "lookup_first" or g.engine.last_unique(0) == torch.unique(keys).numel()
    if how != "lookup_first":
        g.set_deterministic(True)
    grads = whole(3000, 64, 6)
    g.push(grads.cuda()); c.push(grads)
    same_tables(g, c, keys)
    g.set_deterministic(False)
    g.pull(keys.cuda()); c.pull(keys)
    g.push(grads.cuda()); c.push(grads)
    same_tables(g, c, keys)


@pytest.mark.parametrize("insert,for_push,launches", [(False, True, [3, 2, 2]), (True, True, [2, 2]), (True, False, [2, 2]), (False, False, [3, 3])])
def test_a_pull_that_a_push_is_expected_behind_leaves_its_plan(insert, for_push, launches):
    """Pull and push are one launch each. A lookup is planned behind it when a push comes; the next pull that announces one expects it."""
    g, c = pair(32, "adagrad", 4096)
    keys = batch(3000, [200, 33, 2], 8)
    g.pull(keys.cuda()); c.pull(keys)
    grads = whole(3000, 32, 9)
    for want in launches:
        before = g.engine.kernel_launches()
        assert torch.equal(g.pull(keys.cuda(), insert=insert, for_push=for_push).cpu(), c.pull(keys))
        g.push(grads.cuda()); c.push(grads)
        assert g.engine.kernel_launches() - before == want
    same_tables(g, c, keys)


def test_pulls_without_a_push_are_lookups_again():
    g, c = pair(32, "adagrad", 4096)
    keys = batch(3000, [200, 33, 2], 8)
    grads = whole(3000, 32, 9)
    g.pull(keys.cuda()); c.pull(keys)

    def planned():      # how many launches it takes to know the number of distinct keys
        assert torch.equal(g.pull(keys.cuda(), insert=False).cpu(), c.pull(keys))
        before = g.engine.kernel_launches()
        assert g.engine.last_unique(0) == torch.unique(keys).numel()
        return g.engine.kernel_launches() - before

    assert planned() == 1
    g.push(grads.cuda()); c.push(grads)
    assert planned() == 0 and planned() == 1 and planned() == 1
    g.push(grads.cuda()); c.push(grads)
    g.pull(keys.cuda()); c.pull(keys)                # of another sort: nothing to learn from
    assert planned() == 0 and planned() == 1
    g.push(grads.cuda()); c.push(grads)
    same_tables(g, c, keys)


@pytest.mark.parametrize("general", [False, True])
def test_rows_erased_between_pull_and_push_get_nothing(general):
    g, c = pair(32, "sum", 4096)
    keys = batch(2000, [100, 2, 2], 7)
    before = g.pull(keys.cuda()).clone(); c.pull(keys)
    if general:
        g.set_deterministic(True)
    gone = torch.unique(keys)[::2]
    assert g.erase_keys(gone.cuda()) == gone.numel()
    g.push(torch.ones(2000, 32).cuda())
    assert g.status().code() == StatusCode.OUT_OF_MEMORY and g.status().ok()
    kept = ~torch.isin(keys, gone)
    count = (keys[:, None] == keys[None, :]).sum(1).float()
    rows, found = g.get_rows(keys.cuda())
    assert torch.equal(found.cpu().bool(), kept)
    assert torch.allclose(rows.cpu()[kept], before.cpu()[kept] + count[kept][:, None], rtol=2.0 ** -22, atol=0)   # one rounding of the sum


@pytest.mark.parametrize("dim,bags,bag,mean", [(4, 1, 1, False), (16, 1, 5000, False), (8, 3, 1025, False), (16, 64, 1024, True), (64, 1031, 1, False), (32, 257, 8, True),
                                               (100, 77, 3, False), (128, 4099, 2, True), (256, 300, 1, False), (260, 33, 37, False)])
@pytest.mark.parametrize("sms", [0, 3])
def test_lookup_is_the_host_tables_pull(dim, bags, bag, mean, sms):
    """Few large bags, many small ones, one in seven keys unknown; rows are whole numbers, so pooled sums are exact."""
    n = bags * bag
    g = pair(dim, "sum", n, read_only=True, init_range=0.0)[0]
    c = SparseTable(dim, "sum", device="cpu", init_range=0.0)
    if sms:
        g.set_sm_budget(sms, sms)
    keys = batch(n, [n // 5, 3], 11)
    known = torch.unique(keys)
    known = known[torch.arange(known.numel()) % 7 != 3]
    rows = whole(known.numel(), dim, 12)
    if known.numel():
        g.set_rows(known.cuda(), rows.cuda(), emb_only=True); c.set_rows(known, rows, emb_only=True)
    for dt in (torch.float32, torch.bfloat16)[:2 if dim % 8 == 0 else 1]:
        out = g.pull(keys.cuda(), bag, mean, for_push=False, out_dtype=dt)
        g.check()
        assert torch.equal(out.cpu(), c.pull(keys, bag, mean, insert=False).to(dt))
    assert g.size() == known.numel()


@pytest.mark.parametrize("general", [False, True])
def test_keys_that_get_their_row_between_pull_and_push(general):
    """The pull finds the row pool exhausted; the table then has room again and the keys are set. The push updates them."""
    g, c = pair(16, "sum", 8192, slab_shift=11)
    g.reserve(2048, exact=True)
    mem = g.memory_usage()
    g.table.set_limits(mem, mem)
    keys = batch(5200, [2000, 40, 2], 13)               # 3161 distinct keys, 2048 rows
    g.set_deterministic(general)
    g.pull(keys.cuda()); c.pull(keys)
    assert g.status().code() == StatusCode.OUT_OF_MEMORY
    u = torch.unique(keys)
    assert g.table.rows_used() == 2048 and g.size() == u.numel()
    g.table.set_limits(0, 0)
    g.table.set_healthy(True)
    rows = whole(u.numel(), 16, 14)
    g.set_rows(u.cuda(), rows.cuda(), emb_only=True); c.set_rows(u, rows, emb_only=True)
    grads = whole(5200, 16, 15)
    g.push(grads.cuda()); c.push(grads)
    same_tables(g, c, keys)


def test_lookup_of_unknown_keys_probe_chains_and_a_push_that_drops_them():
    """A nearly full index (chains of several slots), erased entries on the chains, unknown keys among the known."""
    g = SparseTable(8, "sum", device="cuda", capacity=1024, max_keys=4096, max_rows=2048, slab_shift=11, init_range=0.0)
    keys = torch.arange(1500) * 31 + 7
    g.set_rows(keys.cuda(), torch.arange(1500).float()[:, None].expand(1500, 8).contiguous().cuda())
    g.erase_keys(keys[::3].cuda())
    want = torch.where(torch.arange(1500) % 3 == 0, 0.0, torch.arange(1500).float())[:, None].expand(1500, 8)
    asked = torch.cat([keys, keys + 1]).cuda()
    out = g.pull(asked, insert=False); g.check()
    assert torch.equal(out.cpu(), torch.cat([want, torch.zeros(1500, 8)])) and g.size() == 1000
    g.push(torch.ones(3000, 8, device="cuda"))
    assert g.status().code() == StatusCode.OUT_OF_MEMORY    # keys without a row: dropped, the others applied
    assert torch.equal(g.pull(asked, insert=False).cpu(), torch.cat([torch.where(want > 0, want + 1, want), torch.zeros(1500, 8)]))
    assert g.size() == 1000
    empty = torch.empty(0, dtype=torch.int64, device="cuda")
    assert g.pull(empty, insert=False).shape == (0, 8) and g.pull(empty).shape == (0, 8)
    g.push(torch.empty(0, 8, device="cuda")); g.check()
