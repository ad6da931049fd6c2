"""What a user of this package has it do, as timed cases.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (tables with resident rows,
inputs, weights), ``run`` is one pass through the public entry points, ``exact`` the same results in 64 bits from plain
torch. ``listed`` names the cases that are always timed, ``draw`` gives more of the same ranges.

Kinds:

* ``train``   one step of a sparse trainer on a resident table: ``SparseTable.push`` of the gradients of the last batch,
  then ``SparseTable.pull`` of the next. The next batch asks for the same keys, so the pulled rows show every row that
  the push changed. ``mode``: "plain"; "reproducible" (sums in a fixed order, ``set_deterministic``); "sync" (buffered
  pushes: ``push(sync=True)`` and ``store``).
* ``lookup``  a predictor's read-only pull, pooled over bags, with one key in fifty unknown to the table.
* ``dense``   ``DenseTable.push`` of one transformer layer's (or a small MLP's) gradients.
* ``mlp``     forward, backward and weight gradients of a ReLU MLP (``ops.gemm.chain``, ``grouped_wgrad``, ``bias_grads``).
* ``linear``  one wide linear layer forward and backward (``linear_fwd``, ``linear_dgrad``, ``linear_wgrad``).
* ``dlrm``    a whole training step of the click model (``DLRM.train_step`` on a captured graph, batch in pinned memory).
"""
import math

import numpy as np
import torch

from parameter_server_b200 import DenseTable, SparseTable
from parameter_server_b200.models import DLRM, DLRMConfig
from parameter_server_b200.ops import gemm as G

SLOTS = {"sgd": 0, "adagrad": 1, "ftrl": 2, "adam": 2}
OPT = {
    "sgd": dict(lr=0.05),
    "adagrad": dict(lr=0.05, init_accumulator=0.1),
    "ftrl": dict(alpha=0.05, beta=1.0, l1=1e-4, l2=0.01),
    "adam": dict(lr=1e-3),
}
TOP = (512, 1024, 1024, 512, 256)   # input width and layers of the click model's top MLP
BOTTOM = (16, 512, 256, 128)        # the same of its bottom MLP (13 dense features, padded)


def listed():
    return [
        # the smallest trainer step: 8192 keys of dim 16 out of a million (two workers on one box); launches and latency
        dict(name="train_8k_d16", kind="train", n=8192, dim=16, opt="adagrad", rows=1_000_000, zipf=1.1, bag=1, bf16=False, mode="plain"),
        # a small batch of a mid-sized model: the low end of the key-throughput sweep
        dict(name="train_64k_d64", kind="train", n=65536, dim=64, opt="adagrad", rows=4_000_000, zipf=1.05, bag=1, bf16=False, mode="plain"),
        # the headline of the key-throughput sweep: 1 Mi keys per GPU and step, dim 64 and an Adagrad slot
        dict(name="train_1m_d64", kind="train", n=1 << 20, dim=64, opt="adagrad", rows=8_000_000, zipf=1.05, bag=1, bf16=False, mode="plain"),
        # its high end
        dict(name="train_4m_d64", kind="train", n=1 << 22, dim=64, opt="adagrad", rows=16_000_000, zipf=1.05, bag=1, bf16=False, mode="plain"),
        # the elastic table under load: 512 Ki keys, dim 32 with two FTRL slots
        dict(name="train_512k_d32_ftrl", kind="train", n=1 << 19, dim=32, opt="ftrl", rows=8_000_000, zipf=1.1, bag=1, bf16=False, mode="plain"),
        # a trainer that asks for reproducible sums, at the click model's batch (8192 samples x 26 fields, dim 128)
        dict(name="train_213k_d128_repro", kind="train", n=212_992, dim=128, opt="adagrad", rows=2_000_000, zipf=1.1, bag=1, bf16=False, mode="reproducible"),
        # serving: one request's keys against a read-only table
        dict(name="lookup_1k_d64", kind="lookup", bags=1000, bag=1, dim=64, rows=1_000_000, zipf=1.05, mean=False, bf16=False),
        # batch scoring with multi-valued features: ragged bag count, mean pooling, activations in bf16
        dict(name="lookup_bags_d128", kind="lookup", bags=4099, bag=37, dim=128, rows=4_000_000, zipf=1.05, mean=True, bf16=True),
        # the optimizer step of one decoder layer (d_model 2048, FFN 8192): 50 M parameters, AdamW
        dict(name="dense_layer_2048", kind="dense", d=2048, f=8192, bf16=False),
        # the click model's top MLP, forward and backward, at its batch per GPU
        dict(name="mlp_top_8192", kind="mlp", batch=8192, widths="top"),
        # the QKV projection of a decoder layer, forward and backward, two sequences
        dict(name="linear_qkv_4096", kind="linear", tokens=4096, d_in=2048, d_out=6144),
        # the whole click-model step
        dict(name="dlrm_8192", kind="dlrm", batch=8192),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train"] * 5 + ["lookup"] * 2 + ["dense", "mlp", "linear", "dlrm"])
    if kind == "train":
        dim = rng.choice([8, 16, 32, 48, 64, 64, 100, 128, 256])
        bag = rng.choice([1, 1, 1, 2, 5])
        n = _log(rng, 1000, min(1 << 22, (1 << 27) // dim))
        return dict(kind="train", n=max(1, n // bag) * bag, dim=dim, opt=rng.choice(["adagrad", "adagrad", "sgd", "ftrl", "adam"]),
                    rows=_log(rng, 200_000, 4_000_000), zipf=rng.choice([1.05, 1.1, 1.2]), bag=bag, bf16=dim % 8 == 0 and rng.random() < 0.3,
                    mode=rng.choice(["plain"] * 6 + ["reproducible", "sync"]))
    if kind == "lookup":
        dim = rng.choice([8, 16, 32, 64, 100, 128, 256])
        bag = rng.choice([1, 1, 3, 10, 37])
        n = _log(rng, 200, min(1 << 21, (1 << 27) // dim))
        return dict(kind="lookup", bags=max(1, n // bag), bag=bag, dim=dim, rows=_log(rng, 200_000, 4_000_000), zipf=rng.choice([1.05, 1.1, 1.2]),
                    mean=rng.random() < 0.5, bf16=dim % 8 == 0 and rng.random() < 0.5)
    if kind == "dense":
        d = _log(rng, 64, 2048)
        return dict(kind="dense", d=d, f=4 * d, bf16=rng.random() < 0.3)
    if kind == "mlp":
        return dict(kind="mlp", batch=_log(rng, 256, 8192), widths=rng.choice(["top", "top", "bottom"]))
    if kind == "linear":
        return dict(kind="linear", tokens=_log(rng, 256, 4096), d_in=64 * rng.randint(4, 32), d_out=64 * rng.randint(4, 96))
    return dict(kind="dlrm", batch=8 * _log(rng, 64, 1024))


# ---- inputs ------------------------------------------------------------------------------------------------------
def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + salt)


def _uniform(g, *shape):
    return torch.rand(shape, generator=g, device="cuda")


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device="cuda")


def _key_of(rank):
    """Ranks scattered over the 40-bit key space (an odd factor: no two ranks meet)."""
    return (rank * 0x9E3779B97F4B) & ((1 << 40) - 1)


def _zipf_ranks(g, n, s, rows):
    """Zipf(s) ranks in [0, rows): the inverse of the bounded power law's distribution function."""
    u = torch.rand((n,), generator=g, device="cuda", dtype=torch.float64)
    top = float(rows + 1) ** (1.0 - s)
    r = (1.0 + u * (top - 1.0)) ** (1.0 / (1.0 - s))
    return (r.floor().to(torch.int64) - 1).clamp_(0, rows - 1)


def _rows_of(case, seed, lo, hi, width):
    """Resident rows [lo, hi) as the table stores them: embedding, then optimizer slots with the values of a table that
    has been trained for a while."""
    g, dim, opt = _gen(seed, 17 + lo), case["dim"], case.get("opt", "sgd")
    r = torch.empty((hi - lo, width), device="cuda")
    r[:, :dim] = _uniform(g, hi - lo, dim) * 0.02 - 0.01
    if opt == "adagrad":
        r[:, dim:2 * dim] = _uniform(g, hi - lo, dim) * 0.1 + 0.1
    elif opt == "ftrl":
        r[:, dim:2 * dim] = _normal(g, hi - lo, dim) * 1e-3
        r[:, 2 * dim:3 * dim] = _uniform(g, hi - lo, dim) * 1e-4
    elif opt == "adam":
        r[:, dim:2 * dim] = _normal(g, hi - lo, dim) * 1e-4
        r[:, 2 * dim:3 * dim] = _uniform(g, hi - lo, dim) * 1e-6
    r[:, (1 + SLOTS[opt]) * dim:] = 0
    return r


CHUNK = 1 << 20


def _fill(table, case, seed, width):
    for lo in range(0, case["rows"], CHUNK):
        hi = min(case["rows"], lo + CHUNK)
        table.set_rows(_key_of(torch.arange(lo, hi, device="cuda")), _rows_of(case, seed, lo, hi, width))


def _train_inputs(case, seed):
    g = _gen(seed, 3)
    ranks = _zipf_ranks(g, case["n"], case["zipf"], case["rows"])
    grads = _normal(g, case["n"] // case["bag"], case["dim"]) * 1e-3
    return ranks, grads


def _lookup_ranks(case, seed):
    g = _gen(seed, 3)
    n = case["bags"] * case["bag"]
    ranks = _zipf_ranks(g, n, case["zipf"], case["rows"])
    unknown = torch.rand((n,), generator=g, device="cuda") < 0.02
    return torch.where(unknown, ranks + case["rows"], ranks)


def _dense_shapes(case):
    d, f = case["d"], case["f"]
    return {"qkv.w": (3 * d, d), "qkv.b": (3 * d,), "proj.w": (d, d), "proj.b": (d,), "fc.w": (f, d), "fc.b": (f,), "out.w": (d, f),
            "out.b": (d,), "ln.g": (d,)}


DENSE_OPT = dict(lr=3e-4, weight_decay=0.1, beta2=0.95)


def _dense_values(case, seed):
    g = _gen(seed, 5)
    gt = torch.bfloat16 if case["bf16"] else torch.float32
    return {k: (_normal(g, *s) * 0.02, (_normal(g, *s) * 1e-3).to(gt)) for k, s in _dense_shapes(case).items()}


def _widths(case):
    return TOP if case["widths"] == "top" else BOTTOM


def _mlp_inputs(case, seed):
    g, w, b = _gen(seed, 7), _widths(case), case["batch"]
    bf = torch.bfloat16
    return dict(x=_normal(g, b, w[0]).to(bf), dy=(_normal(g, b, w[-1]) * 1e-3).to(bf),
                w=[(_normal(g, w[i + 1], w[i]) * (2.0 / w[i]) ** 0.5).to(bf) for i in range(len(w) - 1)],
                b=[(_normal(g, w[i + 1]) * 0.1).to(bf) for i in range(len(w) - 1)])


def _linear_inputs(case, seed):
    g, bf = _gen(seed, 9), torch.bfloat16
    return dict(x=_normal(g, case["tokens"], case["d_in"]).to(bf), w=(_normal(g, case["d_out"], case["d_in"]) * 0.02).to(bf),
                b=(_normal(g, case["d_out"]) * 0.1).to(bf), dy=(_normal(g, case["tokens"], case["d_out"]) * 1e-3).to(bf))


CTR = DLRMConfig()


def _dlrm_shapes():
    n_inter = CTR.emb_dim + (CTR.num_sparse + 1) * CTR.num_sparse // 2
    bd = [(CTR.num_dense + 7) // 8 * 8] + list(CTR.bottom)
    td = [(n_inter + 63) // 64 * 64] + list(CTR.top)
    shapes = {}
    for p, dims in (("bot", bd), ("top", td)):
        for i in range(len(dims) - 1):
            shapes["%s.w%d" % (p, i)] = (dims[i + 1], dims[i])
            shapes["%s.b%d" % (p, i)] = (dims[i + 1],)
    shapes["head.w"] = (td[-1],)
    shapes["head.b"] = (1,)
    return shapes, n_inter


def _dlrm_inputs(case, seed):
    """A batch as the input pipeline leaves it in pinned memory, the weights, and the rows of the batch's keys."""
    rng, b = np.random.default_rng(seed), case["batch"]
    vocab = np.array([int(round(v)) for v in np.logspace(np.log10(CTR.vocab_min), np.log10(CTR.vocab_max), CTR.num_sparse)], dtype=np.int64)
    dense = rng.lognormal(0.0, 1.0, size=(b, CTR.num_dense)).astype(np.float32)
    ids = (rng.zipf(CTR.zipf_s, size=(b, CTR.num_sparse)).astype(np.int64) - 1) % vocab[None, :]
    keys = (np.arange(CTR.num_sparse, dtype=np.int64)[None, :] << 40) | ids
    labels = (rng.random(b) < CTR.label_rate).astype(np.float32)
    batch = tuple(torch.from_numpy(a) for a in (dense, keys, labels))
    shapes, n_inter = _dlrm_shapes()
    g = _gen(seed, 11)
    weights = {}
    for name, shape in shapes.items():
        fan = shape[-1]
        w = _normal(g, *shape) * ((2.0 / fan) ** 0.5 if len(shape) == 2 else fan ** -0.5 if name == "head.w" else 0.01)
        if name == "bot.w0":
            w[:, CTR.num_dense:] = 0
        if name == "top.w0":
            w[:, n_inter:] = 0
        weights[name] = w.to(torch.bfloat16).float()
    uniq = torch.unique(batch[1].reshape(-1)).cuda()
    rows = torch.empty((uniq.numel(), 2 * CTR.emb_dim), device="cuda")
    rows[:, :CTR.emb_dim] = _uniform(g, uniq.numel(), CTR.emb_dim) * 0.2 - 0.1
    rows[:, CTR.emb_dim:] = _uniform(g, uniq.numel(), CTR.emb_dim) * 0.1 + 0.1
    return batch, weights, uniq, rows


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        sync = case["mode"] == "sync"
        t = SparseTable(case["dim"], case["opt"], dict(OPT[case["opt"]]), capacity=case["rows"], max_keys=case["n"], sync=sync)
        t.reserve(case["rows"] + 3 * case["n"], exact=True)
        if case["mode"] == "reproducible":
            t.set_deterministic(True)
        _fill(t, case, seed, case["dim"] * (1 + SLOTS[case["opt"]] + int(sync)))
        ranks, grads = _train_inputs(case, seed)
        keys = _key_of(ranks)
        out = torch.empty((case["n"] // case["bag"], case["dim"]), device="cuda", dtype=torch.bfloat16 if case["bf16"] else torch.float32)
        t.pull(keys, case["bag"], out=out)
        t.check()
        return dict(case=case, table=t, keys=keys, grads=grads, out=out)
    if kind == "lookup":
        # a predictor's table: unknown keys read as zero
        t = SparseTable(case["dim"], "sgd", dict(OPT["sgd"]), capacity=case["rows"], max_keys=case["bags"] * case["bag"], read_only=True, init_range=0.0)
        t.reserve(case["rows"], exact=True)
        _fill(t, case, seed, case["dim"])
        return dict(case=case, table=t, keys=_key_of(_lookup_ranks(case, seed)), dtype=torch.bfloat16 if case["bf16"] else torch.float32)
    if kind == "dense":
        t = DenseTable(_dense_shapes(case), "adamw", dict(DENSE_OPT), grad_dtype=torch.bfloat16 if case["bf16"] else torch.float32)
        values = _dense_values(case, seed)
        t.load({k: v[0] for k, v in values.items()})
        t.zero_grads()
        for k, v in values.items():
            t.grads[k].copy_(v[1])
        return dict(case=case, table=t)
    if kind == "mlp":
        s, w, b = _mlp_inputs(case, seed), _widths(case), case["batch"]
        new = lambda n, dt=torch.bfloat16: torch.empty((b, n), device="cuda", dtype=dt)  # noqa: E731
        s.update(case=case, act=[new(n) for n in w[1:]], dz=[new(n) for n in w[1:-1]] + [s["dy"]], dx=new(w[0]),
                 grad=torch.zeros(sum(w[i + 1] * w[i] + w[i + 1] for i in range(len(w) - 1)), device="cuda"))
        s["dw"], s["db"], at = [], [], 0
        for i in range(len(w) - 1):
            s["dw"].append(s["grad"][at:at + w[i + 1] * w[i]].view(w[i + 1], w[i]))
            at += w[i + 1] * w[i]
        for i in range(len(w) - 1):
            s["db"].append(s["grad"][at:at + w[i + 1]])
            at += w[i + 1]
        return s
    if kind == "linear":
        s = _linear_inputs(case, seed)
        bf = torch.bfloat16
        s.update(case=case, y=torch.empty((case["tokens"], case["d_out"]), device="cuda", dtype=bf),
                 dx=torch.empty((case["tokens"], case["d_in"]), device="cuda", dtype=bf), dw=torch.empty((case["d_out"], case["d_in"]), device="cuda"))
        return s
    batch, weights, uniq, rows = _dlrm_inputs(case, seed)
    m = DLRM(CTR, case["batch"], table_capacity=1 << 20)
    m.dense.load(weights)
    m.sparse.reserve(uniq.numel(), exact=True)
    m.sparse.set_rows(uniq, rows)
    m.enable_graph()
    return dict(case=case, model=m, batch=tuple(t.pin_memory() for t in batch))


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "train":
        t = s["table"]
        if case["mode"] == "sync":
            t.push(s["grads"], sync=True)
            t.store()
        else:
            t.push(s["grads"])
        return t.pull(s["keys"], case["bag"], out=s["out"])
    if kind == "lookup":
        return s["table"].pull(s["keys"], case["bag"], case["mean"], for_push=False, out_dtype=s["dtype"])
    if kind == "dense":
        s["table"].push()
        return dict(params=dict(s["table"].params), master=s["table"].master_slice())
    if kind == "mlp":
        n = len(s["w"])
        G.chain([dict(a=s["act"][i - 1] if i else s["x"], w=s["w"][i], bias=s["b"][i], relu=True, out=s["act"][i]) for i in range(n)])
        G.chain([dict(a=s["dz"][i], w=s["w"][i], mask=s["act"][i - 1] if i else None, out=s["dz"][i - 1] if i else s["dx"]) for i in range(n - 1, -1, -1)],
                b_mn=True)
        s["grad"].zero_()
        G.grouped_wgrad([(s["dz"][i], s["act"][i - 1] if i else s["x"], s["dw"][i]) for i in range(n)])
        G.bias_grads(list(zip(s["dz"], s["db"])))
        return dict(act=s["act"], dz=s["dz"][:-1], dx=s["dx"], dw=s["dw"], db=s["db"])
    if kind == "linear":
        G.linear_fwd(s["x"], s["w"], s["b"], out=s["y"])
        G.linear_dgrad(s["dy"], s["w"], out=s["dx"])
        G.linear_wgrad(s["dy"], s["x"], out=s["dw"])
        return dict(y=s["y"], dx=s["dx"], dw=s["dw"])
    m = s["model"]
    loss = m.train_step(*s["batch"])
    # The first Adam step moves a weight by its gradient's sign alone, so the gradients are what can be compared; the
    # gradients of a second step show what the push left in both tables.
    return dict(loss=loss, dense_grads=m.dense.flat_grads, row_grads=m.d_emb)


# ---- what a pass cannot do without -------------------------------------------------------------------------------
def _distinct(n, s, rows):
    """Expected number of distinct keys among n draws."""
    edge = np.unique(np.concatenate([np.arange(1, 1001), np.geomspace(1001, rows + 1, 4000).astype(np.int64)])).astype(np.float64)
    cdf = (1.0 - edge ** (1.0 - s)) / (1.0 - float(rows + 1) ** (1.0 - s))
    count, p = np.diff(edge), np.diff(cdf) / np.diff(edge)
    return float(np.sum(count * -np.expm1(-n * p)))


def work(case):
    kind = case["kind"]
    if kind == "train":
        n, dim, u = case["n"], case["dim"], _distinct(case["n"], case["zipf"], case["rows"])
        width = dim * (1 + SLOTS[case["opt"]])
        # gradients read, distinct rows read and written by the update, read by the pull; keys read; rows delivered
        return {"bytes": n // case["bag"] * dim * 4 + u * (2 * width + dim) * 4 + 8 * n + n // case["bag"] * dim * (2 if case["bf16"] else 4),
                "flops": float(n * dim * 2)}
    if kind == "lookup":
        n, dim = case["bags"] * case["bag"], case["dim"]
        u = _distinct(n, case["zipf"], case["rows"])
        return {"bytes": 8 * n + u * (dim * 4 + 16) + case["bags"] * dim * (2 if case["bf16"] else 4), "flops": float(n * dim)}
    if kind == "dense":
        p = sum(int(np.prod(s)) for s in _dense_shapes(case).values())
        return {"bytes": p * ((2 if case["bf16"] else 4) + 24 + 2), "flops": 20.0 * p}
    if kind == "mlp":
        w, b = _widths(case), case["batch"]
        weights, acts = sum(w[i] * w[i + 1] for i in range(len(w) - 1)), sum(w)
        return {"bytes": b * 2 * (w[0] * 2 + 2 * sum(w[1:])) + weights * (2 + 4), "flops": 6.0 * b * weights + 2.0 * b * acts}
    if kind == "linear":
        m, k, n = case["tokens"], case["d_in"], case["d_out"]
        return {"bytes": 2 * (2 * m * k + 2 * m * n + n * k) + 4 * n * k, "flops": 6.0 * m * n * k}
    b, d, f = case["batch"], CTR.emb_dim, CTR.num_sparse
    shapes, _ = _dlrm_shapes()
    p = sum(int(np.prod(s)) for s in shapes.values())
    u = 0.47 * b * f
    # rows and their slot read and written by the push, read by the pull, row gradients written, parameters and their
    # moments, activations once each way
    return {"bytes": u * (5 * d * 4) + b * f * (8 + d * 4) + p * 30 + b * 2 * 2 * (sum(CTR.bottom) + sum(CTR.top) + 512), "flops": 6.0 * b * p}


def tolerance(case):
    kind = case["kind"]
    if kind == "train":
        # sums of gradients in fp32 in any order: the hottest key of the largest batch has 200 000 of them, and two runs
        # of one implementation differ by 4e-6 there; a bf16 row is rounded once, so an update that lies near the middle of
        # two values may land on either
        return {"rel": 1e-3} if case["bf16"] else {"rel": 2e-5}
    if kind == "lookup":
        return {"rel": 1e-3} if case["bf16"] else {"rel": 1e-6}
    if kind == "dense":
        return {"rel": 1e-3}
    if kind == "mlp":
        return {"rel": 8e-3}
    if kind == "linear":
        return {"rel": 2e-3}
    return {"rel": 2e-2}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------
class _Kept(torch.autograd.Function):
    """A tensor that is kept in bf16, as its gradient is: sums are exact, but what one layer hands to the next is not wider
    than what the layers are defined on (a ReLU that sees another value than its neighbour passes another gradient)."""

    @staticmethod
    def forward(ctx, x, grad_too=True):
        ctx.grad_too = grad_too
        return x.to(torch.bfloat16).to(x.dtype)

    @staticmethod
    def backward(ctx, g):
        return (g.to(torch.bfloat16).to(g.dtype) if ctx.grad_too else g), None


def _update(opt, w, s0, s1, g):
    """One optimizer step on float64 tensors; returns the new weight."""
    if opt == "sgd":
        return w - 0.05 * g
    if opt == "adagrad":
        return w - 0.05 * g / ((s0 + g * g).sqrt() + 1e-10)
    if opt == "ftrl":
        o = OPT["ftrl"]
        n_new = s1 + g * g
        z = s0 + g - (n_new.sqrt() - s1.sqrt()) / o["alpha"] * w
        step = (torch.sign(z) * o["l1"] - z) / ((o["beta"] + n_new.sqrt()) / o["alpha"] + o["l2"])
        return torch.where(z.abs() <= o["l1"], torch.zeros_like(z), step)
    m, v = 0.9 * s0 + 0.1 * g, 0.999 * s1 + 0.001 * g * g
    return w - 1e-3 * (m / (1 - 0.9)) / ((v / (1 - 0.999)).sqrt() + 1e-8)


def _exact_rows(case, seed, uniq, width):
    """float64 rows of the sorted distinct ranks ``uniq`` (unknown ranks: zero)."""
    rows = torch.zeros((uniq.numel(), width), dtype=torch.float64, device="cuda")
    for lo in range(0, case["rows"], CHUNK):
        hi = min(case["rows"], lo + CHUNK)
        a, b = torch.searchsorted(uniq, torch.tensor([lo, hi], device="cuda")).tolist()
        if b > a:
            rows[a:b] = _rows_of(case, seed, lo, hi, width)[uniq[a:b] - lo].double()
    return rows


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        ranks, grads = _train_inputs(case, seed)
        dim, bag = case["dim"], case["bag"]
        uniq, inv = torch.unique(ranks, return_inverse=True)
        rows = _exact_rows(case, seed, uniq, dim * (1 + SLOTS[case["opt"]]))
        total = torch.zeros((uniq.numel(), dim), dtype=torch.float64, device="cuda")
        for j in range(bag):
            total.index_add_(0, inv[j::bag], grads.double())
        part = [rows[:, k * dim:(k + 1) * dim] if k <= SLOTS[case["opt"]] else None for k in range(3)]
        w = _update(case["opt"], part[0], part[1], part[2], total)
        out = w[inv[0::bag]]
        for j in range(1, bag):
            out += w[inv[j::bag]]
        return out
    if kind == "lookup":
        ranks = _lookup_ranks(case, seed)
        uniq, inv = torch.unique(ranks, return_inverse=True)
        w = _exact_rows(case, seed, uniq, case["dim"])
        out = torch.zeros((case["bags"], case["dim"]), dtype=torch.float64, device="cuda")
        for j in range(case["bag"]):
            out += w[inv[j::case["bag"]]]
        return out / case["bag"] if case["mean"] else out
    if kind == "dense":
        values = _dense_values(case, seed)
        o, new = DENSE_OPT, {}
        for k, (w, g) in values.items():
            w, g = w.double(), g.double()
            new[k] = w * (1 - o["lr"] * o["weight_decay"]) - o["lr"] * g / (g.abs() + 1e-8)
        # every tensor starts on a 64-element boundary of the flat buffer, whose length is a multiple of 8
        flat = torch.cat([torch.nn.functional.pad(v.reshape(-1), (0, -v.numel() % 64)) for v in new.values()])
        return dict(params=new, master=flat)
    if kind == "mlp":
        s = _mlp_inputs(case, seed)
        n = len(s["w"])
        w, b, act = [t.double() for t in s["w"]], [t.double() for t in s["b"]], []
        for i in range(n):
            act.append(_Kept.apply(torch.relu((act[-1] if act else s["x"].double()) @ w[i].t() + b[i])))
        dz, dw, db = [None] * (n - 1) + [s["dy"].double()], [None] * n, [None] * n
        for i in range(n - 1, -1, -1):
            dw[i], db[i] = dz[i].t() @ (act[i - 1] if i else s["x"].double()), dz[i].sum(0)
            d = dz[i] @ w[i]
            if i:
                dz[i - 1] = _Kept.apply(d * (act[i - 1] > 0))
        return dict(act=act, dz=dz[:-1], dx=d, dw=dw, db=db)
    if kind == "linear":
        s = {k: v.double() for k, v in _linear_inputs(case, seed).items()}
        return dict(y=s["x"] @ s["w"].t() + s["b"], dx=s["dy"] @ s["w"], dw=s["dy"].t() @ s["x"])
    batch, weights, uniq, rows = _dlrm_inputs(case, seed)
    dense, keys, labels = (t.cuda() for t in batch)
    b, d, f = case["batch"], CTR.emb_dim, CTR.num_sparse
    p = {k: v.double().requires_grad_(True) for k, v in weights.items()}
    _, n_inter = _dlrm_shapes()
    x = torch.nn.functional.pad(dense, (0, p["bot.w0"].shape[1] - CTR.num_dense)).to(torch.bfloat16).double()
    for i in range(len(CTR.bottom)):
        x = _Kept.apply(torch.relu(_Kept.apply(x @ p["bot.w%d" % i].t() + p["bot.b%d" % i])))
    emb = rows[torch.searchsorted(uniq, keys.reshape(-1)), :d].double().requires_grad_(True)
    t = torch.cat([x[:, None, :], _Kept.apply(emb, False).view(b, f, d)], dim=1)
    i, j = torch.tril_indices(f + 1, f + 1, offset=-1, device="cuda")
    h = _Kept.apply(torch.cat([x, (t @ t.transpose(1, 2))[:, i, j]], dim=1))
    h = torch.nn.functional.pad(h, (0, p["top.w0"].shape[1] - n_inter))
    for i in range(len(CTR.top)):
        h = _Kept.apply(torch.relu(_Kept.apply(h @ p["top.w%d" % i].t() + p["top.b%d" % i])))
    z = h @ p["head.w"] + p["head.b"]
    loss = torch.nn.functional.binary_cross_entropy_with_logits(z, labels.double())
    loss.backward()
    flat = torch.cat([torch.nn.functional.pad(v.grad.reshape(-1), (0, -v.numel() % 64)) for v in p.values()])
    return dict(loss=loss.detach().reshape(1), dense_grads=flat, row_grads=emb.grad)
