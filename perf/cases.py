"""The multi-LoRA work that a serving program has this package do, as cases with sizes.

A case is one step (or one call) of such a program.  ``path`` says through which entry points:

* ``static``  one ``add_lora_bgmv_static`` call: a decode token or a few in a process that may not allocate;
* ``op``      a decode step in the reference's call pattern: ``add_lora_bgmv`` three times (q, k, v) per layer on
              dense pools of one rank, the same index tensor all along;
* ``call``    one ``add_lora_sgmv`` call on adapter-sorted prompts, everything set up inside the call;
* ``mirror``  the ``Lora_GPU`` layer object: ``set_indices`` and the q, k and v calls of every layer (decode), or
              those calls on ``[B, L, H]`` prompts (prefill, with the reference's rounding of the intermediate);
* ``fused``   plan once per step, then per layer one apply for q/k/v and one for o, on a packed (or padded dense)
              pool with per-adapter ranks; decode, prefill or both in one batch; called eagerly or, with
              ``graph``, captured once and replayed, as decode loops do.

Which adapters are in a batch, how many rows each has, and the ranks follow from the case; their order in the
batch, the activations and the weights follow from the seed.  Activations are N(0, 1), A is N(0, 1/h_in), B is
N(0, 1/r), an adapter's scaling is 32/r, and y holds an N(0, 1) base projection that the delta is added to.
Every layer has activations of its own, so that weights and activations come from HBM as they do between the
base model's kernels.
"""
import math
import random

import numpy as np
import torch

import ae296_b200 as b200
from ae296_b200.batching import plan_for_requests

ALPHA = 32.0
ELEM = 2
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def listed():
    return [
        # one token of one request, one projection: the smallest call there is, latency only
        dict(name="static-1tok", path="static", phase="decode", dtype="fp16", hidden=4096, kv=4096, layers=1,
             tokens=1, adapters=8, ranks="16", alpha=0.0, pool="dense", prompts=0, longest=0, graph=False),
        # a lightly loaded server on the reference's operator: odd batch, few adapters, 96 calls
        dict(name="op-decode-7", path="op", phase="decode", dtype="fp16", hidden=4096, kv=4096, layers=32,
             tokens=7, adapters=16, ranks="16", alpha=1.0, pool="dense", prompts=0, longest=0, graph=False),
        # one projection of three ragged prompts by the one-call form
        dict(name="call-3prompts", path="call", phase="prefill", dtype="fp16", hidden=4096, kv=4096, layers=1,
             tokens=0, adapters=8, ranks="8,16,32,64", alpha=0.0, pool="packed", prompts=3, longest=700, graph=False),
        # the layer object at its usual decode batch, indices new in every step
        dict(name="mirror-decode-32", path="mirror", phase="decode", dtype="fp16", hidden=4096, kv=4096, layers=16,
             tokens=32, adapters=32, ranks="16", alpha=1.0, pool="dense", prompts=0, longest=0, graph=False),
        # the layer object on four padded prompts of an odd length
        dict(name="mirror-prefill-4x509", path="mirror", phase="prefill", dtype="fp16", hidden=4096, kv=4096,
             layers=16, tokens=0, adapters=4, ranks="16", alpha=0.0, pool="dense", prompts=4, longest=509,
             graph=False),
        # a single user's decode step, replayed: launches and their gaps
        dict(name="decode-1-graph", path="fused", phase="decode", dtype="bf16", hidden=4096, kv=4096, layers=32,
             tokens=1, adapters=64, ranks="16", alpha=0.0, pool="packed", prompts=0, longest=0, graph=True),
        # a full decode batch of mixed ranks, Zipf popularity
        dict(name="decode-256", path="fused", phase="decode", dtype="fp16", hidden=4096, kv=4096, layers=32,
             tokens=256, adapters=128, ranks="8,16,32,64", alpha=1.0, pool="packed", prompts=0, longest=0,
             graph=False),
        # grouped-query shapes (narrow k and v), rank 64, large batch, replayed: the longest decode launches
        dict(name="decode-512-gqa-graph", path="fused", phase="decode", dtype="bf16", hidden=8192, kv=1024,
             layers=16, tokens=512, adapters=128, ranks="64", alpha=1.2, pool="packed", prompts=0, longest=0,
             graph=True),
        # adapters of any rank in the padded dense pool
        dict(name="decode-93-padded", path="fused", phase="decode", dtype="fp16", hidden=4096, kv=4096, layers=32,
             tokens=93, adapters=32, ranks="8,12,16,24,48,64", alpha=1.0, pool="dense", prompts=0, longest=0,
             graph=False),
        # one short prompt arriving alone: time to first token
        dict(name="prefill-1prompt", path="fused", phase="prefill", dtype="bf16", hidden=4096, kv=4096, layers=32,
             tokens=0, adapters=8, ranks="32", alpha=0.0, pool="packed", prompts=1, longest=333, graph=False),
        # a full prefill batch, one adapter per prompt
        dict(name="prefill-16prompts", path="fused", phase="prefill", dtype="fp16", hidden=4096, kv=4096, layers=32,
             tokens=0, adapters=16, ranks="32", alpha=0.0, pool="packed", prompts=16, longest=1024, graph=False),
        # decode tokens and prompts in one batch, wider model
        dict(name="mixed-448-4prompts", path="fused", phase="mixed", dtype="bf16", hidden=5120, kv=5120, layers=40,
             tokens=448, adapters=128, ranks="16,32,64", alpha=1.0, pool="packed", prompts=4, longest=512,
             graph=False),
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5))))))


def draw(rng):
    most = max(work(c)["bytes"] for c in listed())
    while True:
        c = _draw_one(rng)
        if work(c)["bytes"] <= most and _state_bytes(c) <= 30e9:
            return c


def _draw_one(rng):
    path, phase = rng.choice([("static", "decode"), ("op", "decode"), ("call", "prefill"), ("mirror", "decode"),
                              ("mirror", "prefill"), ("fused", "decode"), ("fused", "decode"), ("fused", "prefill"),
                              ("fused", "mixed")])
    c = dict(path=path, phase=phase, dtype=rng.choice(["fp16", "bf16"]), tokens=0, prompts=0, longest=0,
             alpha=rng.choice([0.0, 1.0, 1.2]), graph=False)
    c["hidden"], c["kv"] = rng.choice([(2048, 2048), (4096, 4096), (4096, 1024), (5120, 5120), (8192, 1024)])
    if path == "static":
        c.update(layers=1, tokens=_log_int(rng, 1, 64), adapters=_log_int(rng, 1, 128), pool="dense",
                 ranks=rng.choice(["8", "16", "32", "64"]))
    elif path == "op":
        c.update(layers=_log_int(rng, 4, 40), tokens=_log_int(rng, 1, 256), adapters=_log_int(rng, 1, 128),
                 pool="dense", ranks=rng.choice(["8", "16", "32", "64"]))
    elif path == "call":
        c.update(layers=1, adapters=_log_int(rng, 1, 32), pool="packed", prompts=_log_int(rng, 1, 12),
                 longest=_log_int(rng, 32, 1024), ranks=rng.choice(["16", "32", "64", "8,16,32,64"]))
    elif path == "mirror":
        c["kv"] = c["hidden"]                               # the layer object has one output width
        c.update(layers=_log_int(rng, 4, 20), pool="dense", ranks=rng.choice(["8", "16", "32", "64"]))
        if phase == "decode":
            c.update(tokens=_log_int(rng, 1, 128))
            c["adapters"] = c["tokens"]                     # its pool has one slot for each row of the batch
        else:
            c.update(prompts=_log_int(rng, 1, 8), longest=_log_int(rng, 16, 1024))
            c["adapters"] = c["prompts"]
    else:
        c.update(layers=_log_int(rng, 8, 40), adapters=_log_int(rng, 2, 256),
                 ranks=rng.choice(["8", "16", "32", "64", "16,32,64", "8,16,32,64", "8,12,16,24,48,64"]))
        c["pool"] = "dense" if "12" in c["ranks"] else "packed"
        if phase in ("decode", "mixed"):
            c["tokens"] = _log_int(rng, 1 if phase == "decode" else 16, 512)
            c["graph"] = phase == "decode" and rng.random() < 0.5
        if phase in ("prefill", "mixed"):
            c.update(prompts=_log_int(rng, 1, 16 if phase == "prefill" else 6), longest=_log_int(rng, 48, 1024))
    return c


# ---- what a case fixes: ranks, rows per adapter --------------------------------------------------
def _layout(case):
    """ranks [N]; adapter of each decode row; (length, adapter) of each prompt.  Independent of the seed."""
    n, t, p = case["adapters"], case["tokens"], case["prompts"]
    rng = np.random.default_rng([n, t, p, case["longest"]])
    ranks = rng.choice([int(r) for r in case["ranks"].split(",")], n).astype(np.int32)
    pop = 1.0 / np.arange(1, n + 1, dtype=np.float64) ** case["alpha"]
    ids = rng.choice(n, t, p=pop / pop.sum()).astype(np.int32)
    if case["path"] == "mirror":
        return ranks, ids, np.full(p, case["longest"]), np.arange(p, dtype=np.int32)     # slot b is request b
    lens = rng.integers(max(1, case["longest"] // 8), case["longest"] + 1, p)
    lens[:1] = case["longest"]
    owner = rng.permutation(np.arange(p) % n).astype(np.int32)
    return ranks, ids, lens, owner


def _groups(case):
    """(h_in, output widths) of the inputs that a layer's projections share."""
    h, kv = case["hidden"], case["kv"]
    if case["path"] in ("static", "call"):
        return [(h, [h])]
    if case["path"] in ("op", "mirror"):
        return [(h, [h, kv, kv])]
    return [(h, [h, kv, kv]), (h, [h])]


def work(case):
    """Every used adapter's A and B once, x once, y read and written (only written where the path makes it), ids."""
    ranks, ids, lens, owner = _layout(case)
    rows = np.concatenate([ids, np.repeat(owner, lens)]).astype(np.int64)
    t, used = len(rows), int(ranks[np.unique(rows)].sum())
    row_ranks = int(ranks[rows].sum())
    nbytes = flops = 0
    for h_in, outs in _groups(case):
        nbytes += t * h_in * ELEM
        for h_out in outs:
            nbytes += used * (h_in + h_out) * ELEM + (1 if case["path"] == "mirror" else 2) * t * h_out * ELEM
            flops += 2 * row_ranks * (h_in + h_out)
    return {"bytes": case["layers"] * nbytes + 4 * t, "flops": case["layers"] * flops}


def _state_bytes(case):
    ranks, ids, lens, _ = _layout(case)
    t = len(ids) + int(lens.sum())
    per_rank = int(ranks.sum()) if case["pool"] == "packed" else len(ranks) * int(ranks.max())
    return ELEM * case["layers"] * sum(per_rank * (h_in + h) + t * (h_in + h) for h_in, outs in _groups(case) for h in outs)


def tolerance(case):
    """One rounding of y to 16 bits is 2^-12 (fp16) or 2^-9 (bf16) of it on the average; where the intermediate is
    rounded too, another of the same size."""
    return {"rel": 1e-3 if case["dtype"] == "fp16" else 8e-3}


# ---- states --------------------------------------------------------------------------------------
def _fill_normal(g, t, std=1.0):
    return t.normal_(0.0, std, generator=g)


def _pool(case, ranks, h_in, h_out, g):
    pool = b200.AdapterPool.empty(len(ranks), case["layers"], h_in, h_out, ranks, ALPHA / ranks,
                                  dtype=DTYPES[case["dtype"]], device="cuda", dense=case["pool"] == "dense")
    _fill_normal(g, pool.wa, h_in ** -0.5)
    if len(set(ranks.tolist())) == 1:
        _fill_normal(g, pool.wb, float(ranks[0]) ** -0.5)
    else:
        _fill_normal(g, pool.wb)
        for a, r in enumerate(ranks):
            pool.b_block(a).mul_(float(r) ** -0.5)
    return pool


def prepare(case, seed):
    ranks, ids, lens, owner = _layout(case)
    order = np.random.default_rng(seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    order.shuffle(ids)
    if case["path"] != "mirror":
        turn = order.permutation(len(lens))
        lens, owner = lens[turn], owner[turn]
    t, layers = len(ids) + int(lens.sum()), case["layers"]
    s = {"case": case, "tokens": t}

    def i32(a):
        return torch.from_numpy(np.ascontiguousarray(a, np.int32)).cuda()

    if case["path"] == "mirror":
        decode = case["phase"] == "decode"
        lora = b200.Lora_GPU(dict(n_layers=layers, batch_size=case["adapters"] if decode else 1,
                                  lora_rank=int(ranks[0]), hidden_dim=case["hidden"], tp_degree=1,
                                  max_prefill_batch_size=1 if decode else case["prompts"]), dtype=dt)
        for p in "qkv":
            tail = "" if decode else "_prefill"
            _fill_normal(g, getattr(lora, f"{p}_down{tail}"), case["hidden"] ** -0.5)
            _fill_normal(g, getattr(lora, f"{p}_up{tail}"), ALPHA / ranks[0] * float(ranks[0]) ** -0.5)
        shape = (layers, t) if decode else (layers, case["prompts"], case["longest"])
        s["lora"], s["ids"] = lora, torch.from_numpy(ids.astype(np.int64)).cuda()
        s["xs"] = list(_fill_normal(g, torch.empty(*shape, case["hidden"], dtype=dt, device="cuda")))
        return s

    groups = _groups(case)
    pools = [[_pool(case, ranks, h_in, h, g) for h in outs] for h_in, outs in groups]
    xs = [_fill_normal(g, torch.empty(layers, t, h_in, dtype=dt, device="cuda")) for h_in, _ in groups]
    ys = [[torch.empty(layers, t, h, dtype=dt, device="cuda") for h in outs] for _, outs in groups]

    def base():
        gy = torch.Generator(device="cuda").manual_seed(seed + 1)
        for y in (y for group in ys for y in group):
            _fill_normal(gy, y)

    base()
    s["ys"] = [y for group in ys for y in group]
    s["pool"] = pools[0][0]
    s["calls"] = [[[(x[layer], y[layer], pool) for y, pool in zip(group, group_pools)]
                   for x, group, group_pools in zip(xs, ys, pools)] for layer in range(layers)]
    if case["path"] in ("static", "op"):
        s["scale"] = ALPHA / float(ranks[0])
        s["ids"] = torch.from_numpy(ids.astype(np.int64)).cuda()
    elif case["phase"] == "prefill":
        s["lora_ids"], s["seq_len"] = i32(owner), i32(lens)
        starts = np.concatenate([[0], np.cumsum(lens)])
        s["start_loc"], s["seg_starts"] = i32(starts[:-1]), i32(starts)
    else:
        s["ids"] = i32(np.concatenate([ids, np.repeat(owner, lens)]))
    if case["path"] == "fused":
        s["batch"] = b200.LoraBatch(t, len(ranks), case["hidden"], 3)
    if case["graph"]:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _step(s)
        torch.cuda.current_stream().wait_stream(side)
        s["replay"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["replay"]):
            _step(s)
        base()
    return s


# ---- one pass ------------------------------------------------------------------------------------
def _step(s):
    """The fused step of a batch: its plan, then every layer's q/k/v and o."""
    case, batch = s["case"], s["batch"]
    if case["phase"] == "prefill":
        plan_for_requests(batch, s["pool"], s["lora_ids"], s["start_loc"], s["seq_len"], s["tokens"], prefill=True)
    else:
        batch.set_ids(s["ids"], s["pool"], tiles=case["phase"] == "mixed")
    for layer, groups in enumerate(s["calls"]):
        for projs in groups:
            batch.apply(projs, layer)


def run(s):
    case = s["case"]
    if case["path"] == "static":
        (x, y, pool), = s["calls"][0][0]
        b200.add_lora_bgmv_static(y, x, pool.wa, pool.wb, s["ids"], 0, s["scale"])
    elif case["path"] == "op":
        for layer, (projs,) in enumerate(s["calls"]):
            for x, y, pool in projs:
                b200.add_lora_bgmv(y, x, pool.wa, pool.wb, s["ids"], layer, s["scale"])
    elif case["path"] == "call":
        (x, y, pool), = s["calls"][0][0]
        b200.add_lora_sgmv(y, x, pool, s["seg_starts"], s["lora_ids"], 0)
    elif case["path"] == "mirror":
        lora, prefill = s["lora"], case["phase"] == "prefill"
        if not prefill:
            lora.set_indices(s["ids"])
        outs = []
        for layer, x in enumerate(s["xs"]):
            outs += [lora.invoke_one_layer_q(x, layer, prefill), lora.invoke_one_layer_k(x, layer, prefill),
                     lora.invoke_one_layer_v(x, layer, prefill)]
        return outs
    elif case["graph"]:
        s["replay"].replay()
    else:
        _step(s)
    return s["ys"]
