r"""
The calls that performance work on this framework is measured by.

A case is one pass through the public entry points (``FMoETransformerMLP``, ``FMoELinear``, ``FMoE``
with the user's own expert modules, the gates, ``GraphedStep``) on one GPU.  ``listed()`` names
twelve of them, ``draw()`` gives more of the same ranges.

The fields of a case:

* ``kind``: ``mlp`` (``FMoETransformerMLP``), ``linear`` (``FMoELinear`` on rows the caller has
  grouped, counts on the host) or ``custom`` (``FMoE`` around user modules);
* ``mode``: ``train`` is forward and backward with a gradient arriving at the output, as in the middle
  of a network, and returns the output and every gradient; ``infer`` is a forward without autograd;
* ``graph``: the same step captured once and replayed by ``GraphedStep``;
* ``tokens`` (rows for ``linear``), ``d``, ``h``, ``experts``, ``k``, ``dtype``, ``gate``, ``act``, and ``zipf``,
  the exponent of the gate bias that skews expert popularity (0 = near-uniform routing).
"""
import math
import random
from functools import partial

import torch
import torch.nn as nn

from fastmoe_b200 import FMoE, FMoELinear, FMoETransformerMLP
from fastmoe_b200.gates import GShardGate, NaiveGate, SwitchGate
from fastmoe_b200.utils.graph import GraphedStep

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}
# The random parts of the training-time gates (GShard's random second expert, Switch's jitter) are
# turned off by the gates' own options, so that a pass depends on its inputs alone.
GATES = {"naive": NaiveGate, "gshard": partial(GShardGate, random_routing=False),
         "switch": partial(SwitchGate, switch_eps=0.0)}
CAPACITY = {"train": 1.2, "infer": 2.4}   # the gates' defaults


def _case(name, kind, mode, tokens, d, h, experts, k=2, dtype="bf16", gate="naive", act="gelu",
          zipf=0.0, graph=False):
    c = dict(kind=kind, mode=mode, tokens=tokens, d=d, h=h, experts=experts, k=k, dtype=dtype, gate=gate,
             act=act, zipf=zipf, graph=graph)
    return dict(c, name=name) if name else c


def listed():
    return [
        # A small layer in an eager training loop, the size of the tests and the smoke run: what a
        # pass costs when there is next to nothing to compute.
        _case("train_small", "mlp", "train", 512, 256, 512, 4),
        # The benchmark's headline layer, replayed from a graph as the benchmark does.
        _case("train_layer_graph", "mlp", "train", 4096, 1024, 4096, 2, graph=True),
        # The benchmark's skewed, capacity-limited layer: most slots dropped, most experts idle.
        _case("train_skewed_gshard", "mlp", "train", 8192, 2048, 8192, 8, gate="gshard", zipf=1.2),
        # The feed-forward block of the benchmark's GPT: top-1 Switch gate with skewed popularity,
        # here in fp16.
        _case("train_switch_fp16", "mlp", "train", 8192, 1024, 4096, 2, k=1, dtype="fp16", gate="switch", zipf=1.2),
        # The reference harness's layer (examples/benchmark_mlp.py): 64 experts with 128 rows each.
        _case("train_many_experts", "mlp", "train", 4096, 1024, 4096, 64),
        # The feed-forward block of the Transformer-XL example: 22 sequences of 512 tokens, and
        # ReLU followed by a Dropout module (at p = 0) between the two linears.
        _case("train_relu_dropout", "mlp", "train", 11264, 512, 2048, 8, act="relu_dropout"),
        # A layer as the constructor leaves it: fp32 parameters and inputs.
        _case("train_fp32", "mlp", "train", 2048, 512, 2048, 8, dtype="fp32"),
        # One decoding step of a small batch, eager: latency.
        _case("decode_8", "mlp", "infer", 8, 1024, 4096, 8),
        # A decoding step over many experts from a graph: the weights' bytes.
        _case("decode_64_graph", "mlp", "infer", 64, 1024, 4096, 64, graph=True),
        # The prompt of a request: an odd number of tokens.
        _case("prefill_fp16", "mlp", "infer", 3001, 1024, 4096, 8, dtype="fp16"),
        # The grouped linear by itself in a user's own expert: ragged host-side counts.
        _case("linear_ragged", "linear", "train", 6007, 1024, 4096, 16),
        # The general layer around user-defined expert modules.
        _case("custom_experts", "custom", "train", 2048, 512, 2048, 8),
    ]


def draw(rng):
    most = {m: max(work(c)[m] for c in listed()) for m in ("flops", "bytes")}
    while True:
        c = _draw(rng)
        w = work(c)
        # a capacity of zero rows (GShard with fewer tokens than experts) leaves nothing to do
        if all(w[m] <= most[m] for m in most) and sum(_loads(c)) > 0:
            return c


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw(rng):
    kind = rng.choice(["mlp"] * 6 + ["linear", "custom"])
    mode = rng.choice(["train", "train", "infer"]) if kind == "mlp" else "train"
    dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
    if kind == "custom":
        dtype = rng.choice(["bf16", "fp32"])
    d = 64 * _log(rng, 2, 32)
    h = min(8192, d * rng.choice([2, 4, 4]))
    experts = rng.choice([2, 4, 8, 16, 32, 64])
    if dtype == "fp32":
        d, h = rng.choice([(d // 4, h // 4), (min(d, 1024), min(h, 4096))])
    if kind == "custom":
        experts = min(experts, 8)
    gate, k = "naive", rng.choice([1, 2, 2, 2, 4])
    k = min(k, experts)
    if kind == "mlp" and rng.random() < 0.4:
        gate, k = rng.choice([("gshard", 2), ("switch", 1)])
    act = rng.choice(["gelu", "gelu", "relu", "relu_dropout"]) if kind == "mlp" else "gelu"
    zipf = 1.2 if kind == "mlp" and rng.random() < 0.3 else 0.0
    tokens = _log(rng, 1, 16384) if mode == "infer" else _log(rng, 64, 16384)
    graph = kind == "mlp" and dtype != "fp32" and rng.random() < 0.4
    return _case(None, kind, mode, tokens, d, h, experts, k, dtype, gate, act, zipf, graph)


# ------------------------------------------------------------------------------ what a user holds
class MLPExpert(nn.Module):
    r"""A user-defined expert: called with its rows and their count."""

    def __init__(self, d, h):
        super().__init__()
        self.fc1, self.fc2 = nn.Linear(d, h), nn.Linear(h, d)

    def forward(self, x, _count):
        return self.fc2(nn.functional.gelu(self.fc1(x)))


def _activation(act):
    if act == "relu_dropout":
        return nn.Sequential(nn.ReLU(), nn.Dropout(0.0))
    return nn.ReLU() if act == "relu" else nn.GELU()


def _layer(case):
    d, h, experts = case["d"], case["h"], case["experts"]
    if case["kind"] == "linear":
        layer = FMoELinear(experts, d, h)
    elif case["kind"] == "custom":
        layer = FMoE(num_expert=experts, d_model=d, top_k=case["k"], expert=lambda width: MLPExpert(width, h))
    else:
        layer = FMoETransformerMLP(num_expert=experts, d_model=d, d_hidden=h, top_k=case["k"],
                                   gate=GATES[case["gate"]], activation=_activation(case["act"]))
        if case["zipf"] > 0:
            with torch.no_grad():
                layer.gate.gate.weight.mul_(0.1)
                layer.gate.gate.bias.copy_(-case["zipf"] * torch.arange(1, experts + 1.0).log())
    return layer


def _row_counts(case, seed):
    r"""How many rows each expert of a ``linear`` case has: ragged, one expert without any."""
    rng = random.Random(seed)
    rows, experts = case["tokens"], case["experts"]
    weight = [rng.uniform(0.2, 1.8) for _ in range(experts)]
    weight[rng.randrange(experts)] = 0.0
    counts = [int(rows * w / sum(weight)) for w in weight]
    counts[max(range(experts), key=lambda e: weight[e])] += rows - sum(counts)
    return torch.tensor(counts, dtype=torch.int64)


def _drawn(case, seed):
    r"""The layer with its weights, the input rows and the gradient that arrives at the output."""
    torch.manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    with torch.device("cuda"):
        layer = _layer(case).to(dtype)
        x = torch.randn(case["tokens"], case["d"]).to(dtype)
        gy = torch.randn(case["tokens"], case["h"] if case["kind"] == "linear" else case["d"]).to(dtype)
    return layer, x, gy


def prepare(case, seed):
    layer, x, gy = _drawn(case, seed)
    layer.train(case["mode"] == "train")
    held = {"layer": layer, "gy": gy, "aux": case["gate"] != "naive"}
    if case["kind"] == "linear":
        held["counts"] = _row_counts(case, seed)
    step = partial(_train if case["mode"] == "train" else _infer, held)
    return {"layer": layer, "x": x, "step": GraphedStep(step, x) if case["graph"] else step}


# ------------------------------------------------------------------------------ one pass
def _call(held, x):
    return held["layer"](x, held["counts"]) if "counts" in held else held["layer"](x)


def _infer(held, x):
    with torch.no_grad():
        return _call(held, x)


def _train(held, x):
    layer = held["layer"]
    layer.zero_grad(set_to_none=True)
    x = x.detach().requires_grad_(True)
    y = _call(held, x)
    roots, grads = [y], [held["gy"]]
    if held["aux"]:   # the gate's balance loss joins the training loss
        roots.append(layer.gate.get_loss())
        grads.append(None)
    torch.autograd.backward(roots, grads)
    return {"y": y.detach(), "dx": x.grad, "grads": {n: p.grad for n, p in layer.named_parameters()}}


def run(state):
    return state["step"](state["x"])


# ------------------------------------------------------------------------------ in 64 bits
def _keep_within(ids, experts, cap):
    r"""``ids`` with every slot beyond the first ``cap`` of its expert (in slot order) set to -1."""
    one = nn.functional.one_hot(ids.reshape(-1), experts)
    rank = (one.cumsum(0) * one).sum(1) - 1
    return torch.where(rank < cap, ids.reshape(-1), -1).view_as(ids)


def _exact_gate(case, x, w, b):
    r"""Expert ids and scores ``[tokens, k]`` and the balance loss (or ``None``).  Which experts a
    token goes to is decided on logits rounded to the layer's type, ties to the lower id, as any
    implementation that holds them in that type does; the scores are those of the unrounded ones."""
    n, experts, k, mode = case["tokens"], case["experts"], case["k"], case["mode"]
    logits = x @ w.t() + b
    rounded = logits.detach().to(DTYPES[case["dtype"]])
    ids = rounded.sort(dim=1, descending=True, stable=True).indices[:, :k]
    prob = torch.softmax(logits, dim=1)
    if case["gate"] == "switch":
        kept = _keep_within(ids, experts, math.ceil(CAPACITY[mode] * n / experts))
        share = nn.functional.one_hot(kept[kept >= 0], experts).sum(0)
        n_kept = share.sum().clamp(min=1)
        return kept, prob.gather(1, ids), experts * ((share / n_kept) * (prob.sum(0) / n_kept)).sum()
    score = torch.softmax(logits.gather(1, ids), dim=1)
    if case["gate"] == "gshard":
        share = nn.functional.one_hot(ids[:, 0], experts).sum(0) / n
        loss = (share * prob.mean(0)).mean() * experts ** 2
        return _keep_within(ids, experts, math.ceil(CAPACITY[mode] * n) * k // experts), score, loss
    return ids, score, None


def exact(case, seed):
    layer, x, gy = _drawn(case, seed)
    train, experts, kind = case["mode"] == "train", case["experts"], case["kind"]
    par = {n: p.detach().double().requires_grad_(train) for n, p in layer.named_parameters()}
    x, gy = x.double().requires_grad_(train), gy.double()
    act = nn.functional.gelu if case["act"] == "gelu" else torch.relu
    loss = None
    if kind == "linear":
        rows = x.split(_row_counts(case, seed).tolist())
        y = torch.cat([r @ par["weight"][e].t() + par["bias"][e] for e, r in enumerate(rows)])
    else:
        ids, score, loss = _exact_gate(case, x, par["gate.gate.weight"], par["gate.gate.bias"])
        y = torch.zeros_like(x)
        for e in range(experts):
            token, slot = (ids == e).nonzero(as_tuple=True)
            if kind == "custom":
                w1, b1, w2, b2 = (par["experts.%d.%s" % (e, n)] for n in
                                  ("fc1.weight", "fc1.bias", "fc2.weight", "fc2.bias"))
            else:
                w1, b1, w2, b2 = (par["experts.%s" % n][e] for n in
                                  ("htoh4.weight", "htoh4.bias", "h4toh.weight", "h4toh.bias"))
            out = act(x[token] @ w1.t() + b1) @ w2.t() + b2
            y = y.index_add(0, token, out * score[token, slot, None])
    if not train:
        return y
    torch.autograd.backward([y] if loss is None else [y, loss], [gy] if loss is None else [gy, None])
    return {"y": y.detach(), "dx": x.grad, "grads": {n: p.grad for n, p in par.items()}}


# ------------------------------------------------------------------------------ what it needs
def _loads(case):
    r"""Expected rows of every expert, after the gate's capacity limit."""
    n, experts, k = case["tokens"], case["experts"], case["k"]
    if case["kind"] == "linear":
        return [n / experts] * experts
    if case["zipf"] > 0:
        loads = [n] * k + [0] * (experts - k)   # the bias outweighs the scaled-down gate weights
    else:
        loads = [n * k / experts] * experts
    cap = n
    if case["gate"] == "gshard":
        cap = math.ceil(CAPACITY[case["mode"]] * n) * k // experts
    elif case["gate"] == "switch":
        cap = math.ceil(CAPACITY[case["mode"]] * n / experts)
    return [min(cap, v) for v in loads]


def work(case):
    n, d, h, experts = case["tokens"], case["d"], case["h"], case["experts"]
    train, size = case["mode"] == "train", BYTES[case["dtype"]]
    loads = _loads(case)
    rows = sum(loads)
    # experts that get at least one row: those whose weights have to be read
    active = sum(1 - (1 - 1 / experts) ** rows if case["zipf"] == 0 else v > 0 for v in loads)
    if case["kind"] == "linear":
        flops, per_expert, gate, io = 2 * rows * d * h, d * h + h, 0, n * (d + h)
    else:
        flops, per_expert, gate = 4 * rows * d * h + 2 * n * d * experts, 2 * d * h + d + h, experts * d
        io = 2 * n * d
    elems = io + active * per_expert + gate
    if train:   # the gradients of input and output, and every expert's weight gradient
        flops *= 3
        elems += io + experts * per_expert + gate
    return {"bytes": float(size * elems), "flops": float(flops)}


# About four times what the outputs move by when the hidden units of every expert are permuted (the
# sums of the second linear, of the input gradient and of the gate's gradient in another order):
# at most 2.1e-3 and 2.1e-2 in bf16, 3.8e-4 and 2.7e-3 in fp16, 1.1e-6 and 8.9e-6 in fp32, over the
# listed cases.
TOLERANCE = {"bf16": {"rel": 1e-2, "max": 1e-1}, "fp16": {"rel": 2e-3, "max": 1.5e-2},
             "fp32": {"rel": 1e-5, "max": 5e-5}}


def tolerance(case):
    return dict(TOLERANCE[case["dtype"]])
