"""Workloads of the MoE layer as its users run it, for timing one pass of each on one GPU.

A case is one ``FMoETransformerMLP`` (gate, routing, permutation, grouped expert products, combine) at one size:

* ``infer``: the forward pass under ``torch.no_grad()`` -- a decoding step (few tokens, the expert weights are
  most of the traffic) or a prefill (many tokens);
* ``train``: forward and backward launched from Python, the gradient of the output given, gradients of the input
  and of every parameter returned;
* ``graph``: the same step through ``GraphedStep`` (one CUDA graph replay per batch, loss = sum of the output).

Sizes are those of the benchmark workloads in ``bench.py``, of the tests, and generic ones between and below them.
Activations are N(0, 1), expert weights U(+-1/sqrt(fan_in)), gate weights N(0, 0.02) (near-uniform routing), with
``zipf`` > 0 a gate bias that gives expert r popularity about r^-zipf.
"""
import math

import torch

from fastermoe_b200 import FMoETransformerMLP, GraphedStep
from fastermoe_b200.gates import GShardGate, NaiveGate

DTYPES = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}
ACTIVATIONS = {"gelu": torch.nn.GELU, "relu": torch.nn.ReLU, "silu": torch.nn.SiLU}

#: What a drawn case may cost at most.  16-bit products of feature sizes that are multiples of 64 run on the tensor
#: cores; fp32 and other feature sizes are given less work, as their users give them.
MAX_FLOPS, MAX_FLOPS_SMALL = 2.0e13, 3.0e11
MAX_WEIGHTS = 32 * 2 * 2048 * 8192


def _case(name, mode, tokens, d_model, d_hidden, experts, top_k=2, dtype="bfloat16", act="gelu", gate="softmax",
          zipf=0.0, bias=True):
    c = dict(mode=mode, tokens=tokens, d_model=d_model, d_hidden=d_hidden, experts=experts, top_k=top_k, dtype=dtype,
             act=act, gate=gate, zipf=zipf, bias=bias)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one decoding step of a handful of sequences: launches and latency
        _case("decode_4", "infer", 4, 1024, 4096, 16),
        # one decoding step of a serving batch on a layer of 32 wide experts: every expert's weights are read
        _case("decode_96_wide", "infer", 96, 2048, 8192, 32, zipf=1.2),
        # a prompt of a few thousand tokens through the same layer
        _case("prefill_4096", "infer", 4096, 2048, 8192, 32, zipf=1.2),
        # the repository's headline training step
        _case("train_headline", "train", 16384, 1024, 4096, 16),
        # wide experts under skewed routing: long and very short segments in one launch
        _case("train_skewed", "train", 8192, 2048, 8192, 32, zipf=1.2),
        # the widest workload of the benchmark: two experts, long contractions
        _case("train_widest", "train", 16384, 4096, 16384, 2, act="relu", gate="naive", bias=False),
        # full precision, the size of the reference's own numerical tests and CPU baseline
        _case("train_fp32", "train", 2048, 512, 2048, 4, dtype="float32", gate="naive"),
        # half precision, an odd batch, widths of an ordinary encoder
        _case("train_fp16_odd_batch", "train", 3001, 768, 3072, 12, dtype="float16", act="relu", gate="naive"),
        # a small model whose widths are not multiples of a tensor-core tile
        _case("train_narrow", "train", 1999, 200, 712, 6, gate="naive"),
        # top-2 gate with capacity limit and balance loss
        _case("train_capacity", "train", 8192, 1024, 4096, 16, gate="gshard"),
        # many small experts, four per token, an activation applied between the two expert layers
        _case("train_many_experts", "train", 4096, 1024, 512, 64, top_k=4, act="silu", bias=False),
        # a small step replayed as a CUDA graph
        _case("graph_small", "graph", 512, 512, 2048, 8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        mode = rng.choice(["infer", "infer", "infer", "train", "train", "train", "train", "graph"])
        tokens = {"infer": lambda: _log_int(rng, 1, 8192), "train": lambda: _log_int(rng, 256, 16384),
                  "graph": lambda: _log_int(rng, 128, 4096)}[mode]()
        step = rng.choice([64, 64, 64, 256, 8])         # most models' widths are multiples of 64
        d_model = max(step, _log_int(rng, 128, 4096) // step * step)
        d_hidden = max(step, int(d_model * rng.choice([0.5, 1, 2, 3, 4, 4])) // step * step)
        experts = _log_int(rng, 2, 64)
        gate = rng.choice(["softmax", "softmax", "naive", "naive", "gshard"])
        top_k = 2 if gate == "gshard" or rng.random() < 0.6 else rng.choice([1, 3, 4, 6, 8])
        if top_k == 1 or experts < 4:
            gate = "naive"                      # one softmax over (nearly) all there is has (nearly) nothing to learn
        dtype = rng.choice(["bfloat16", "bfloat16", "bfloat16", "float16", "float32"])
        act = rng.choice(["gelu", "gelu", "relu", "silu"])
        case = _case(None, mode, tokens, d_model, d_hidden, experts, top_k, dtype, act, gate,
                     zipf=rng.choice([0.0, 0.0, 0.6, 1.2]), bias=rng.random() < 0.75)
        on_tiles = dtype != "float32" and d_model % 64 == 0 and d_hidden % 64 == 0 and min(d_model, d_hidden) >= 256
        if top_k <= experts and experts * 2 * d_model * d_hidden <= MAX_WEIGHTS and \
                work(case)["flops"] <= (MAX_FLOPS if on_tiles else MAX_FLOPS_SMALL):
            return case


def prepare(case, seed):
    dev, dtype = torch.device("cuda"), DTYPES[case["dtype"]]
    T, d, h, E = case["tokens"], case["d_model"], case["d_hidden"], case["experts"]
    g = torch.Generator(device=dev).manual_seed(seed)
    gate = GShardGate if case["gate"] == "gshard" else NaiveGate
    with dev:
        layer = FMoETransformerMLP(num_expert=E, d_model=d, d_hidden=h, top_k=case["top_k"], gate=gate,
                                   activation=ACTIVATIONS[case["act"]](), bias=case["bias"]).to(dtype)
        with torch.no_grad():
            layer.gate.gate.weight.copy_(torch.randn(E, d, generator=g) * 0.02)
            layer.gate.gate.bias.copy_(-case["zipf"] * torch.log(torch.arange(1, E + 1).float()))
            for lin, fan_in in ((layer.experts.htoh4, d), (layer.experts.h4toh, h)):
                for p in lin.parameters():
                    p.uniform_(-fan_in ** -0.5, fan_in ** -0.5, generator=g)
        x = torch.randn(T, d, generator=g, dtype=dtype)
        grad_out = torch.randn(T, d, generator=g, dtype=dtype)
    layer.gate.softmax_scores = case["gate"] == "softmax"
    if case["gate"] == "gshard":
        layer.gate.random_routing = False       # the second expert is kept or dropped by capacity alone
    state = {"layer": layer, "params": dict(layer.named_parameters()), "mode": case["mode"]}
    if case["mode"] == "infer":
        layer.eval()
        return dict(state, x=x)
    if case["mode"] == "graph":
        return dict(state, x=x, step=GraphedStep(layer, x, input_grad=True))
    return dict(state, x=x.requires_grad_(True), grad_out=grad_out)


def run(state):
    layer, x = state["layer"], state["x"]
    if state["mode"] == "infer":
        with torch.no_grad():
            return layer(x)
    if state["mode"] == "graph":
        step = state["step"]
        loss = step(x)
        return {"loss": loss, "out": step.output, "grad_x": step.input_grad,
                "grads": {n: p.grad for n, p in state["params"].items()}}
    x.grad = None
    layer.zero_grad(set_to_none=True)
    out = layer(x)
    balance = layer.gate.get_loss()             # the capacity gate's auxiliary loss, trained with the output
    if balance is None:
        out.backward(state["grad_out"])
    else:
        torch.autograd.backward([out, balance], [state["grad_out"], None])
    return {"out": out, "grad_x": x.grad, "grads": {n: p.grad for n, p in state["params"].items()}}


def touched_experts(case):
    """How many experts a pass is expected to choose at all: the share of tokens that choose each one, from 2048
    sampled rows of logits, then the chance that at least one of the case's tokens does."""
    E = case["experts"]
    logits = torch.randn(2048, E, generator=torch.Generator().manual_seed(0)) * (0.02 * case["d_model"] ** 0.5)
    logits -= case["zipf"] * torch.log(torch.arange(1, E + 1).float())
    chosen = torch.bincount(logits.topk(case["top_k"], dim=1)[1].reshape(-1), minlength=E).double() / 2048
    return float((1 - (1 - chosen).clamp(min=0) ** case["tokens"]).sum())


def work(case):
    """Bytes: every tensor that comes in read once, every one that goes out written once.  An expert that no token
    chose need not be read (its gradient is still written in training).  Flops: the gate's product and the two
    expert products of every (token, expert) pair, three times that in training."""
    T, d, h, E, k = (case[n] for n in ("tokens", "d_model", "d_hidden", "experts", "top_k"))
    size = DTYPES[case["dtype"]].itemsize
    touched = touched_experts(case)
    per_expert = 2 * d * h + (d + h if case["bias"] else 0)
    gate = E * (d + 1)
    flops = 2 * T * d * E + 4 * T * k * d * h
    if case["mode"] == "infer":
        return {"bytes": size * (2 * T * d + gate + touched * per_expert), "flops": flops}
    return {"bytes": size * (4 * T * d + 2 * gate + (touched + E) * per_expert), "flops": 3 * flops}


def tolerance(case):
    """About four times the largest error against the same step in 64 bits (given the same choice of experts):
    1.8e-6 in fp32, 7.5e-4 in fp16, 7e-3 in bf16 (1.2e-2 the gradient of a few-expert gate bias).  Single elements: a
    pre-activation within a rounding of zero opens or closes a ReLU, and that element's gradient is all or
    nothing on either side (seen: 0.33 of the gradient's root mean square)."""
    rel = {"float32": 1e-5, "float16": 3e-3, "bfloat16": 2.5e-2}[case["dtype"]]
    return {"rel": rel, "max": 0.9} if case["act"] == "relu" else {"rel": rel}
