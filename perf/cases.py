"""Workloads that the speed of this framework is judged by, and how to make, run and compare them.

A case is a dict of plain values:
  op     "experts"   the operator `yamoe_b200.experts` (inference forward)
         "layer"     the `Yamoe` module under `torch.no_grad()`: router, capacity, experts
         "backward"  the operator `yamoe_b200.experts_backward` (recomputes the forward)
         "train"     `experts_autograd(..., save_activations=True)`, forward and backward
  T, H, E, K         tokens, hidden size, experts, experts per token
  dtype  "bf16" or "fp32"
  skew   router logits with a bias of -1.2 ln(e + 1): a few experts get most of the rows
  dense  routing weights as the dense [T, E] matrix that the router produces, else the compact [T, K]

Shapes are those of bench.py, perf_sweep.py and the README workload; weights and biases are
N(0, 0.02), activations and upstream gradients N(0, 1), router logits N(0, 1) through softmax and
top-k without renormalisation.  Operators get a capacity that drops nothing; the layer keeps its
default capacity ceil(T K / E), which drops the surplus of over-subscribed experts.
"""
import math
import types

import torch

import yamoe_b200

#: (H, E, K) of the repository's own configurations
OSS_20B, OSS_120B = (2880, 32, 4), (2880, 128, 4)
HALF, SMALL, SMALL_16, WIDE, README = (2880, 16, 2), (1024, 32, 4), (1024, 16, 2), (2048, 64, 8), (2880, 8, 2)

STD = 0.02


def _case(op, T, shape, dtype="bf16", skew=False, dense=True):
    H, E, K = shape
    return dict(op=op, T=T, H=H, E=E, K=K, dtype=dtype, skew=skew, dense=dense)


def listed():
    named = {
        # one user, one token at a time: latency, and the weights of four experts from HBM
        "decode_1": _case("experts", 1, OSS_120B),
        # decoding a small batch: weight streaming, few rows for each expert hit
        "decode_16": _case("experts", 16, OSS_120B),
        # decoding 64 sequences through the whole layer, router and default capacity included
        "layer_64": _case("layer", 64, OSS_20B),
        # a narrow layer on one prompt: launches and latency count as much as the arithmetic
        "prefill_2048_narrow": _case("experts", 2048, SMALL_16, dense=False),
        # one prompt: every expert's weights are read for some 64 rows each
        "prefill_512": _case("experts", 512, OSS_20B),
        # a ragged batch on many experts with top-8
        "prefill_1531_wide": _case("experts", 1531, WIDE),
        # the headline workload: 16 prompts of 256 tokens
        "prefill_4096": _case("experts", 4096, OSS_20B),
        # long prefill with Zipf-like load: experts from tens of thousands of rows down to none
        "prefill_16384_skew": _case("experts", 16384, OSS_120B, skew=True),
        # the largest: gradients of a training batch, forward recomputed as the reference does
        "backward_8192": _case("backward", 8192, OSS_20B),
        # a training step of a ragged batch that keeps its activations, compact routing weights
        "train_1531_wide": _case("train", 1531, WIDE, dense=False),
        # single precision: the README workload, and a training step of a small layer
        "fp32_512": _case("experts", 512, README, "fp32"),
        "fp32_train_600": _case("train", 600, SMALL_16, "fp32"),
    }
    return [dict(c, name=n) for n, c in named.items()]


#: op, dtype, shapes, smallest and largest T; decode and prefill are two ranges of one operator
RANGES = [
    ("experts", "bf16", (OSS_120B, OSS_20B, SMALL, WIDE), 1, 64),
    ("experts", "bf16", (OSS_20B, OSS_120B, HALF, SMALL, SMALL_16, WIDE), 65, 16384),
    ("layer", "bf16", (OSS_20B, OSS_120B, SMALL, WIDE), 1, 4096),
    ("backward", "bf16", (OSS_20B, HALF, SMALL, SMALL_16, WIDE), 100, 8192),
    ("train", "bf16", (OSS_20B, HALF, SMALL, SMALL_16, WIDE), 100, 8192),
    ("experts", "fp32", (README, SMALL, SMALL_16), 32, 1100),
    ("train", "fp32", (README, SMALL, SMALL_16), 32, 1100),
]


def _flops(case):
    """Forward 2 S H (2H + H); backward twice that, and 4 S H H to recompute the pre-activations."""
    per_pass = {"experts": 6, "layer": 6, "backward": 16, "train": 18}[case["op"]]
    return per_pass * case["T"] * case["K"] * case["H"] * case["H"]


def _cost(case):
    """For the bound on drawn cases: an fp32 operation counts as much as 40 on the bf16 tensor cores."""
    return _flops(case) * (40 if case["dtype"] == "fp32" else 1)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        op, dtype, shapes, low, high = rng.choice(RANGES)
        T = min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))
        case = _case(op, T, rng.choice(shapes), dtype, skew=op == "experts" and rng.random() < 0.25,
                     dense=op == "layer" or rng.random() < 0.7)
        if _cost(case) <= most:
            return case


def _routing(case, gen, dtype):
    T, E, K = case["T"], case["E"], case["K"]
    logits = torch.randn(T, E, generator=gen, device="cuda")
    if case["skew"]:
        logits -= 1.2 * torch.log(torch.arange(1, E + 1, device="cuda", dtype=torch.float32))
    weights, indices = torch.topk(torch.softmax(logits, dim=-1), K, dim=-1)
    if case["dense"]:
        weights = torch.zeros(T, E, device="cuda").scatter_(1, indices, weights)
    return indices, weights.to(dtype)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    T, H, E, K = (case[k] for k in "THEK")

    def normal(*shape, std=1.0):
        return torch.empty(*shape, dtype=dtype, device="cuda").normal_(0, std, generator=gen)

    hidden = normal(T, H)
    weights = dict(gate_up_proj=normal(E, H, 2 * H, std=STD), gate_up_proj_bias=normal(E, 2 * H, std=STD),
                   down_proj=normal(E, H, H, std=STD), down_proj_bias=normal(E, H, std=STD))
    if case["op"] == "layer":
        layer = yamoe_b200.Yamoe()
        layer.router = types.SimpleNamespace(weight=normal(E, H, std=H ** -0.5), bias=normal(E, std=STD))
        layer.experts = types.SimpleNamespace(**weights)
        layer.num_experts, layer.top_k = E, K
        return dict(op="layer", layer=layer, hidden=hidden.view(1, T, H))
    indices, routing = _routing(case, gen, dtype)
    state = dict(op=case["op"], args=[hidden, indices, routing, *weights.values()], numbers=(T, E, K))
    if case["op"] != "experts":
        state["grad"] = normal(T, H)
    if case["op"] == "train":
        state["leaves"] = [t.requires_grad_(True) for t in state["args"] if t.is_floating_point()]
    return state


def run(state):
    if state["op"] == "layer":
        with torch.no_grad():
            return state["layer"](state["hidden"])
    if state["op"] == "experts":
        return yamoe_b200.experts(*state["args"], *state["numbers"])
    if state["op"] == "backward":
        return yamoe_b200.experts_backward(state["grad"], *state["args"], *state["numbers"])
    out = yamoe_b200.experts_autograd(*state["args"], *state["numbers"], save_activations=True)
    return [out.detach(), *torch.autograd.grad(out, state["leaves"], state["grad"])]


def _experts_hit(case):
    """Expected number of experts that at least one of T tokens chooses (uniform routing)."""
    E, K, T = case["E"], case["K"], case["T"]
    return E * (1 - (1 - K / E) ** T)


def work(case):
    T, H, E, K = (case[k] for k in "THEK")
    size = 2 if case["dtype"] == "bf16" else 4
    weights = _experts_hit(case) * (3 * H * H + 3 * H) * size
    rows, routing = T * H * size, T * K * 8 + T * (E if case["dense"] else K) * size
    nbytes = weights + 2 * rows + routing                       # forward: weights, tokens in and out
    if case["op"] == "layer":
        nbytes = weights + 2 * rows + E * H * size + T * E * size
    elif case["op"] == "backward":                              # every expert's gradients are written
        nbytes += rows + E * (3 * H * H + 3 * H) * size + routing
    elif case["op"] == "train":
        nbytes += 2 * rows + E * (3 * H * H + 3 * H) * size + routing
    return {"bytes": nbytes, "flops": _flops(case)}


def tolerance(case):
    # against the same path in fp32 (bf16 cases) or fp64 (fp32 cases) sums the largest relative error of
    # any output is 3.6e-3 and 1.6e-6
    return {"rel": 1.2e-2} if case["dtype"] == "bf16" else {"rel": 7e-6}


def _exact_expert(x, gate_up, gate_up_bias, down, down_bias):
    pre = x @ gate_up + gate_up_bias
    gate, up = pre[:, 0::2].clamp(max=7.0), pre[:, 1::2].clamp(-7.0, 7.0)
    return ((up + 1) * gate * torch.sigmoid(1.702 * gate)) @ down + down_bias


def exact(case, seed):
    """`run`'s outputs in 64 bits.  The layer picks its experts by rounded logits, near ties and the
    capacity among them, so that its outputs have no value apart from that rounding."""
    if case["op"] == "layer":
        return None
    state = prepare(case, seed)
    hidden, indices, routing, *p = [t.detach() for t in state["args"]]
    x, routing64 = hidden.double(), routing.double()
    w_of = routing64.gather(1, indices) if case["dense"] else routing64
    out, d_hidden, d_w = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(w_of)
    with_grad = case["op"] != "experts"
    d = [torch.zeros(t.shape, dtype=torch.float64, device=t.device) for t in p] if with_grad else []
    for e in range(case["E"]):
        tok, slot = torch.nonzero(indices == e, as_tuple=True)
        if tok.numel() == 0:
            continue
        w = w_of[tok, slot, None]
        leaves = [t.requires_grad_(with_grad) for t in (x[tok], *(t[e].double() for t in p))]
        y = _exact_expert(*leaves)
        out.index_add_(0, tok, y.detach() * w)
        if with_grad:
            gy = state["grad"][tok].double()
            grads = torch.autograd.grad(y, leaves, gy * w)
            d_hidden.index_add_(0, tok, grads[0])
            d_w[tok, slot] = (y.detach() * gy).sum(-1)
            for whole, part in zip(d, grads[1:]):
                whole[e] = part
    if not with_grad:
        return out
    d_routing = torch.zeros_like(routing64).scatter_(1, indices, d_w) if case["dense"] else d_w
    grads = [d_hidden, d_routing, *d]
    return grads if case["op"] == "backward" else [out, *grads]
