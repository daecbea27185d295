"""Performance cases: the calls a program that differentiates attention twice makes, over the range it makes them in.

Six kinds of call, each through the public entry point a user's program calls:

* ``bwdbwd``    ``fhob.flash_bwdbwd`` on device tensors: the double backward, the reason the framework exists
* ``host``      the same call on pinned host tensors (staged through the device by the call itself)
* ``forward``   ``fhob.attention_forward``: O and the logsumexp the other two calls consume
* ``lse``       ``fhob.produce_L``: the logsumexp alone
* ``backward``  ``fhob.attention_backward``: dQ, dK, dV
* ``grad2``     ``fhob.attention`` under autograd, differentiated twice: a gradient-penalty step

``listed`` has twelve of them, ``draw`` spreads over the same ranges.
"""
import math
import os
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "flash-hob_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import fhob  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _case(kind, dtype, batch, heads, n_q, n_k, d, d_v=None, causal=False, window=0, layout="bhnd", cotangent=1.0):
    """``layout`` "bnhd": the tensors are (batch, sequence, head, dim) projections seen as (batch, head, sequence, dim)."""
    return {"kind": kind, "dtype": dtype, "batch": batch, "heads": heads, "n_q": n_q, "n_k": n_k, "d": d,
            "d_v": d if d_v is None else d_v, "causal": causal, "window": window, "layout": layout,
            "cotangent": cotangent}


def listed():
    def named(name, *a, **k):
        return dict(_case(*a, **k), name=name)

    return [
        # The correctness-sized fp32 problem (a unit test, a toy model): launches and host work are all there is.
        named("op fp32 2h n256 d64", "bwdbwd", "fp32", 1, 2, 256, 256, 64),
        # An ordinary self-attention layer with small heads.
        named("op bf16 64h n2048 d64", "bwdbwd", "bf16", 4, 16, 2048, 2048, 64),
        # A causal language-model layer; cotangents a tenth of the activations, as gradients are.
        named("op bf16 causal 128h n4096", "bwdbwd", "bf16", 8, 16, 4096, 4096, 128, causal=True, cotangent=0.1),
        # Long context, one GPU's share of an eight-way head split.
        named("op bf16 causal 4h n32768", "bwdbwd", "bf16", 1, 4, 32768, 32768, 128, causal=True),
        # Cross-attention, one GPU's share of an eight-way head split of the 512-head job.
        named("op bf16 64h 4096x8192", "bwdbwd", "bf16", 2, 32, 4096, 8192, 128),
        # Sliding-window layer with a head dim and a length off the tile grid, read in place from projections.
        named("op fp16 window ragged d80", "bwdbwd", "fp16", 2, 12, 3333, 3333, 80, causal=True, window=512, layout="bnhd"),
        # A few latent queries over a long memory, values wider than keys, batch of one: little of the chip has work.
        named("op bf16 16h 100x6000", "bwdbwd", "bf16", 1, 16, 100, 6000, 64, d_v=128),
        # fp32 at the large head dim: a numerically careful run, or the check of a 16-bit one.
        named("op fp32 8h n1024 d128", "bwdbwd", "fp32", 1, 8, 1024, 1024, 128),
        # The producers of what the operator consumes: the forward of the causal layer ...
        named("forward bf16 causal 32h", "forward", "bf16", 2, 16, 4096, 4096, 128, causal=True),
        # ... and a first backward.
        named("backward bf16 32h n2048", "backward", "bf16", 2, 16, 2048, 2048, 128),
        # A gradient-penalty step of a small model through autograd: forward, first and second backward.
        named("grad2 bf16 causal 8h n512", "grad2", "bf16", 2, 4, 512, 512, 64, causal=True),
        # Tensors that live in (pinned) host memory.
        named("host bf16 32h n1024 d64", "host", "bf16", 2, 16, 1024, 1024, 64),
    ]


def _log_between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _too_large(c):
    """Whether a drawn case has more operations than its kind of arithmetic does in the time of the largest listed
    one, or more bytes than the larger listed ones."""
    w = work(c)
    if c["kind"] == "host":
        return w["flops"] > 4e11 or w["bytes"] > 2e8
    if c["dtype"] == "fp32":
        flops = 8e11 if max(c["d"], c["d_v"]) <= 64 else 2.5e10
    else:
        flops = 4e12
    return w["flops"] > flops or w["bytes"] > 1.2e9


def draw(rng):
    kind = rng.choice(["bwdbwd"] * 6 + ["forward", "backward", "lse", "host"] + ["grad2"] * 2)
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"])
    d = rng.choice([32, 64, 64, 80, 96, 128, 128])
    d_v = d if kind == "lse" or rng.random() < 0.8 else rng.choice([32, 64, 96, 128])
    n_q = _log_between(rng, 64, 32768)
    shape = rng.random()
    if shape < 0.6:
        n_k = n_q                                   # self-attention
    elif shape < 0.8:
        n_k = _log_between(rng, n_q, 32768)         # cross-attention, or queries that continue a sequence
    else:
        n_k = n_q + rng.randint(1, n_q)
    causal = rng.random() < 0.5
    window = _log_between(rng, 64, 4096) if causal and rng.random() < 0.25 else 0
    batch, heads = rng.choice([1, 1, 2, 4, 8]), rng.choice([1, 2, 4, 8, 12, 16, 32])
    layout = "bnhd" if rng.random() < 0.25 and kind != "host" else "bhnd"
    if rng.random() < 0.5:                          # half the lengths on the grid that models like, half off it
        n_q, n_k = max(64, n_q // 64 * 64), max(64, n_k // 64 * 64)
    c = _case(kind, dtype, batch, heads, n_q, n_k, d, d_v, causal, window, layout, rng.choice([1.0, 0.1]))
    while _too_large(c):
        if c["batch"] * c["heads"] > 1 and (c["n_q"] < 2048 or rng.random() < 0.7):
            c["batch" if c["batch"] > 1 else "heads"] //= 2
        else:
            c["n_q"], c["n_k"] = max(64, c["n_q"] * 2 // 3), max(64, c["n_k"] * 2 // 3)
        if c["causal"] and c["n_k"] < c["n_q"]:
            c["n_k"] = c["n_q"]
    return c


def _pairs(c):
    """(query, key) pairs the mask leaves visible, per head."""
    n_q, n_k = c["n_q"], c["n_k"]
    if not c["causal"]:
        return n_q * n_k
    off = n_k - n_q                                 # query i sees keys up to i + off (n_k >= n_q here)
    seen = n_q * (2 * off + n_q + 1) // 2
    w = c["window"]
    if w and n_k > w:                               # queries whose reach is longer than the window lose the difference
        first = max(0, w - off)                     # first query with i + off + 1 > w
        m = n_q - first
        lo, hi = first + off + 1 - w, n_q + off - w
        seen -= m * (lo + hi) // 2
    return seen


def work(case):
    """Inputs read once, results written once; the distinct contractions of the mathematics, over visible pairs."""
    c = case
    bh, es = c["batch"] * c["heads"], DTYPES[c["dtype"]].itemsize
    q, k = bh * c["n_q"] * c["d"], bh * c["n_k"] * c["d"]
    v, o, rows = bh * c["n_k"] * c["d_v"], bh * c["n_q"] * c["d_v"], bh * c["n_q"]
    pairs = 2 * bh * _pairs(c)
    # contractions over (or onto) the q/k head dim and the v head dim
    forward = pairs * (c["d"] + c["d_v"])
    backward = pairs * (3 * c["d"] + 2 * c["d_v"])
    second = pairs * (7 * c["d"] + 5 * c["d_v"])
    if c["kind"] == "forward":
        return {"bytes": (q + k + v + o) * es + 4 * rows, "flops": forward}
    if c["kind"] == "lse":
        return {"bytes": (q + k) * es + 4 * rows, "flops": pairs * c["d"]}
    if c["kind"] == "backward":
        return {"bytes": (2 * q + 2 * k + 2 * v + 2 * o) * es + 4 * rows, "flops": backward}
    if c["kind"] == "grad2":
        return {"bytes": (4 * q + 4 * k + 4 * v + 3 * o) * es, "flops": forward + backward + second}
    return {"bytes": (3 * q + 3 * k + 3 * v + 3 * o) * es + 4 * rows, "flops": second}


def tolerance(case):
    """Results are rounded to the storage type, and 16-bit problems also round the probabilities and their
    derivatives before the output products; fp32 results are sums that cancel (dP - D, dP2 - b)."""
    return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 3e-5}[case["dtype"]]}


def prepare(case, seed):
    """Activations N(0, 1), cotangents scaled; O and L saved from the forward, as training saves them."""
    c, dtype = case, DTYPES[case["dtype"]]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def tensor(n, d, mul=1.0):
        if c["layout"] == "bnhd":
            t = torch.randn(c["batch"], n, c["heads"], d, generator=g, device="cuda", dtype=dtype).transpose(1, 2)
        else:
            t = torch.randn(c["batch"], c["heads"], n, d, generator=g, device="cuda", dtype=dtype)
        return t.mul_(mul) if mul != 1.0 else t

    s = {"kind": c["kind"], "scale": c["d"] ** -0.5,
         "mask": {"is_causal": c["causal"], "sliding_window": c["window"] or None},
         "q": tensor(c["n_q"], c["d"]), "k": tensor(c["n_k"], c["d"])}
    if c["kind"] == "lse":
        return s
    s["v"] = tensor(c["n_k"], c["d_v"])
    if c["kind"] == "forward":
        return s
    s["d_o"] = tensor(c["n_q"], c["d_v"], c["cotangent"])
    if c["kind"] != "backward":
        s["ddq"], s["ddk"] = tensor(c["n_q"], c["d"], c["cotangent"]), tensor(c["n_k"], c["d"], c["cotangent"])
        s["ddv"] = tensor(c["n_k"], c["d_v"], c["cotangent"])
    if c["kind"] == "grad2":
        for n in ("q", "k", "v", "d_o"):
            s[n].requires_grad_(True)
        return s
    s["o"], s["lse"] = fhob.attention_forward(s["q"], s["k"], s["v"], s["scale"], **s["mask"])
    if c["kind"] == "host":
        for n, t in list(s.items()):
            if isinstance(t, torch.Tensor):
                s[n] = torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)
    return s


def run(state):
    s = state
    kind = s["kind"]
    if kind in ("bwdbwd", "host"):
        return fhob.flash_bwdbwd(s["q"], s["k"], s["v"], s["o"], s["d_o"], s["ddq"], s["ddk"], s["ddv"], s["lse"],
                                 s["scale"], **s["mask"])
    if kind == "forward":
        return fhob.attention_forward(s["q"], s["k"], s["v"], s["scale"], **s["mask"])
    if kind == "lse":
        return fhob.produce_L(s["q"], s["k"], s["mask"]["is_causal"], s["scale"], s["mask"]["sliding_window"])
    if kind == "backward":
        return fhob.attention_backward(s["q"], s["k"], s["v"], s["o"], s["d_o"], s["lse"], s["scale"], **s["mask"])
    o = fhob.attention(s["q"], s["k"], s["v"], s["scale"], **s["mask"])
    first = torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["d_o"], create_graph=True)
    second = torch.autograd.grad(first, (s["q"], s["k"], s["v"], s["d_o"]), (s["ddq"], s["ddk"], s["ddv"]))
    return (o, *first, *second)
