"""The work that is timed when this package is made faster: its public operators and layers as a
user's program calls them, at sizes from the benchmark's configurations, the tests and the windows
of published neighborhood-attention backbones.

A case is a dict of plain values. Sizes per token axis are texts such as "32x48x80".

  op       "na" (na1d / na2d / na3d), "layer" (NeighborhoodAttention2D), "attention" (dense)
  train    forward, then the gradients of every input (and parameter) for a given output gradient;
           otherwise the forward alone, without gradients
  extra    additional key/value tokens that every query attends
  keys     dense attention only: key/value tokens (``tokens`` is the number of queries)
"""
import math
import random

import torch

import natten_b200 as nb

DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16,
          "fp8": torch.float8_e4m3fn}
BYTES = {"fp32": 4, "fp16": 2, "bf16": 2, "fp8": 1}


def _case(name, op, dtype, batch, heads, tokens, head_dim, kernel="", stride="", dilation="",
          causal="", heads_kv=0, extra=0, keys=0, train=False, lse=False, spread=1.0):
    nd = tokens.count("x") + 1
    ones, zeros = "x".join("1" * nd), "x".join("0" * nd)
    return {"name": name, "op": op, "dtype": dtype, "batch": batch, "heads": heads,
            "heads_kv": heads_kv or heads, "tokens": tokens, "head_dim": head_dim,
            "kernel": kernel, "stride": stride or ones, "dilation": dilation or ones,
            "causal": causal or zeros, "extra": extra, "keys": keys, "train": train, "lse": lse,
            "spread": spread}


def listed():
    return [
        # The smallest call: one feature map in single precision with its logsumexp. Launch and
        # host latency are what a user waits for.
        _case("map2d-fp32", "na", "fp32", 1, 4, "32x32", 32, "7x7", lse=True),
        # One image through one layer of a backbone at inference: projections and the operator on
        # strided views of the fused projection, narrow heads.
        _case("layer2d-infer", "layer", "bf16", 1, 4, "56x56", 32, "7x7"),
        # A training step of the same layer on a batch of images.
        _case("layer2d-train", "layer", "bf16", 32, 4, "56x56", 32, "7x7", train=True),
        # Single-precision training (the default precision of a PyTorch program) on maps of odd
        # size.
        _case("map2d-fp32-train", "na", "fp32", 2, 6, "61x45", 64, "9x9", train=True),
        # Long causal sequences with a sliding window, forward.
        _case("seq1d-causal", "na", "bf16", 4, 16, "32768", 128, "2048", causal="1"),
        # The same kind of model in training: grouped query heads, a ragged length.
        _case("seq1d-gqa-train", "na", "bf16", 2, 16, "8190", 128, "512", causal="1", heads_kv=4,
              train=True),
        # A dilated window over a batch of feature maps: small windows, so memory-bound in theory.
        _case("map2d-dilated", "na", "bf16", 8, 16, "128x128", 128, "13x13", dilation="2x2"),
        # High-resolution image generation: strided (block-sparse) windows plus text tokens.
        _case("image2d-text", "na", "fp16", 1, 24, "256x256", 128, "32x32", stride="16x16",
              extra=256, spread=0.5),
        # Video diffusion, the largest workload.
        _case("video3d", "na", "bf16", 1, 24, "32x48x80", 128, "16x24x24", stride="1x8x8",
              causal="1x0x0"),
        # A smaller video model in training, sizes that no tile divides.
        _case("video3d-train", "na", "bf16", 1, 12, "15x30x52", 64, "7x15x15", train=True),
        # Video inference with 8-bit operands.
        _case("video3d-fp8", "na", "fp8", 1, 12, "15x44x80", 128, "9x16x24"),
        # Dense self attention in training: what a window as large as its map becomes, and the
        # dense layers that such models mix in.
        _case("dense-train", "attention", "bf16", 2, 12, "1370", 64, train=True),
    ]


# ---- cases of the same ranges ---------------------------------------------------------------------

def _log(rng, lo, hi):
    """An integer between lo and hi, spread evenly over its logarithm."""
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))


def _windows(rng, sides, kernels, strides, dilations):
    """Per axis a window of `kernels` = (low, high) tokens that fits the axis with its dilation."""
    ks, ss, ds = [], [], []
    for x in sides:
        d = rng.choice(dilations)
        while d > 1 and 2 * d > x:
            d -= 1
        k = min(_log(rng, *kernels), x // d)
        ks.append(max(2, k))
        ds.append(d)
        ss.append(min(k, rng.choice(strides)))
    return ["x".join(str(v) for v in vs) for vs in (ks, ss, ds)]


def _draw(rng, base):
    """The listed case `base` with other sizes and options out of the range it stands for."""
    c = dict(base)
    del c["name"]
    nd = c["tokens"].count("x") + 1
    causal = [0] * nd
    if base["name"].startswith("map2d-fp32"):
        sides = [_log(rng, 7, 96) for _ in range(2)]
        c.update(batch=_log(rng, 1, 8), heads=_log(rng, 1, 8), head_dim=rng.choice([24, 32, 48, 64, 128]),
                 lse=rng.random() < 0.5 and not c["train"])
        win = _windows(rng, sides, (3, 15), [1, 1, 1, 2], [1, 1, 2])
    elif base["op"] == "layer":
        sides = [_log(rng, 14, 112) for _ in range(2)]
        c.update(batch=_log(rng, 1, 64), heads=rng.choice([2, 3, 4, 6, 8, 16]),
                 head_dim=rng.choice([32, 32, 64]))
        win = _windows(rng, sides, (5, 13), [1], [1, 1, 2, 4])
    elif base["name"].startswith("seq1d"):
        sides = [_log(rng, 512, 65536)]
        kv = rng.choice([1, 2, 4, 8])
        c.update(batch=_log(rng, 1, 8), heads=kv * rng.choice([1, 2, 4]), heads_kv=kv,
                 head_dim=rng.choice([64, 128]))
        win = _windows(rng, sides, (64, 4096), [1, 1, 64], [1, 1, 1, 4])
        causal = [int(rng.random() < 0.7)]
    elif nd == 2 and c["op"] == "na":
        sides = [_log(rng, 24, 320) for _ in range(2)]
        c.update(batch=_log(rng, 1, 16), heads=_log(rng, 2, 24), head_dim=rng.choice([32, 64, 80, 128, 128]),
                 extra=rng.choice([0, _log(rng, 16, 512)]) if c["extra"] else 0)
        c["heads_kv"] = c["heads"]
        win = _windows(rng, sides, (5, 64), [1, 1, 8, 16] if c["extra"] else [1], [1, 2] if not c["extra"] else [1])
    elif nd == 3:
        sides = [_log(rng, 4, 32), _log(rng, 16, 80), _log(rng, 16, 96)]
        dims = [128] if c["dtype"] == "fp8" else [64, 128]
        c.update(heads=_log(rng, 2, 24), head_dim=rng.choice(dims))
        win = _windows(rng, sides, (3, 24), [1, 1, 4, 8], [1])
        causal = [int(rng.random() < 0.3), 0, 0]
    else:  # dense: self attention in training, or a forward over another number of keys
        sides = [_log(rng, 49, 4096)]
        kv = rng.choice([1, 2, 4, 12])
        c.update(batch=_log(rng, 1, 8), heads=kv * rng.choice([1, 1, 2]), heads_kv=kv,
                 head_dim=rng.choice([32, 64, 128]), train=rng.random() < 0.6)
        win = ["", "1", "1"]
        causal = [int(rng.random() < 0.4)]
        if not c["train"] and rng.random() < 0.7:
            c["keys"], causal = _log(rng, 64, 16384), [0]
            if rng.random() < 0.5:
                sides = [_log(rng, 1, 512)]
    if c["op"] != "attention" and c["dtype"] in ("bf16", "fp16"):
        c["dtype"] = rng.choice(["bf16", "bf16", "fp16"])
    if c["op"] == "layer" or c["dtype"] == "fp32":
        c["heads_kv"] = c["heads"]
    if nd == 3:
        c["heads_kv"] = c["heads"]
    c.update(tokens="x".join(str(x) for x in sides), kernel=win[0], stride=win[1], dilation=win[2],
             causal="x".join(str(x) for x in causal))
    return c


def draw(rng: random.Random):
    """One more case: a listed one with its sizes and options drawn again, no more work than the
    largest listed case of its kind."""
    base = rng.choice(listed())
    kin = [c for c in listed() if (c["op"], c["dtype"] == "fp32", c["train"])
           == (base["op"], base["dtype"] == "fp32", base["train"])]
    most = {k: max(work(c)[k] for c in kin) for k in ("flops", "bytes")}
    if base["name"] == "map2d-fp32":     # one call of a few maps, not a batch
        most = {k: 64 * v for k, v in most.items()}
    if base["name"] == "layer2d-infer":
        most = {k: 32 * v for k, v in most.items()}
    while True:
        c = _draw(rng, base)
        w = work(c)
        if w["flops"] <= most["flops"] and w["bytes"] <= most["bytes"]:
            return c


# ---- one pass ---------------------------------------------------------------------------------------

def _ints(text):
    return tuple(int(v) for v in text.split("x"))


def _na_arguments(case):
    return {"kernel_size": _ints(case["kernel"]), "stride": _ints(case["stride"]),
            "dilation": _ints(case["dilation"]),
            "is_causal": tuple(v == 1 for v in _ints(case["causal"]))}


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[case["dtype"]]

    def normal(*shape, spread=case["spread"]):
        return (torch.randn(*shape, device="cuda", generator=gen) * spread).to(dtype)

    tokens, heads, kv, dim = _ints(case["tokens"]), case["heads"], case["heads_kv"], case["head_dim"]
    batch, train = case["batch"], case["train"]
    state = {"case": case}
    if case["op"] == "layer":
        embed = heads * dim
        with torch.device("cuda"):
            layer = nb.NeighborhoodAttention2D(embed, heads, **_na_arguments(case)).to(dtype)
        with torch.no_grad():
            for p in layer.parameters():
                p.copy_(normal(*p.shape, spread=embed ** -0.5))
        layer.train(train)
        state.update(layer=layer, inputs=[normal(batch, *tokens, embed)])
        out_shape = (batch, *tokens, embed)
    else:
        keys = (case["keys"],) if case["keys"] else tokens
        state["inputs"] = [normal(batch, *tokens, heads, dim), normal(batch, *keys, kv, dim),
                           normal(batch, *keys, kv, dim)]
        if case["extra"]:
            state["inputs"] += [normal(batch, case["extra"], kv, dim) for _ in range(2)]
        out_shape = (batch, *tokens, heads, dim)
        if case["op"] == "na":
            state["arguments"] = _na_arguments(case)
            state["operator"] = {1: nb.na1d, 2: nb.na2d, 3: nb.na3d}[len(tokens)]
        else:
            state["arguments"] = {"is_causal": case["causal"] == "1"}
            state["operator"] = nb.attention
    if train:
        state["inputs"] = [t.requires_grad_() for t in state["inputs"]]
        state["wrt"] = state["inputs"] + (list(state["layer"].parameters()) if "layer" in state else [])
        state["d_out"] = normal(*out_shape, spread=1.0)
    return state


def run(state):
    case, inputs = state["case"], state["inputs"]
    with torch.set_grad_enabled(case["train"]):
        if case["op"] == "layer":
            out = state["layer"](*inputs)
        elif case["extra"]:
            q, k, v, extra_k, extra_v = inputs
            out = state["operator"](q, k, v, additional_keys=extra_k, additional_values=extra_v,
                                    **state["arguments"])
        else:
            out = state["operator"](*inputs, return_lse=case["lse"], **state["arguments"])
        if not case["train"]:
            return out
        return [out.detach(), *torch.autograd.grad(out, state["wrt"], state["d_out"])]


# ---- what a pass cannot do without --------------------------------------------------------------------

def _window_sum(length, kernel, stride, causal):
    """Keys attended along one axis of `length` tokens, summed over its queries."""
    if not causal:
        return length * kernel
    total = 0
    for i in range(length):
        lead = min((i // stride) * stride + stride - 1, length - 1)
        total += min(i + 1, length) - max(lead - kernel + 1, 0)
    return total


def _pairs(case):
    """(query, key) pairs of one head and batch entry."""
    tokens = _ints(case["tokens"])
    if case["op"] == "attention":
        n = tokens[0]
        return n * (n + 1) // 2 if case["causal"] == "1" else n * (case["keys"] or n)
    pairs = 1
    axes = zip(tokens, *(_ints(case[k]) for k in ("kernel", "stride", "dilation", "causal")))
    for x, k, s, d, causal in axes:
        pairs *= sum(_window_sum(len(range(g, x, d)), k, s, causal) for g in range(d))
    return pairs + math.prod(tokens) * case["extra"]


def work(case):
    n_q = math.prod(_ints(case["tokens"])) * case["batch"]
    n_kv = (case["keys"] * case["batch"] or n_q) + case["extra"] * case["batch"]
    heads, dim, size, train = case["heads"], case["head_dim"], BYTES[case["dtype"]], case["train"]
    flops = 4.0 * dim * _pairs(case) * heads * case["batch"] * (3.5 if train else 1.0)
    if case["op"] == "layer":
        embed = heads * dim
        flops += 8.0 * n_q * embed * embed * (3 if train else 1)
        weights = (4 * embed * embed + 4 * embed) * size
        moved = 2 * n_q * embed * size + weights
    else:
        moved = (2 * n_q * heads + 2 * n_kv * case["heads_kv"]) * dim * size
        moved += 4 * n_q * heads * case["lse"]
    # training adds the output gradient and writes a gradient for every input
    return {"bytes": float(moved * (2 if train else 1)), "flops": flops}


def tolerance(case):
    # fp32: sums of a few hundred terms in another order. 16 bits: rounding of the probabilities
    # (and of dS) and of the results, 2^-9 for bf16 and 2^-12 for fp16 relative, several of them in
    # a row. 8 bits: results rounded to three mantissa bits, where a difference far below one step
    # moves some of them by a whole step (up to 1/8).
    if case["dtype"] == "fp32":
        return {"rel": 1e-5, "max": 2e-4}
    if case["dtype"] == "fp8":
        return {"rel": 3e-2, "max": 0.5}
    return {"rel": 1e-2, "max": 0.2} if case["dtype"] == "bf16" else {"rel": 2e-3, "max": 4e-2}
