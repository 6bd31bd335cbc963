"""What a user of this package has it do, as measurable cases.

A case names a kind of call, the patterns, the type, the layout and the number of batch entries:

* ``factor``: one ``Kernel.forward`` (the reference's own entry point);
* ``layer``:  one ``KSLinear`` with a bias;
* ``mlp``:    the two ``KSLinear`` layers of a transformer's MLP with the GELU between them, batch-first
  in and out, the wide activations kept batch-last (as ``ksmm_b200.ksvit.KSFeedForward`` does);
* ``qkv``:    three ``KSLinear`` layers on one input (``KSLinearGroup``);
* ``train``:  forward and backward of a trainable ``KSLinear``; the outputs are the layer's result and
  every gradient.

Inputs are N(0,1) (what a LayerNorm hands on) and weights U(-1/sqrt(c), 1/sqrt(c)) (the layer's own
initialisation), both drawn on the GPU from the seed.
"""
from __future__ import annotations

import math

import torch

import ksmm_b200 as kb

DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16,
          "fp8": torch.float8_e4m3fn}
ESIZE = {"fp32": 4, "fp16": 2, "bf16": 2, "fp8": 2}   # of what goes in and comes out: an fp8 layer takes and returns bf16

README = "6,64,64,1 1,768,192,2"                  # 384 -> 1536
FC1 = "4,192,192,1 1,768,192,4"                   # 768 -> 3072
FC2 = "1,192,768,4 4,192,192,1"                   # 3072 -> 768
CHAIN3 = "1,64,64,16 4,64,64,4 16,64,64,1"        # 1024 -> 1024, butterfly-like
SQUARE = "4,192,192,1 1,192,192,4"                # 768 -> 768, an attention projection


def _case(name, kind, patterns, dtype, bs_last, batch):
    return {"name": name, "kind": kind, "patterns": patterns, "dtype": dtype, "bs_last": bs_last, "batch": batch}


def listed():
    return [
        # online inference, a handful of rows: launches and host work are all there is
        _case("online_fp16_first", "layer", README, "fp16", False, 16),
        # one image of 196 patches and a class token through a transformer MLP
        _case("image_mlp_fp16_first", "mlp", FC1 + " | " + FC2, "fp16", False, 197),
        # 33 images of 197 tokens, batch-last: the batch is not a multiple of anything
        _case("ragged_fp16_last", "layer", README, "fp16", True, 6501),
        # the MLP of a vision transformer at the batch of the benchmark (128 images of 196 tokens)
        _case("mlp_fp16_first", "mlp", FC1 + " | " + FC2, "fp16", False, 25088),
        # a three-factor butterfly-like layer in bf16
        _case("chain3_bf16_first", "layer", CHAIN3, "bf16", False, 12544),
        # one fp32 factor through the reference's entry point, at the benchmark's batch
        _case("factor_fp32_last", "factor", "1,768,192,4", "fp32", True, 25088),
        # an fp32 layer whose first factor interleaves its blocks inside a row
        _case("fc2_fp32_first", "layer", FC2, "fp32", False, 12544),
        # the q, k and v projections of an attention layer, 64 images of 197 tokens
        _case("qkv_bf16_first", "qkv", SQUARE, "bf16", False, 12608),
        # fp8 inference: per-tensor scales, weights quantised once
        _case("fp8_first", "layer", FC1, "fp8", False, 12544),
        # a training step of one layer in fp16, 64 images
        _case("train_fp16_first", "train", FC1, "fp16", False, 12544),
        # a training step of one layer in fp32, 32 images
        _case("train_fp32_last", "train", README, "fp32", True, 6272),
        # throughput inference: 512 images at once
        _case("large_fp16_last", "layer", FC1, "fp16", True, 100352),
    ]


# what draw() combines: (kind, patterns, types, layouts, largest batch)
_BOTH = (False, True)
_RANGES = [
    ("layer", README, ("fp16", "bf16", "fp32"), _BOTH, 50176),
    ("layer", README, ("fp8",), (True,), 50176),
    ("layer", FC1, ("fp16", "bf16", "fp32", "fp8"), _BOTH, 50176),
    ("layer", FC2, ("fp16", "bf16", "fp32"), _BOTH, 50176),
    ("layer", CHAIN3, ("fp16", "bf16", "fp32"), _BOTH, 50176),
    ("mlp", FC1 + " | " + FC2, ("fp16", "bf16"), (False,), 50176),
    ("qkv", SQUARE, ("fp16", "bf16"), (False,), 50176),
    ("train", README, ("fp16", "bf16", "fp32"), _BOTH, 12544),
    ("train", FC1, ("fp16", "bf16"), _BOTH, 12544),
    ("factor", "1,768,192,4", ("fp16", "bf16", "fp32"), _BOTH, 25088),
    ("factor", "1,192,768,4", ("fp16", "bf16", "fp32"), _BOTH, 25088),
    ("factor", "1,768,192,2", ("fp16", "bf16", "fp32"), _BOTH, 25088),
    ("factor", "4,64,64,4", ("fp16", "bf16", "fp32"), _BOTH, 25088),
    ("factor", "1,128,128,6", ("fp16", "bf16", "fp32"), _BOTH, 25088),
]


def draw(rng):
    kind, patterns, dtypes, layouts, most = rng.choice(_RANGES)
    batch = int(round(math.exp(rng.uniform(math.log(16), math.log(most)))))
    shape = rng.choice(("rows", "images", "tokens"))
    if shape == "images" and batch >= 196:       # whole images of 196 patches, or of 197 tokens
        batch -= batch % 196
    elif shape == "tokens" and batch >= 197:
        batch -= batch % 197
    case = _case("", kind, patterns, rng.choice(dtypes), rng.choice(layouts), batch)
    del case["name"]
    return case


def _chains(case):
    """The chains of a case, each a list of (a, b, c, d)."""
    return [[tuple(int(v) for v in p.split(",")) for p in part.split()] for part in case["patterns"].split("|")]


def _randn(gen, *shape):
    return torch.randn(*shape, device="cuda", generator=gen)


def _weights(gen, patterns):
    return [(torch.rand(*p, device="cuda", generator=gen) * 2 - 1) / math.sqrt(p[2]) for p in patterns]


def _layer(gen, patterns, dtype, bs_last, **kw):
    layer = kb.KSLinear(patterns, weights=_weights(gen, patterns), bias=True, algo="kernel", dtype=dtype,
                        bs_last=bs_last, device="cuda", **kw)
    bound = 1 / math.sqrt(layer.in_size)
    with torch.no_grad():
        bias = (torch.rand(layer.out_size, device="cuda", generator=gen) * 2 - 1) * bound
        layer.bias.copy_(bias.reshape(layer.bias.shape))
    return layer


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype, bs_last, batch, kind = DTYPES[case["dtype"]], bool(case["bs_last"]), case["batch"], case["kind"]
    chains = _chains(case)
    a, _, c, d = chains[0][0]
    x = _randn(gen, a * c * d, batch) if bs_last else _randn(gen, batch, a * c * d)
    x = x.to(torch.bfloat16 if case["dtype"] == "fp8" else dtype)
    state = {"kind": kind, "x": x, "bs_last": bs_last}
    if kind == "factor":
        p = chains[0][0]
        state["pattern"] = p
        state["w"] = kb.generate_factor(*p, "kernel", _weights(gen, [p])[0], dtype, "cuda")
        state["dtype"] = str(dtype)
    elif kind == "layer":
        state["layer"] = _layer(gen, chains[0], dtype, bs_last)
    elif kind == "mlp":
        state["fc1"] = _layer(gen, chains[0], dtype, False, activation="gelu", out_bs_last=True)
        state["fc2"] = _layer(gen, chains[1], dtype, True, out_bs_last=False)
    elif kind == "qkv":
        state["group"] = kb.KSLinearGroup([_layer(gen, chains[0], dtype, bs_last) for _ in range(3)])
    else:
        layer = _layer(gen, chains[0], dtype, bs_last, requires_grad=True)
        g = _randn(gen, layer.out_size, batch) if bs_last else _randn(gen, batch, layer.out_size)
        state["layer"], state["grad"] = layer, g.to(dtype)
        state["x"] = x.requires_grad_(True)
    return state


def run(state):
    kind, x = state["kind"], state["x"]
    if kind == "factor":
        return kb.Kernel.forward(x, state["w"], state["bs_last"], *state["pattern"], state["dtype"])
    if kind == "layer":
        return state["layer"](x)
    if kind == "mlp":
        return state["fc2"](state["fc1"](x))
    if kind == "qkv":
        return state["group"](x)
    layer = state["layer"]
    layer.zero_grad(set_to_none=True)
    x.grad = None
    y = layer(x)
    y.backward(state["grad"])
    return [y.detach(), x.grad, layer.bias.grad] + [f.grad for f in layer.factors]


def work(case):
    chains, batch, es = _chains(case), case["batch"], ESIZE[case["dtype"]]
    first, last = chains[0][0], chains[-1][-1]
    n_in, n_out = first[0] * first[2] * first[3], last[0] * last[1] * last[3]
    weights = sum(a * b * c * d for chain in chains for a, b, c, d in chain)
    wes = 1 if case["dtype"] == "fp8" else es
    if case["kind"] == "qkv":
        return {"bytes": es * batch * (n_in + 3 * n_out) + 3 * es * weights, "flops": 3 * 2.0 * weights * batch}
    if case["kind"] == "train":
        # forward: x in, y out; backward: x (or what was kept of it) and the output's gradient in,
        # the input's gradient out; the weights are read by both and their gradient is written
        return {"bytes": es * (batch * (2 * n_in + n_out) + batch * (n_in + n_out)) + 3 * es * weights,
                "flops": 3 * 2.0 * weights * batch}
    return {"bytes": es * batch * (n_in + n_out) + wes * weights, "flops": 2.0 * weights * batch}


def tolerance(case):
    # About four times what the paths show against the same computation in fp64: fp32 2.8e-6 (three
    # tf32 products per term, c = 768; largest single difference 9e-6), fp16 4.8e-4 (2.1e-3), bf16
    # 3.9e-3 (1.9e-2), the two-layer MLP being the worst.  fp8 is stated against the same quantised
    # weights: a value next to a rounding border of e4m3 may land on its other side, which moves
    # the result by about half a percent.
    return {"fp32": {"rel": 1e-5, "max": 4e-5}, "fp16": {"rel": 2e-3, "max": 8e-3},
            "bf16": {"rel": 1.6e-2, "max": 8e-2}, "fp8": {"rel": 2e-2}}[case["dtype"]]
