"""The work a user has the grouped n:m kernels do, as measurable cases.

A case is one call (or one short sequence of calls) through the package's public entry points on operands that are already
on the GPU.  ``op`` names the entry point:

``linear``    a ``torch.nn.Linear`` whose weight ``SparsityBuilder`` turned into a ``GroupedNMTensor``, without gradients
``mm``        ``torch.mm(sparse weight, dense matrix)``, without gradients
``ffn``       ``activation(x W1^T + b1)`` and ``h W2^T + b2 + x`` through ``sparse_linear_fused`` (transformer inference)
``ffn_dx``    linear -> GELU -> linear with frozen sparse weights, forward and the gradient of the input
``train``     forward and backward of a trainable sparse linear: gradients of the input, the bias and -- in the weight's own
              layout -- the weight
``sparsify``  dense weight -> ``GroupedNMTensor`` (magnitude selection)
``densify``   ``GroupedNMTensor`` -> dense weight

``rows`` x ``cols`` is the weight (``rows`` = output features), ``tokens`` the batch, ``n``, ``m``, ``g`` the format.
"""
import math

import torch

import sten_b200 as sten

_DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
_PATTERNS = ((1, 4), (2, 4), (1, 8), (2, 8), (1, 16))  # the density sweep's patterns: every one has specialised kernels


def _case(op, dtype, n, m, rows, cols, tokens, g=16, name=None):
    c = {"op": op, "dtype": dtype, "n": n, "m": m, "g": g, "rows": rows, "cols": cols, "tokens": tokens}
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # one token through one attention projection of the fp16 encoder: the smallest call, all latency
        _case("linear", "f16", 2, 4, 1024, 1024, 1, name="linear_1_token"),
        # a decode step of a small batch of requests on a wide layer: the weight is the traffic
        _case("linear", "bf16", 2, 4, 4096, 4096, 16, name="linear_16_tokens"),
        # a classifier-like layer whose sizes are multiples of nothing, a batch of uneven requests
        _case("linear", "f16", 1, 8, 1023, 777, 333, name="linear_ragged"),
        # one sequence of the encoder benchmark through its first feed-forward linear
        _case("linear", "f16", 2, 4, 4096, 1024, 384, name="linear_384_tokens"),
        # the density sweep's layer and batch at 12.5 % density
        _case("linear", "bf16", 1, 8, 4096, 4096, 4096, name="linear_4096_tokens"),
        # the large row-shardable product on one GPU: the largest case
        _case("linear", "bf16", 2, 8, 16384, 16384, 16384, name="linear_16384_tokens"),
        # the plumbing configuration: fp32 weight times a dense matrix
        _case("mm", "f32", 2, 4, 1024, 1024, 256, name="mm_fp32"),
        # the feed-forward half of one encoder layer, batch 32 x 384, epilogues fused
        _case("ffn", "f16", 2, 4, 4096, 1024, 12288, name="ffn_fused"),
        # fp32 feed-forward pair at 75 % sparsity, batch 8 x 512, forward plus the input's gradient
        _case("ffn_dx", "f32", 1, 4, 3072, 768, 4096, name="ffn_fp32_forward_dx"),
        # one linear of a fine-tuning step, weight gradient kept packed
        _case("train", "bf16", 2, 4, 4096, 1024, 4096, name="train_linear"),
        # importing a dense fp32 checkpoint's layer
        _case("sparsify", "f32", 2, 4, 4096, 4096, 0, name="sparsify_fp32"),
        # exporting a large 16-bit layer
        _case("densify", "bf16", 2, 8, 8192, 8192, 0, name="densify_bf16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _feature_count(rng, lo, hi):
    """Layer widths: mostly multiples of 64, some of 8, a few of nothing."""
    v, u = _log_int(rng, lo, hi), rng.random()
    step = 64 if u < 0.6 else 8 if u < 0.85 else 1
    return min(hi, max(lo, (v + step - 1) // step * step))


def draw(rng):
    op = rng.choices(("linear", "mm", "ffn", "ffn_dx", "train", "sparsify", "densify"), (8, 2, 2, 2, 2, 2, 2))[0]
    dtype = {"ffn": ("f16", "bf16"), "train": ("f16", "bf16", "f32")}.get(op, ("f16", "bf16", "f32"))
    dtype = rng.choice(dtype)
    n, m = rng.choice(_PATTERNS)
    rows, cols = _feature_count(rng, 128, 16384), _feature_count(rng, 256, 16384)
    groups = [g for g in (4, 8, 16, 16, 16, 16, 32, 64) if math.comb(m, n) * g <= cols]
    g = rng.choice(groups or [4])
    if op in ("sparsify", "densify"):
        while rows * cols > 1 << (27 if dtype == "f32" else 28):
            rows = (rows + 1) // 2
        return _case(op, dtype, n, m, rows, cols, 0, g)
    tokens = _log_int(rng, 1, 16384)
    if tokens >= 64 and rng.random() < 0.5:
        tokens = tokens // 64 * 64
    # products executed per pass, and the rate of the slower arithmetic, keep a case below the largest listed one
    products = {"linear": 1, "mm": 1, "ffn": 2, "ffn_dx": 4, "train": 3}[op]
    ragged = cols % 8 != 0 or (op in ("ffn", "ffn_dx", "train") and rows % 8 != 0)
    budget = (1 << 42) // products
    budget >>= 4 if dtype == "f32" else 0
    budget >>= 7 if ragged else 0
    tokens = max(1, min(tokens, budget // (rows * cols)))
    return _case(op, dtype, n, m, rows, cols, tokens, g)


def _normal(shape, seed, salt, dtype, scale=1.0):
    gen = torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)
    return (torch.randn(*shape, generator=gen, device="cuda") * scale).to(dtype)


def _linear(case, rows, cols, seed, salt, trainable=False):
    """A dense linear with a trained layer's weight scale, sparsified the way a user's program does it."""
    dtype = _DTYPES[case["dtype"]]
    lin = torch.nn.Linear(cols, rows, device="cuda", dtype=dtype)
    with torch.no_grad():
        lin.weight.copy_(_normal((rows, cols), seed, salt, dtype, cols ** -0.5))
        lin.bias.copy_(_normal((rows,), seed, salt + 1, dtype, 0.1))
    sb = sten.SparsityBuilder()
    sb.set_weight("weight", initial_sparsifier=sten.GroupedNMSparsifier(n=case["n"], m=case["m"], g=case["g"]), out_format=sten.GroupedNMTensor)
    if trainable:
        sb.set_weight_grad("weight", inline_sparsifier=sten.WeightLayoutSparsifier(), tmp_format=sten.GroupedNMTensor,
                           external_sparsifier=sten.KeepAll(), out_format=sten.GroupedNMTensor)
    lin = sb.sparsify_model_inplace(lin)
    if not trainable:
        for p in lin.parameters():
            p.requires_grad_(False)
    return lin


def prepare(case, seed):
    op, dtype = case["op"], _DTYPES[case["dtype"]]
    rows, cols, tokens = case["rows"], case["cols"], case["tokens"]
    state = {"op": op, "format": (case["n"], case["m"], case["g"])}
    if op in ("sparsify", "densify"):
        w = _normal((rows, cols), seed, 1, dtype, cols ** -0.5)
        n, m, g = state["format"]
        state["weight"] = w if op == "sparsify" else sten.GroupedNMTensor.from_dense(w, n, m, sparse_dim=0, group_size=g, group_dim=1)
        return state
    state["x"] = _normal((cols, tokens) if op == "mm" else (tokens, cols), seed, 2, dtype)
    state["fc1"] = _linear(case, rows, cols, seed, 10, trainable=op == "train")
    if op in ("ffn", "ffn_dx"):
        state["fc2"] = _linear(case, cols, rows, seed, 20)
    if op in ("ffn_dx", "train"):
        state["x"].requires_grad_(True)
        state["dy"] = _normal((tokens, cols if op == "ffn_dx" else rows), seed, 3, dtype)
    if op == "ffn_dx":
        state["model"] = torch.nn.Sequential(state["fc1"], torch.nn.GELU(), state["fc2"])
    return state


def run(state):
    op = state["op"]
    if op == "linear":
        with torch.no_grad():
            return state["fc1"](state["x"])
    if op == "mm":
        with torch.no_grad():
            return torch.mm(state["fc1"].weight, state["x"])
    if op == "ffn":
        x, fc1, fc2 = state["x"], state["fc1"], state["fc2"]
        with torch.no_grad():
            h = sten.sparse_linear_fused(x, fc1.weight.wrapped_tensor, fc1.bias, activation="gelu")
            return sten.sparse_linear_fused(h, fc2.weight.wrapped_tensor, fc2.bias, residual=x)
    if op == "ffn_dx":
        y = state["model"](state["x"])
        (dx,) = torch.autograd.grad(y, state["x"], state["dy"])
        return {"y": y.detach(), "dx": dx}
    if op == "train":
        x, lin = state["x"], state["fc1"]
        x.grad = lin.bias.grad = lin.weight.grad = None
        y = lin(x)
        y.backward(state["dy"])
        return {"y": y.detach(), "dx": x.grad, "db": lin.bias.grad, "dw": lin.weight.grad.wrapped_tensor.val}
    n, m, g = state["format"]
    if op == "sparsify":
        t = sten.GroupedNMTensor.from_dense(state["weight"], n, m, sparse_dim=0, group_size=g, group_dim=1)
        return {"val": t.val, "idx": t.idx}
    return state["weight"].to_dense()


def work(case):
    """Every operand read once, every result written once; flops are those of the kept values."""
    es = 4 if case["dtype"] == "f32" else 2
    op, n, m, g = case["op"], case["n"], case["m"], case["g"]
    rows, cols, tokens = case["rows"], case["cols"], case["tokens"]
    cc = math.comb(m, n) * g

    def weight(r, c):  # kept values and their int16 column positions
        slots = -(-r // m) * (-(-c // cc) * cc)
        return slots * (n * es + 2)

    product = 2.0 * rows * cols * tokens * n / m
    if op in ("sparsify", "densify"):
        return {"bytes": rows * cols * es + weight(rows, cols), "flops": 0}
    x, y = tokens * cols * es, tokens * rows * es
    if op in ("linear", "mm"):
        return {"bytes": weight(rows, cols) + x + y + (rows * es if op == "linear" else 0), "flops": product}
    if op == "ffn":
        return {"bytes": weight(rows, cols) + weight(cols, rows) + (rows + cols) * es + 2 * x, "flops": 2 * product}
    if op == "ffn_dx":  # x, dy in; y, dx out; the hidden activation is kept for the backward pass
        return {"bytes": 2 * (weight(rows, cols) + weight(cols, rows)) + (rows + cols) * es + 4 * x + 2 * y, "flops": 4 * product}
    # train: weight, x, dy in; y, dx, db and the packed weight gradient out
    return {"bytes": 2 * weight(rows, cols) + 2 * x + 2 * y + 2 * rows * es, "flops": 3 * product}


def tolerance(case):
    if case["op"] in ("sparsify", "densify"):
        return "exact"
    return {"rel": {"f32": 1e-5, "f16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
