"""The work that programs have this library do, as cases with inputs, one pass and its outputs.

Each case is a pass through the public entry points: `torch.compile` with the library's backend, the eager
operations of `tessiq_b200.ops` and the registered `torch.ops.tessiq.*`. The sizes are those of the
benchmark's workloads (the fused chain over [4096, 4096], row operations over [32768, 4096] and over its
transposed view, the 8192 x 4096 x 16384 projection, the decoder block of 768 wide tokens, tensors of 2^20
to 2^30 elements) with smaller, odd and ragged ones beside them.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs, weights and compiled functions, on the GPU
    run(state)          one pass, its outputs
    work(case)          bytes and flops that a pass cannot do without
    tolerance(case)     how far another correct implementation at this precision may be off
    exact(case, seed)   the outputs of a pass in 64 bits, from plain torch
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from tessiq_b200 import ops
from tessiq_b200.backend import compile_graph

# every shape compiles for itself (a program that serves several batch sizes keeps one compiled graph for each)
torch._dynamo.config.recompile_limit = 256
torch._dynamo.config.accumulated_recompile_limit = 1024

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
SIZES = {"f32": 4, "bf16": 2, "f16": 2}
EPS = 1e-5


def listed():
    return [
        # a script that works on small tensors with eager operations: launches and host time are all it pays for
        {"name": "eager_small_f32", "kind": "eager", "rows": 64, "width": 512, "dtype": "f32"},
        # the compiled elementwise chain with a bias row, at its ordinary size
        {"name": "chain_4096x4096_f32", "kind": "chain", "rows": 4096, "width": 4096, "dtype": "f32"},
        # six fused operations with a predicate and a cast, then global sum and maximum: a large tensor of odd length
        {"name": "sweep_134217757_bf16", "kind": "sweep", "n": (1 << 27) + 29, "dtype": "bf16"},
        # reductions, softmax and LayerNorm over rows: the large activation tensor
        {"name": "rows_32768x4096_f32", "kind": "rows", "rows": 32768, "width": 4096, "dtype": "f32"},
        # the same over rows of an odd width (class scores, a vocabulary, an unpadded feature count)
        {"name": "rows_20000x1003_bf16", "kind": "rows", "rows": 20000, "width": 1003, "dtype": "bf16"},
        # the same over the last axis of a transposed view, and the packed copy of that view
        {"name": "view_32768x4096_f32", "kind": "view", "rows": 32768, "width": 4096, "dtype": "f32"},
        {"name": "view_5003x1250_bf16", "kind": "view", "rows": 5003, "width": 1250, "dtype": "bf16"},
        # linear layer + bias + GELU: a large batch of tokens, and the few rows of a decoding step
        {"name": "gemm_8192x4096x16384_bf16", "kind": "gemm", "m": 8192, "k": 4096, "n": 16384, "act": "tanh", "dtype": "bf16"},
        {"name": "gemm_64x4096x4096_bf16", "kind": "gemm", "m": 64, "k": 4096, "n": 4096, "act": "tanh", "dtype": "bf16"},
        # attention: causal over whole sequences (prefill), and one new token against the keys so far (decode)
        {"name": "attention_64x12x1024x64_bf16", "kind": "attention", "batch": 64, "heads": 12, "q": 1024, "kv": 1024, "head": 64,
         "causal": True, "dtype": "bf16"},
        {"name": "decode_64x12x1000x64_bf16", "kind": "attention", "batch": 64, "heads": 12, "q": 1, "kv": 1000, "head": 64,
         "causal": False, "dtype": "bf16"},
        # the compiled decoder block, inference, at the batch one GPU of eight serves
        {"name": "block_8x1024_bf16", "kind": "block", "batch": 8, "tokens": 1024, "d": 768, "heads": 12, "dtype": "bf16"},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["eager", "chain", "sweep", "rows", "rows", "view", "view", "gemm", "gemm", "attention", "attention", "block"])
    dtype = rng.choice(["f32", "bf16", "f16"])
    half = rng.choice(["bf16", "bf16", "f16"])
    if kind == "eager":
        return {"kind": kind, "rows": _log(rng, 8, 512), "width": _log(rng, 64, 1024), "dtype": dtype}
    if kind == "chain":
        width = _log(rng, 64, 8192) if rng.random() < 0.4 else rng.choice([768, 1024, 3072, 4096, 8192])
        return {"kind": kind, "rows": max(1, _log(rng, 1 << 14, 1 << 27) // width), "width": width, "dtype": dtype}
    if kind == "sweep":
        return {"kind": kind, "n": _log(rng, 1 << 17, 1 << 27) + rng.choice([0, 0, 1, 5]), "dtype": dtype}
    if kind in ("rows", "view"):
        # up to the size of the large activation tensor; widths a model uses, or any at all
        width = _log(rng, 32, 16384) if rng.random() < 0.5 else rng.choice([768, 1000, 1024, 3072, 4096, 8192])
        rows = max(8, _log(rng, 1 << 16, 1 << 27) // width)
        if kind == "view" and rng.random() < 0.5:
            rows = -(-rows // 64) * 64 if rows >= 64 else 64
        return {"kind": kind, "rows": min(rows, (1 << 27) // width), "width": width, "dtype": dtype}
    if kind == "gemm":
        k, n = rng.choice([(768, 768), (768, 2304), (768, 3072), (3072, 768), (1024, 4096), (4096, 1024), (4096, 4096), (4096, 16384),
                           (8 * _log(rng, 32, 512), 8 * _log(rng, 32, 512)), (768, _log(rng, 1000, 16384))])
        return {"kind": kind, "m": _log(rng, 1, 8192), "k": k, "n": n, "act": rng.choice(["tanh", "tanh", "erf", "none"]), "dtype": half}
    if kind == "attention":
        head = rng.choice([64, 64, 64, 32, 128])
        if rng.random() < 0.5:
            batch, heads, kv = _log(rng, 1, 64), rng.choice([6, 8, 12, 16]), _log(rng, 100, 8192)
            while batch * heads * kv * head > 64 * 12 * 4096 * 64:
                kv //= 2
            return {"kind": kind, "batch": batch, "heads": heads, "q": rng.choice([1, 1, 1, 4]), "kv": kv, "head": head,
                    "causal": False, "dtype": half}
        tokens, heads = _log(rng, 100, 4096), rng.choice([6, 8, 12, 16])
        batch = max(1, int(_log(rng, 1 << 10, 1 << 16) // tokens))
        while batch > 1 and batch * heads * tokens * tokens * head > 64 * 12 * 1024 * 1024 * 64:
            batch -= 1
        return {"kind": kind, "batch": batch, "heads": heads, "q": tokens, "kv": tokens, "head": head, "causal": rng.random() < 0.75,
                "dtype": half}
    tokens = rng.choice([128, 200, 256, 512, 1000, 1024])
    d, heads = rng.choice([(768, 12), (768, 12), (512, 8), (1024, 16)])
    return {"kind": kind, "batch": _log(rng, 1, 32), "tokens": tokens, "d": d, "heads": heads, "dtype": "bf16"}


# ---- the functions and modules that a program compiles ---------------------------------------


def chain(x, b):
    """GELU of the biased value gated by a sigmoid: one fused kernel."""
    return F.gelu(x + b, approximate="tanh") * torch.sigmoid(x) - 0.5 * x


def six_op_chain(a, b, dtype):
    """add, exp, mul, tanh, where on a > 0, cast: one fused kernel."""
    return torch.where(a > 0, torch.tanh(torch.exp(a + b) * b), a).to(dtype)


class Block(torch.nn.Module):
    """A pre-norm decoder block with causal attention, written the plain way."""

    def __init__(self, d, heads):
        super().__init__()
        self.d, self.heads = d, heads
        self.ln1, self.qkv, self.proj = torch.nn.LayerNorm(d), torch.nn.Linear(d, 3 * d), torch.nn.Linear(d, d)
        self.ln2, self.fc, self.out = torch.nn.LayerNorm(d), torch.nn.Linear(d, 4 * d), torch.nn.Linear(4 * d, d)

    def forward(self, x):
        b, n, d = x.shape
        q, k, v = self.qkv(self.ln1(x)).split(d, dim=-1)
        q, k, v = (z.view(b, n, self.heads, d // self.heads).transpose(1, 2) for z in (q, k, v))
        scores = (q @ k.transpose(-1, -2)) / (d // self.heads) ** 0.5
        mask = torch.tril(torch.ones(n, n, dtype=torch.bool, device=x.device))
        scores = scores.masked_fill(~mask, float("-inf"))
        y = (torch.softmax(scores, -1) @ v).transpose(1, 2).reshape(b, n, d)
        x = x + self.proj(y)
        return x + self.out(F.gelu(self.fc(self.ln2(x)), approximate="tanh"))


# ---- cases -----------------------------------------------------------------------------------


def _inputs(case, seed):
    """Tensors and weights, made from the seed alone."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    dtype = DTYPES[case["dtype"]]
    kind = case["kind"]

    def normal(*shape, std=1.0, mean=0.0, to=dtype):
        return torch.empty(shape, device="cuda").normal_(mean, std, generator=g).to(to)

    def uniform(*shape):
        return torch.empty(shape, device="cuda").uniform_(-1.0, 1.0, generator=g).to(dtype)

    state = {"kind": kind, "case": dict(case)}
    if kind == "eager":
        rows, width = case["rows"], case["width"]
        state.update(x=normal(rows, width), b=normal(width, std=0.02), gamma=normal(width, std=0.02, mean=1.0),
                     beta=normal(width, std=0.02), mean=normal(width, std=0.1), var=normal(width, std=0.1).abs() + 1)
    elif kind == "chain":
        state.update(x=normal(case["rows"], case["width"]), b=normal(case["width"], std=0.02))
    elif kind == "sweep":
        state.update(a=uniform(case["n"]), b=uniform(case["n"]), to=torch.bfloat16 if dtype == torch.float32 else torch.float32)
    elif kind in ("rows", "view"):
        extent = case["width"] if kind == "rows" else case["rows"]
        state.update(x=normal(case["rows"], case["width"]), gamma=normal(extent, std=0.02, mean=1.0), beta=normal(extent, std=0.02))
    elif kind == "gemm":
        m, k, n = case["m"], case["k"], case["n"]
        # a Linear's weight is [n, k]; unit-variance results put the GELU where it bends
        state.update(x=normal(m, k), w=normal(n, k, std=k ** -0.5), bias=normal(n, std=0.02))
    elif kind == "attention":
        batch, heads, q, kv, head = (case[name] for name in ("batch", "heads", "q", "kv", "head"))
        if q == kv:      # views of a fused projection's result
            qkv = normal(batch, q, 3 * heads * head)
            state.update(zip("qkv", (z.view(batch, q, heads, head).transpose(1, 2) for z in qkv.split(heads * head, dim=-1))))
        else:            # the new tokens' queries against a cache
            state.update(q=normal(batch, q, heads, head).transpose(1, 2), k=normal(batch, heads, kv, head), v=normal(batch, heads, kv, head))
    else:
        d = case["d"]
        block = Block(d, case["heads"]).cuda().eval().requires_grad_(False)
        for p in block.parameters():
            p.copy_(normal(*p.shape, std=0.02, to=torch.float32))
        for norm in (block.ln1, block.ln2):
            norm.weight.add_(1.0)
        state.update(x=normal(case["batch"], case["tokens"], d), block=block.to(dtype))
    return state


def prepare(case, seed):
    state = _inputs(case, seed)
    kind = state["kind"]
    if kind == "gemm":
        ops.register_custom_ops()
    elif kind in ("chain", "sweep", "block"):
        function = {"chain": chain, "sweep": six_op_chain}.get(kind) or state["block"]
        state["fn"] = torch.compile(function, backend=compile_graph, dynamic=False)
    return state


def _six(x, gamma, beta):
    return {"sum": ops.sum(x, -1), "mean": ops.mean(x, -1), "amax": ops.amax(x, -1), "argmax": ops.argmax(x, -1),
            "softmax": ops.softmax(x, -1), "layer_norm": ops.layer_norm(x, [x.shape[-1]], gamma, beta, EPS)}


def run(state):
    kind = state["kind"]
    with torch.no_grad():
        if kind == "eager":
            x = state["x"]
            y = ops.elementwise("gelu_tanh", ops.elementwise("add", x, state["b"]))
            out = {"y": y, "scaled": ops.elementwise("mul", y, 0.5), "packed": ops.contiguous(y.t())}
            out["batch_norm"] = ops.batch_norm_eval(y, state["gamma"], state["beta"], state["mean"], state["var"], EPS)
            out.update(_six(y, state["gamma"], state["beta"]))
            return out
        if kind == "chain":
            return state["fn"](state["x"], state["b"])
        if kind == "sweep":
            a = state["a"]
            return {"chain": state["fn"](a, state["b"], state["to"]), "sum": ops.sum(a), "amax": ops.amax(a)}
        if kind == "rows":
            return _six(state["x"], state["gamma"], state["beta"])
        if kind == "view":
            view = state["x"].t()
            return dict(_six(view, state["gamma"], state["beta"]), packed=ops.contiguous(view))
        if kind == "gemm":
            x, w, bias = state["x"], state["w"], state["bias"]
            act = state["case"]["act"]
            if act == "tanh":
                return torch.ops.tessiq.gemm_bias_gelu_tanh(x, w, bias)
            if act == "erf":
                return torch.ops.tessiq.gemm_bias_gelu(x, w, bias)
            return ops.addmm(bias, x, w.t())
        if kind == "attention":
            return ops.attention(state["q"], state["k"], state["v"], None, state["case"]["causal"])
        return state["fn"](state["x"])


def _six_bytes(rows, width, size):
    """sum, mean, amax, argmax read the tensor and write a value (argmax: eight bytes) a row; the other two write it whole."""
    n = rows * width
    return 6 * n * size + 2 * n * size + rows * (3 * size + 8) + 2 * width * size


def work(case):
    kind, size = case["kind"], SIZES[case["dtype"]]
    if kind == "eager":
        n, width = case["rows"] * case["width"], case["width"]
        return {"bytes": 10 * n * size + 5 * width * size + _six_bytes(case["rows"], width, size), "flops": 40 * n}
    if kind == "chain":
        n = case["rows"] * case["width"]
        return {"bytes": (2 * n + case["width"]) * size, "flops": 20 * n}
    if kind == "sweep":
        n = case["n"]
        return {"bytes": n * (4 * size + (2 if size == 4 else 4)), "flops": 20 * n}
    if kind in ("rows", "view"):
        n = case["rows"] * case["width"]
        outer, extent = (case["rows"], case["width"]) if kind == "rows" else (case["width"], case["rows"])
        return {"bytes": _six_bytes(outer, extent, size) + (2 * n * size if kind == "view" else 0), "flops": 20 * n}
    if kind == "gemm":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": (m * k + k * n + n + m * n) * size, "flops": 2 * m * k * n}
    if kind == "attention":
        batch, heads, q, kv, head = (case[name] for name in ("batch", "heads", "q", "kv", "head"))
        pairs = q * (q + 1) // 2 if case["causal"] else q * kv
        return {"bytes": 2 * batch * heads * (q + kv) * head * size, "flops": 4 * batch * heads * pairs * head}
    batch, tokens, d = case["batch"], case["tokens"], case["d"]
    rows = batch * tokens
    return {"bytes": (2 * rows * d + 12 * d * d + 13 * d) * size, "flops": 24 * rows * d * d + 2 * batch * tokens * (tokens + 1) * d}


def tolerance(case):
    # About four times what the results are off from the same in 64 bits. 32-bit: sums in another order and exponentials to
    # a few units in the last place (3e-7, a single value 9e-7; a global sum of signed values cancels to a small one).
    # 16-bit: a rounding each of the result and, in attention, the probabilities (2.5e-3, a value 2.4e-2 for bf16).
    # argmax is whole: the lowest index of the largest value, whatever the order.
    if case["dtype"] == "f32":
        return {"rel": 1e-5, "max": 1e-5} if case["kind"] == "sweep" else {"rel": 2e-6, "max": 1e-5}
    scale = 1.0 if case["dtype"] == "bf16" else 0.125
    return {"rel": 1e-2 * scale, "max": 0.1 * scale}


def _six_exact(x, gamma, beta):
    # argmax picks among equal values by its own rule: its result is whole and is compared as such
    return {"sum": x.sum(-1), "mean": x.mean(-1), "amax": x.amax(-1), "argmax": None, "softmax": torch.softmax(x, -1),
            "layer_norm": F.layer_norm(x, [x.shape[-1]], gamma, beta, EPS)}


def exact(case, seed):
    state = _inputs(case, seed)
    kind = state["kind"]
    s = {name: value.double() for name, value in state.items() if isinstance(value, torch.Tensor)}
    with torch.no_grad():
        if kind == "eager":
            y = F.gelu(s["x"] + s["b"], approximate="tanh")
            out = {"y": y, "scaled": y * 0.5, "packed": y.t().contiguous()}
            out["batch_norm"] = F.batch_norm(y, s["mean"], s["var"], s["gamma"], s["beta"], False, 0.0, EPS)
            out.update(_six_exact(y, s["gamma"], s["beta"]))
            return out
        if kind == "chain":
            return chain(s["x"], s["b"])
        if kind == "sweep":
            return {"chain": six_op_chain(s["a"], s["b"], torch.float64), "sum": s["a"].sum(), "amax": s["a"].amax()}
        if kind == "rows":
            return _six_exact(s["x"], s["gamma"], s["beta"])
        if kind == "view":
            view = s["x"].t()
            return dict(_six_exact(view, s["gamma"], s["beta"]), packed=view.contiguous())
        if kind == "gemm":
            y = F.linear(s["x"], s["w"], s["bias"])
            act = case["act"]
            return y if act == "none" else F.gelu(y, approximate="tanh" if act == "tanh" else "none")
        if kind == "attention":
            outs = []
            for q, k, v in zip(s["q"], s["k"], s["v"]):     # one sequence after another: the scores of all are large
                scores = (q @ k.transpose(-1, -2)) / case["head"] ** 0.5
                if case["causal"]:
                    n = scores.shape[-1]
                    scores = scores.masked_fill(~torch.ones(n, n, dtype=torch.bool, device=q.device).tril(), float("-inf"))
                outs.append(torch.softmax(scores, -1) @ v)
            return torch.stack(outs)
        block = state["block"].double()
        return torch.cat([block(part) for part in s["x"].split(4)])
