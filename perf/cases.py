"""The work that users of this package have it do, as measurable cases.

Every case is a compiled schedule called the way a serving program calls it:
``CompiledModel(schedule, parameters, Config(), "cuda")`` once, then
``compiled(*inputs)`` per request with the inputs in device memory.  Three families:

* ``shipped`` -- the schedules under ``mlc_compiler_b200/schedules``: BERT-base,
  GPT-2 small, the encoder block and the three fused-kernel modules, at the batch
  sizes and dtypes they are shipped in (sequence 128);
* ``encoder`` -- a stack of post-LN encoder layers (heads of 64, FFN 4x, exact
  GELU, additive padding mask) at any batch, sequence and width, lowered to kernel
  IR in the form the frontend gives the shipped encoder block and BERT-base;
* ``rows`` -- one fused kernel alone over ``[rows, cols]``: LayerNorm, softmax,
  bias + GELU + residual; a softmax or LayerNorm row longer than
  ``Config.max_persistent_row`` takes the streamed form, as the frontend decides it.

Weights are N(0, 0.02), biases N(0, 0.02), LayerNorm gains 1 + N(0, 0.02); token ids
are uniform over the vocabulary, activations N(0, 1), and the sentences of a batch
have lengths between half and all of the sequence, the rest of it masked.
"""

from __future__ import annotations

import functools
import math

import torch

from mlc_compiler_b200 import CompiledModel, Config, kir, load_schedule

#: batch sizes each shipped configuration exists in, by (model, dtype)
SHIPPED = {("bert-base", "float16"): (1, 4, 8, 16, 32), ("bert-base", "bfloat16"): (1, 4, 8, 16, 32),
           ("gpt2-small", "float16"): (1, 4, 8, 16, 32), ("gpt2-small", "bfloat16"): (1, 4, 8, 16, 32),
           ("bert-base", "float32"): (1,), ("encoder-block", "float32"): (1,),
           ("bert-base-streamed", "float16"): (1,), ("gpt2-small-streamed", "float16"): (1,)}
SHIPPED.update({(f"micro-{m}", dt): (1, 8, 32) for m in ("layernorm", "softmax", "gelu")
                for dt in ("float16", "bfloat16")})


def listed() -> list[dict]:
    return [
        # one sentence, answer wanted now: launch count and latency are everything
        dict(name="bert_b1_fp16", kind="shipped", model="bert-base", batch=1, dtype="float16"),
        # a small serving batch
        dict(name="bert_b8_bf16", kind="shipped", model="bert-base", batch=8, dtype="bfloat16"),
        # a throughput batch: matmuls fill the machine
        dict(name="bert_b32_fp16", kind="shipped", model="bert-base", batch=32, dtype="float16"),
        # full precision, one sentence
        dict(name="bert_b1_fp32", kind="shipped", model="bert-base", batch=1, dtype="float32"),
        # scoring one prompt with a decoder (logits over the whole vocabulary)
        dict(name="gpt2_b1_bf16", kind="shipped", model="gpt2-small", batch=1, dtype="bfloat16"),
        # scoring a batch of prompts: the largest shipped configuration
        dict(name="gpt2_b32_fp16", kind="shipped", model="gpt2-small", batch=32, dtype="float16"),
        # a ragged batch of short sentences through a small encoder
        dict(name="encoder_b3_s77_fp16", kind="encoder", batch=3, seq=77, heads=12, layers=4,
             dtype="float16"),
        # long documents through a wide encoder
        dict(name="encoder_b8_s384_bf16", kind="encoder", batch=8, seq=384, heads=16, layers=2,
             dtype="bfloat16"),
        # one LayerNorm of one sentence: the smallest call there is
        dict(name="layernorm_small_fp16", kind="rows", op="layernorm", rows=128, cols=768,
             dtype="float16"),
        # softmax over rows of odd length, full precision
        dict(name="softmax_odd_fp32", kind="rows", op="softmax", rows=3001, cols=1001,
             dtype="float32"),
        # token probabilities over a vocabulary: rows too long for registers
        dict(name="softmax_vocab_fp16", kind="rows", op="softmax", rows=512, cols=50257,
             dtype="float16"),
        # feed-forward activation of a throughput batch
        dict(name="gelu_large_bf16", kind="rows", op="gelu", rows=4096, cols=3072,
             dtype="bfloat16"),
    ]


def draw(rng) -> dict:
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["shipped", "encoder", "encoder", "rows"])
    if kind == "shipped":
        model, dtype = rng.choice(sorted(SHIPPED))
        return dict(kind=kind, model=model, batch=rng.choice(SHIPPED[model, dtype]), dtype=dtype)
    while True:
        if kind == "encoder":
            case = dict(kind=kind, batch=log_int(1, 32), seq=log_int(16, 512),
                        heads=rng.choice([4, 6, 8, 12, 16]), layers=rng.randint(1, 6),
                        dtype=rng.choice(["float16", "bfloat16", "float16", "bfloat16", "float32"]))
            limit = 4e11 if case["dtype"] != "float32" else 4e10
        else:
            case = dict(kind=kind, op=rng.choice(["layernorm", "softmax", "gelu"]),
                        rows=log_int(16, 16384), cols=log_int(48, 65536),
                        dtype=rng.choice(["float16", "bfloat16", "float32"]))
            limit = 1e11
        w = work(case)
        if w["flops"] <= limit and w["bytes"] <= 6e8:
            return case


# --------------------------------------------------------------------------
# kernel IR of the hand-lowered families
# --------------------------------------------------------------------------

def _ref(n):
    return kir.Ref(n)


def _call(fn, *args):
    return kir.Call(fn, args)


def _map(var: str, numel: int, terms) -> kir.Axis:
    return kir.Axis(var, numel, tuple(terms))


def _flat(name: str, buffer: str, dtype: str, numel: int, terms=None) -> kir.Operand:
    return kir.Operand(name, buffer, dtype,
                       kir.IndexMap((_map("idx", numel, terms or [(numel, 1, 1)]),)))


def _row(name: str, dtype: str, rows: int, cols: int, row_terms=None) -> kir.Operand:
    """A ``[rows, cols]`` operand; ``row_terms=[]`` makes it a row all rows share."""
    terms = [(rows, 1, cols)] if row_terms is None else row_terms
    return kir.Operand(name, name, dtype, kir.IndexMap((_map("row", rows, terms),
                                                        _map("col", cols, [(cols, 1, 1)]))))


class _Binds:
    """Numbered temporaries, as the frontend names them."""

    def __init__(self):
        self.steps: list = []

    def bind(self, expr) -> kir.Ref:
        self.steps.append(kir.Bind(f"t{len(self.steps)}", expr))
        return _ref(self.steps[-1].name)

    def reduce(self, kind, expr) -> kir.Ref:
        self.steps.append(kir.Reduce(f"r{len(self.steps)}", kind, expr))
        return _ref(self.steps[-1].name)

    def store(self, expr, dtype) -> kir.Ref:
        return expr if dtype == "float32" else self.bind(kir.Cast(expr, dtype))

    def body(self):
        return [(s.name, s.expr) for s in self.steps]


def _layernorm(name, rows, cols, dtype, summands, gain, bias, out, eps, row_space, streamed=False):
    """LayerNorm of the sum of ``summands`` (operands; a bias row is shared)."""
    b = _Binds()
    x = kir.Load(0)
    if len(summands) == 3:                       # residual + (matmul + its bias)
        x = b.bind(_call("add", kir.Load(0), kir.Load(1)))
        x = b.bind(_call("add", kir.Load(2), x))
    n = len(summands)
    mean = b.bind(_call("div", b.reduce("sum", x), kir.Const(float(cols))))
    d = b.bind(_call("sub", x, mean))
    sq = b.bind(_call("mul", d, d))
    var = b.bind(_call("div", b.reduce("sum", sq), kir.Const(float(cols))))
    inv = b.bind(_call("rsqrt", b.bind(_call("add", var, kir.Const(eps)))))
    y = b.bind(_call("mul", b.bind(_call("mul", d, inv)), kir.Load(n)))
    y = b.store(b.bind(_call("add", y, kir.Load(n + 1))), dtype)
    return kir.ReductionKernel(name, row_space, (cols,), summands + [gain, bias], [out], b.steps,
                               {out.name: y}, set(), streamed, ["layernorm"])


def _softmax(name, rows, cols, dtype, x, mask, out, row_space, streamed=False):
    b = _Binds()
    v = kir.Load(0)
    if mask is not None:
        v = b.bind(_call("div", v, kir.Const(8.0)))
        v = b.bind(_call("add", v, kir.Load(1)))
    e = b.bind(_call("exp", b.bind(_call("sub", v, b.reduce("max", v)))))
    p = b.store(b.bind(_call("div", e, b.reduce("sum", e))), dtype)
    return kir.ReductionKernel(name, row_space, (cols,), [x] + ([mask] if mask is not None else []),
                               [out], b.steps, {out.name: p}, set(), streamed, ["softmax"])


def _gelu(b: _Binds, x, dtype, tanh: bool):
    if tanh:
        cube = b.bind(_call("mul", b.bind(_call("mul", x, x)), x))
        inner = b.bind(_call("add", x, b.bind(_call("mul", cube, kir.Const(0.044715)))))
        inner = b.bind(_call("mul", inner, kir.Const(math.sqrt(2.0 / math.pi))))
        half = b.bind(_call("mul", x, kir.Const(0.5)))
        t = b.bind(_call("tanh", inner))
    else:
        half = b.bind(_call("mul", x, kir.Const(0.5)))
        t = b.bind(_call("erf", b.bind(_call("mul", x, kir.Const(math.sqrt(0.5))))))
    t = b.bind(_call("add", t, kir.Const(1, "int64")))
    return b.store(b.bind(_call("mul", half, t)), dtype)


def rows_schedule(op: str, rows: int, cols: int, dtype: str) -> kir.Schedule:
    """One fused kernel over ``[rows, cols]``."""
    s = kir.Schedule(f"{op}-{rows}x{cols}-{dtype}")

    def buffer(name, shape, kind):
        s.buffers[name] = kir.BufferSpec(name, shape, dtype, kind)
        if kind == "param":
            s.params[name] = name
        elif kind in ("input", "output"):
            strides = tuple(math.prod(shape[i + 1:]) for i in range(len(shape)))
            getattr(s, kind + "s").append(kir.View(name, name, shape, strides))

    streamed = op != "gelu" and cols > Config().max_persistent_row
    buffer("x", (rows, cols), "input")
    out = _row("y", dtype, rows, cols)
    if op == "layernorm":
        buffer("norm.weight", (cols,), "param")
        buffer("norm.bias", (cols,), "param")
        s.kernels.append(_layernorm("k0", rows, cols, dtype, [_row("x", dtype, rows, cols)],
                                    _row("norm.weight", dtype, rows, cols, []),
                                    _row("norm.bias", dtype, rows, cols, []), out, 1e-5, (rows,),
                                    streamed))
    elif op == "softmax":
        s.kernels.append(_softmax("k0", rows, cols, dtype, _row("x", dtype, rows, cols), None, out,
                                  (rows,), streamed))
    else:
        buffer("bias", (cols,), "param")
        buffer("res", (rows, cols), "input")
        n = rows * cols
        b = _Binds()
        g = _gelu(b, b.bind(_call("add", kir.Load(0), kir.Load(1))), dtype, tanh=True)
        y = b.bind(_call("add", kir.Load(2), g))
        s.kernels.append(kir.PointwiseKernel(
            "k0", (rows, cols), [_flat("x", "x", dtype, n), _flat("bias", "bias", dtype, n, [(cols, 1, 1)]),
                                 _flat("res", "res", dtype, n)], [_flat("y", "y", dtype, n)],
            b.body(), {"y": y}, ["gelu"]))
    buffer("y", (rows, cols), "output")
    return s


@functools.lru_cache(maxsize=64)
def encoder_schedule(batch: int, seq: int, heads: int, layers: int, dtype: str) -> kir.Schedule:
    """A stack of encoder layers, kernel for kernel as the frontend lowers them: at
    batch 1 the attention matmuls read views of the projections, above it they read
    head-major copies; the bias adds and GELU are pointwise kernels, softmax and the
    residual LayerNorms row reductions."""
    B, S, H, dh = batch, seq, heads, 64
    D, F, T = H * dh, 4 * H * dh, batch * seq
    s = kir.Schedule(f"encoder-b{B}-s{S}-h{H}-l{layers}-{dtype}")
    names = iter(range(1 << 20))

    def buffer(name, shape, kind="intermediate"):
        s.buffers[name] = kir.BufferSpec(name, shape, dtype, kind)
        if kind == "param":
            s.params[name] = name
        return name

    def extern(op, a, b, out):
        s.kernels.append(kir.ExternKernel(f"k{next(names)}", f"aten.{op}.default", [a, b], {}, [out]))

    def view(buf, shape, strides=None):
        strides = strides or tuple(math.prod(shape[i + 1:]) for i in range(len(shape)))
        return kir.View(buf, buf, shape, strides)

    def linear(x, name, n_in, n_out, out):
        w = buffer(name + ".weight", (n_out, n_in), "param")
        buffer(name + ".bias", (n_out,), "param")
        extern("mm", view(x, (T, n_in)), view(w, (n_in, n_out), (1, n_in)),
               view(buffer(out, (T, n_out)), (T, n_out)))

    def pointwise(space, ins, out, body, expr, op):
        s.kernels.append(kir.PointwiseKernel(f"k{next(names)}", space, ins, [out], body,
                                             {out.name: expr}, [op]))

    def bias_add(mm, name, n, out):
        b = _Binds()
        y = b.bind(_call("add", kir.Load(0), kir.Load(1)))
        pointwise((T, n), [_flat(mm, mm, dtype, T * n), _flat(name, name, dtype, T * n, [(n, 1, 1)])],
                  _flat(buffer(out, (T, n)), out, dtype, T * n), b.body(), y, "add")

    def copy(src, out, space, terms):
        n = math.prod(space)
        pointwise(space, [_flat(src, src, dtype, n, terms)],
                  _flat(buffer(out, space), out, dtype, n), [], kir.Load(0), "clone")

    x = buffer("x", (B, S, D), "input")
    s.inputs.append(view(x, (B, S, D)))
    buffer("mask", (B, 1, 1, S), "input")
    s.inputs.append(view("mask", (B, 1, 1, S)))
    for layer in range(layers):
        p = f"layers.{layer}."
        for j in "qkv":
            linear(x, p + j, D, D, p + j + ".mm")
            bias_add(p + j + ".mm", p + j + ".bias", D, p + j)
        q, k, v = p + "q", p + "k", p + "v"
        if B == 1:
            qv, kv = view(q, (H, S, dh), (dh, D, 1)), view(k, (H, dh, S), (dh, 1, D))
            vv = view(v, (H, S, dh), (dh, D, 1))
        else:
            heads_first = [(B, S * D, S * D), (H, S * dh, dh), (S, dh, D), (dh, 1, 1)]
            copy(q, q + ".heads", (B, H, S, dh), heads_first)
            copy(k, k + ".heads", (B, H, dh, S), [(B, S * D, S * D), (D, S, 1), (S, 1, D)])
            qv, kv = view(q + ".heads", (B * H, S, dh)), view(k + ".heads", (B * H, dh, S))
            vv = view(v + ".heads", (B * H, S, dh))
        scores, probs, ctx = (buffer(p + n, shape) for n, shape in
                              (("scores", (B * H, S, S)), ("probs", (B, H, S, S)), ("ctx", (B * H, S, dh))))
        extern("bmm", qv, kv, view(scores, (B * H, S, S)))
        rows = B * H * S
        s.kernels.append(_softmax(f"k{next(names)}", rows, S, dtype, _row(scores, dtype, rows, S),
                                  _row("mask", dtype, rows, S, [(B, H * S, S)] if B > 1 else []),
                                  _row(probs, dtype, rows, S), (B, H, S)))
        if B > 1:
            copy(v, v + ".heads", (B, H, S, dh), heads_first)
        extern("bmm", view(probs, (B * H, S, S)), vv, view(ctx, (B * H, S, dh)))
        merged = [(S, D, dh), (H, dh, S * dh), (dh, 1, 1)]
        copy(ctx, p + "merged", (B, S, H, dh), ([(B, S * D, S * D)] if B > 1 else []) + merged)
        linear(p + "merged", p + "o", D, D, p + "o.mm")

        def residual_norm(mm, name, res, norm, out, kind="intermediate"):
            buffer(norm + ".weight", (D,), "param")
            buffer(norm + ".bias", (D,), "param")
            buffer(out, (B, S, D), kind)
            s.kernels.append(_layernorm(
                f"k{next(names)}", T, D, dtype,
                [_row(mm, dtype, T, D), _row(name + ".bias", dtype, T, D, []), _row(res, dtype, T, D)],
                _row(norm + ".weight", dtype, T, D, []), _row(norm + ".bias", dtype, T, D, []),
                _row(out, dtype, T, D), 1e-12, (B, S)))
            return out

        h = residual_norm(p + "o.mm", p + "o", x, p + "attn_norm", p + "h")
        linear(h, p + "up", D, F, p + "up.mm")
        b = _Binds()
        g = _gelu(b, b.bind(_call("add", kir.Load(0), kir.Load(1))), dtype, tanh=False)
        pointwise((T, F), [_flat(p + "up.mm", p + "up.mm", dtype, T * F),
                           _flat(p + "up.bias", p + "up.bias", dtype, T * F, [(F, 1, 1)])],
                  _flat(buffer(p + "act", (T, F)), p + "act", dtype, T * F), b.body(), g, "gelu")
        linear(p + "act", p + "down", F, D, p + "down.mm")
        x = residual_norm(p + "down.mm", p + "down", h, p + "ffn_norm", p + "out",
                          "output" if layer == layers - 1 else "intermediate")
    s.outputs.append(view(x, (B, S, D)))
    _plan_arena(s)
    return s


def _plan_arena(s: kir.Schedule) -> None:
    """Greedy arena: largest first, lowest 256-byte aligned offset that clears every
    buffer alive at the same time."""
    first, last = {}, {}
    for i, k in enumerate(s.kernels):
        for b in list(k.reads()) + list(k.writes()):
            if s.buffers[b].plannable:
                first.setdefault(b, i)
                last[b] = i
    placed: list[tuple[int, int, str]] = []
    for b in sorted(first, key=lambda n: (-s.buffers[n].nbytes, first[n])):
        size, offset = -(-s.buffers[b].nbytes // 256) * 256, 0
        for lo, hi, other in sorted(placed):
            if first[b] <= last[other] and first[other] <= last[b] and lo < offset + size and offset < hi:
                offset = hi
        placed.append((offset, offset + size, b))
        s.plan.offsets[b] = offset
    s.plan.arena_bytes = s.plan.peak_bytes = max(hi for _, hi, _ in placed)
    s.plan.total_bytes = sum(s.buffers[b].nbytes for b in first)


@functools.lru_cache(maxsize=64)
def _shipped(model: str, batch: int, dtype: str) -> kir.Schedule:
    return load_schedule(f"{model}_b{batch}_s128_{dtype}")


def _schedule(case: dict) -> kir.Schedule:
    if case["kind"] == "shipped":
        return _shipped(case["model"], case["batch"], case["dtype"])
    if case["kind"] == "encoder":
        return encoder_schedule(case["batch"], case["seq"], case["heads"], case["layers"], case["dtype"])
    return rows_schedule(case["op"], case["rows"], case["cols"], case["dtype"])


# --------------------------------------------------------------------------
# the interface
# --------------------------------------------------------------------------

def _parameter(origin: str, spec: kir.BufferSpec, g: torch.Generator) -> torch.Tensor:
    dt = kir.torch_dtype(spec.dtype)
    if origin == "position_ids":
        return torch.arange(spec.numel, device="cuda", dtype=dt).view(spec.shape)
    if origin in ("causal", "mask"):             # additive causal mask [1, 1, n, n]
        n = spec.shape[-1]
        keep = torch.tril(torch.ones(n, n, device="cuda"))
        return ((1.0 - keep) * torch.finfo(torch.float32).min).to(dt).view(spec.shape)
    t = torch.randn(spec.shape, generator=g, device="cuda") * 0.02
    return (t + 1.0 if origin.endswith("norm.weight") else t).to(dt)


def prepare(case: dict, seed: int) -> dict:
    """The compiled model, called once (which captures its graph), and a request."""
    g = torch.Generator("cuda").manual_seed(seed)
    s = _schedule(case)
    params = {origin: _parameter(origin, s.buffers[b], g) for b, origin in s.params.items()}
    if "tok.weight" in params and "head.weight" in params:      # GPT-2 ties them
        params["head.weight"] = params["tok.weight"]
    inputs = []
    for v in s.inputs:
        spec = s.buffers[v.buffer]
        dt = kir.torch_dtype(spec.dtype)
        if spec.dtype == "int64":
            vocab = s.buffers["p_tok_weight"].shape[0]
            t = torch.randint(0, vocab, v.shape, generator=g, device="cuda")
        elif "mask" in v.buffer:
            # sentences of different lengths: 1 = token (0 additive), 0 = padding
            batch, seq = v.shape[0], v.shape[-1]
            length = torch.randint((seq + 1) // 2, seq + 1, (batch, 1), generator=g, device="cuda")
            keep = (torch.arange(seq, device="cuda")[None] < length).to(dt).view(v.shape)
            t = keep if v.buffer == "attention_mask" else (1 - keep) * torch.finfo(dt).min
        else:
            t = torch.randn(v.shape, generator=g, device="cuda").to(dt)
        inputs.append(t)
    compiled = CompiledModel(s, params, Config(), "cuda")
    compiled(*inputs)
    return {"compiled": compiled, "inputs": inputs}


def run(state: dict):
    return state["compiled"](*state["inputs"])


def work(case: dict) -> dict:
    """Inputs, outputs and every parameter once (of an embedding table, the rows that
    are fetched); two operations per multiply-add of the matmuls, ten per element of a
    lone fused kernel."""
    if case["kind"] == "rows":
        n, item = case["rows"] * case["cols"], kir.ITEMSIZE[case["dtype"]]
        passes = 3 if case["op"] == "gelu" else 2
        return {"bytes": (passes * n + 2 * case["cols"]) * item, "flops": 10 * n}
    if case["kind"] == "encoder":
        item = kir.ITEMSIZE[case["dtype"]]
        B, S, L, D = case["batch"], case["seq"], case["layers"], 64 * case["heads"]
        per_layer = 12 * D * D + 13 * D
        return {"bytes": item * (2 * B * S * D + B * S + L * per_layer),
                "flops": 2 * L * (12 * B * S * D * D + 2 * B * S * S * D)}
    s = _schedule(case)
    tables = {v.buffer for k in s.kernels if isinstance(k, kir.ExternKernel) and "embedding" in k.op
              for v in k.args[:1]}
    matmul_reads = {v.buffer for k in s.kernels if isinstance(k, kir.ExternKernel)
                    and "embedding" not in k.op for v in k._views()}
    tokens, nbytes, flops = case["batch"] * 128, 0, 0
    for b in s.live_buffers():
        spec = s.buffers[b]
        if spec.kind in ("input", "output"):
            nbytes += spec.nbytes
        elif b in s.params:
            rows = tokens if b in tables and b not in matmul_reads else spec.shape[0]
            full = spec.shape[0]
            nbytes += spec.nbytes * min(rows, full) // full
    for k in s.kernels:
        if isinstance(k, kir.ExternKernel) and "embedding" not in k.op:
            flops += 2 * k.outputs[0].numel * k.args[0].shape[-1]
    if not flops:
        flops = 10 * s.buffers[s.outputs[0].buffer].numel
    return {"bytes": nbytes, "flops": flops}


def tolerance(case: dict):
    """Half-precision matmul results are rounded to 11 (fp16) or 8 (bf16) bits after
    every matmul and every fused kernel; a stack of layers accumulates a few such
    roundings.  A lone kernel rounds once, at its store."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5 if case["kind"] != "rows" else 5e-6}
    narrow = {"float16": 1e-3, "bfloat16": 8e-3}[case["dtype"]]
    if case["kind"] == "rows" or case.get("model", "").startswith("micro"):
        return {"rel": narrow / 2, "max": 4 * narrow}
    return {"rel": 2.5 * narrow}
