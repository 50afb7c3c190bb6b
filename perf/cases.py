"""The calls this backend is timed on: compiled modules called with tensors on the GPU.

A case is one module a user compiles (a Linear, an MLP, a LayerNorm, a softmax, an activation, a
pre-LN transformer block for one sequence or a batch of them) at one size and precision, called
through ``GPUExecutable``, or a server's step of several requests in flight through
``StreamedBatch``.  The launch plans are the ones Kiln's passes produce for these modules, written
here for any size: one kernel per fusion group, intermediates placed in the arena largest first at
the lowest free offset.
"""

import os
import sys
from math import prod

import numpy as np
import torch

sys.path.insert(1, os.path.join(os.getcwd(), "kiln-compiler_b200"))

from kiln_b200.codegen import program_from_plan  # noqa: E402
from kiln_b200.runtime import GPUExecutable, StreamedBatch  # noqa: E402
from kiln_b200.spec import KernelSpec, NodeSpec, OperandSpec, PlanSpec  # noqa: E402

PRECISIONS = ("fp32", "tf32", "bf16")
ALIGNMENT = 64          # bytes, of every planned buffer


# ---- launch plans ---------------------------------------------------------------------------

def _strides(shape):
    return tuple(prod(shape[i + 1:]) for i in range(len(shape)))


class _View:
    """A tensor of the plan seen with some shape, offset and strides."""

    def __init__(self, buffer, shape, offset=0, strides=None):
        self.buffer, self.shape, self.offset = buffer, tuple(shape), offset
        self.strides = tuple(strides) if strides else _strides(shape)

    def as_(self, shape, strides=None, offset=0):
        return _View(self.buffer, shape, self.offset + offset, strides)


class _Plan:
    """Collects kernels, then places the arena buffers."""

    def __init__(self, name, input_shape, output_shape):
        self.name, self.input_shape, self.output_shape = name, tuple(input_shape), tuple(output_shape)
        self.consts, self.kernels, self.sizes, self.uses = {}, [], {}, {}
        self.x = _View(("input", 0), input_shape)
        self.y = _View(("output", 0), output_shape)

    def const(self, name, *shape):
        self.consts[name] = tuple(shape)
        return _View(("const", name), shape)

    def buffer(self, *shape):
        key = ("arena", len(self.sizes))
        self.sizes[key] = -(-prod(shape) * 4 // ALIGNMENT) * ALIGNMENT
        return _View(key, shape)

    def kernel(self, kind, nodes, inputs, outputs):
        """``nodes``: (op, inputs, shape[, attrs]); ``outputs``: (node index, view)."""
        for v in list(inputs) + [v for _, v in outputs]:
            self.uses.setdefault(v.buffer, []).append(len(self.kernels))
        self.kernels.append((kind, nodes, inputs, outputs))

    def _place(self):
        """Byte offsets of the arena buffers: largest first, each at the lowest offset that is free
        over its whole life (ties: the one defined first)."""
        placed, end = {}, 0
        for key in sorted(self.sizes, key=lambda k: (-self.sizes[k], self.uses[k][0])):
            lo, hi, size = min(self.uses[key]), max(self.uses[key]), self.sizes[key]
            busy = sorted((o, o + self.sizes[k]) for k, o in placed.items()
                          if min(self.uses[k]) <= hi and lo <= max(self.uses[k]))
            at = 0
            for b, e in busy:
                if at + size <= b:
                    break
                at = max(at, e)
            placed[key] = at
            end = max(end, at + size)
        return placed, end

    def spec(self):
        placed, arena_bytes = self._place()

        def operand(v):
            if v.buffer[0] == "arena":
                return OperandSpec(("arena",), placed[v.buffer] // 4 + v.offset, v.shape, v.strides)
            return OperandSpec(v.buffer, v.offset, v.shape, v.strides)

        kernels = []
        for i, (kind, nodes, inputs, outputs) in enumerate(self.kernels):
            kernels.append(KernelSpec(f"k{i}", kind, [NodeSpec(n[0], n[1], tuple(n[2]), dict(n[3]) if len(n) > 3 else {}) for n in nodes],
                                      [operand(v) for v in inputs], [(j, operand(v)) for j, v in outputs]))
        return PlanSpec(self.name, [self.input_shape], [self.output_shape], arena_bytes, dict(self.consts), kernels)

    # -- the fusion groups Kiln makes of these modules --

    def layernorm(self, x, prefix, out, add=None, sum_out=None):
        shape, d = x.shape, x.shape[-1]
        row = shape[:-1] + (1,)
        dims, inv, eps = {"dims": [len(shape) - 1]}, float(np.float32(1.0 / d)), float(np.float32(1e-5))
        inputs = [x] + ([add] if add else []) + [self.const(prefix + "weight", d), self.const(prefix + "bias", d)]
        nodes = [("add", [("operand", 0), ("operand", 1)], shape)] if add else []
        n = len(nodes)
        v = ("node", 0) if add else ("operand", 0)
        nodes += [("reduce_sum", [v], row, dims), ("mul", [("node", n), ("scalar", inv)], row), ("sub", [v, ("node", n + 1)], shape),
                  ("mul", [("node", n + 2), ("node", n + 2)], shape), ("reduce_sum", [("node", n + 3)], row, dims),
                  ("mul", [("node", n + 4), ("scalar", inv)], row), ("add", [("node", n + 5), ("scalar", eps)], row),
                  ("rsqrt", [("node", n + 6)], row), ("mul", [("node", n + 2), ("node", n + 7)], shape),
                  ("mul", [("node", n + 8), ("operand", len(inputs) - 2)], shape),
                  ("add", [("node", n + 9), ("operand", len(inputs) - 1)], shape)]
        self.kernel("reduction", nodes, inputs, ([(0, sum_out)] if sum_out else []) + [(n + 10, out)])

    def softmax(self, x, out, scale=None, mask=None):
        shape = x.shape
        row, dims = shape[:-1] + (1,), {"dims": [len(shape) - 1]}
        nodes, v, inputs = [], ("operand", 0), [x]
        if scale is not None:
            nodes = [("mul", [v, ("scalar", scale)], shape), ("add", [("node", 0), ("operand", 1)], shape)]
            v, inputs = ("node", 1), [x, mask]
        n = len(nodes)
        nodes += [("reduce_max", [v], row, dims), ("sub", [v, ("node", n)], shape), ("exp", [("node", n + 1)], shape),
                  ("reduce_sum", [("node", n + 2)], row, dims), ("div", [("node", n + 2), ("node", n + 3)], shape)]
        self.kernel("reduction", nodes, inputs, [(n + 4, out)])

    def linear(self, x, prefix, n, out, gelu=False, residual=None):
        m, k = x.shape
        nodes = [("matmul", [("operand", 0), ("operand", 1)], (m, n)), ("add", [("node", 0), ("operand", 2)], (m, n))]
        inputs = [x, self.const(prefix + "weight.transpose", k, n), self.const(prefix + "bias", n)]
        if gelu:
            nodes.append(("gelu", [("node", 1)], (m, n), {"approximate": "tanh"}))
        if residual is not None:
            nodes.append(("add", [("operand", 3), ("node", 1)], (m, n)))
            inputs.append(residual)
        self.kernel("matmul", nodes, inputs, [(len(nodes) - 1, out)])

    def copy(self, x, out):
        self.kernel("copy", [("copy", [("operand", 0)], x.shape)], [x], [(0, out)])

    def bmm(self, a, b, out, scale=None, mask=None):
        nodes, inputs = [("matmul", [("operand", 0), ("operand", 1)], out.shape)], [a, b]
        if scale is not None:
            nodes += [("mul", [("node", 0), ("scalar", scale)], out.shape), ("add", [("node", 1), ("operand", 2)], out.shape)]
            inputs.append(mask)
        self.kernel("matmul", nodes, inputs, [(len(nodes) - 1, out)])


def _block_plan(t, heads):
    """Pre-LN block for one sequence [t, d]."""
    d, hd = 64 * heads, 64
    p = _Plan("block", (t, d), (t, d))
    h, qkv = p.buffer(t, d), p.buffer(t, 3 * d)
    p.layernorm(p.x, "ln1.", h)
    p.linear(h, "c_attn.", 3 * d, qkv)
    kt = p.buffer(heads, hd, t)
    p.copy(qkv.as_((heads, hd, t), (hd, 1, 3 * d), d), kt)
    s, w, o, merged = p.buffer(heads, t, t), p.buffer(heads, t, t), p.buffer(heads, t, hd), p.buffer(t, heads, hd)
    p.bmm(qkv.as_((heads, t, hd), (hd, 3 * d, 1)), kt, s, 0.125, p.const("mask", t, t))
    p.softmax(s, w)
    p.bmm(w, qkv.as_((heads, t, hd), (hd, 3 * d, 1), 2 * d), o)
    p.copy(o.as_((t, heads, hd), (hd, t * hd, 1)), merged)
    x1, h2, f = p.buffer(t, d), p.buffer(t, d), p.buffer(t, 4 * d)
    p.linear(merged.as_((t, d)), "c_proj.", d, x1, residual=p.x)
    p.layernorm(x1, "ln2.", h2)
    p.linear(h2, "fc.", 4 * d, f, gelu=True)
    p.linear(f, "proj.", d, p.y, residual=x1)
    return p.spec()


def _batched_block_plan(b, t, heads):
    """The same block for [b, t, d]: Linears on b * t rows, attention per sequence and head."""
    d, hd = 64 * heads, 64
    p = _Plan("batched_block", (b, t, d), (b, t, d))
    h, qkv = p.buffer(b, t, d), p.buffer(b * t, 3 * d)
    p.layernorm(p.x, "ln1.", h)
    p.linear(h.as_((b * t, d)), "c_attn.", 3 * d, qkv)
    q, kt = p.buffer(b, heads, t, hd), p.buffer(b, heads, hd, t)
    p.copy(qkv.as_((b, heads, t, hd), (t * 3 * d, hd, 3 * d, 1)), q)
    p.copy(qkv.as_((b, heads, hd, t), (t * 3 * d, hd, 1, 3 * d), d), kt)
    s, w = p.buffer(b * heads, t, t), p.buffer(b, heads, t, t)
    p.bmm(q.as_((b * heads, t, hd)), kt.as_((b * heads, hd, t)), s)
    p.softmax(s.as_((b, heads, t, t)), w, 0.125, p.const("mask", t, t))
    v, o, merged = p.buffer(b, heads, t, hd), p.buffer(b * heads, t, hd), p.buffer(b, t, heads, hd)
    p.copy(qkv.as_((b, heads, t, hd), (t * 3 * d, hd, 3 * d, 1), 2 * d), v)
    p.bmm(w.as_((b * heads, t, t)), v.as_((b * heads, t, hd)), o)
    p.copy(o.as_((b, t, heads, hd), (heads * t * hd, hd, t * hd, 1)), merged)
    a, x1, h2 = p.buffer(b * t, d), p.buffer(b, t, d), p.buffer(b, t, d)
    p.linear(merged.as_((b * t, d)), "c_proj.", d, a)
    p.layernorm(p.x, "ln2.", h2, add=a.as_((b, t, d)), sum_out=x1)
    f, g, z = p.buffer(b * t, 4 * d), p.buffer(b, t, 4 * d), p.buffer(b * t, d)
    p.linear(h2.as_((b * t, d)), "fc.", 4 * d, f)
    p.kernel("elementwise", [("gelu", [("operand", 0)], g.shape, {"approximate": "tanh"})], [f.as_((b, t, 4 * d))], [(0, g)])
    p.linear(g.as_((b * t, 4 * d)), "proj.", d, z)
    p.kernel("elementwise", [("add", [("operand", 0), ("operand", 1)], (b, t, d))], [x1, z.as_((b, t, d))], [(0, p.y)])
    return p.spec()


def _plan(c):
    kind = c["kind"]
    if kind == "linear":
        p = _Plan("linear", (c["m"], c["k"]), (c["m"], c["n"]))
        p.linear(p.x, "", c["n"], p.y)
    elif kind == "mlp":
        t, d = c["tokens"], c["d"]
        p = _Plan("mlp", (t, d), (t, d))
        f = p.buffer(t, 4 * d)
        p.linear(p.x, "0.", 4 * d, f, gelu=True)
        p.linear(f, "2.", d, p.y)
    elif kind == "layernorm":
        p = _Plan("layernorm", (c["rows"], c["d"]), (c["rows"], c["d"]))
        p.layernorm(p.x, "", p.y)
    elif kind == "softmax":
        shape = (c["heads"], c["rows"], c["cols"])
        p = _Plan("softmax", shape, shape)
        p.softmax(p.x, p.y)
    elif kind == "bias_gelu":
        shape = (c["rows"], c["d"])
        p = _Plan("bias_gelu", shape, shape)
        p.kernel("elementwise", [("add", [("operand", 0), ("operand", 1)], shape), ("gelu", [("node", 0)], shape, {"approximate": "tanh"})],
                 [p.x, p.const("bias", c["d"])], [(1, p.y)])
    elif kind == "block":
        return _block_plan(c["tokens"], c["heads"])
    else:
        return _batched_block_plan(c["batch"], c["tokens"], c["heads"])
    return p.spec()


# ---- the cases ------------------------------------------------------------------------------

def listed():
    return [
        # one token through a Linear: decoding, the smallest call (latency)
        {"name": "linear_decode", "kind": "linear", "m": 1, "n": 3072, "k": 768, "precision": "fp32"},
        # the projection behind a 128-token prompt's MLP: few tiles, long K
        {"name": "linear_128_tf32", "kind": "linear", "m": 128, "n": 768, "k": 3072, "precision": "tf32"},
        # a Linear over 2048 tokens, the Linear this backend is quoted on
        {"name": "linear_2048_bf16", "kind": "linear", "m": 2048, "n": 3072, "k": 768, "precision": "bf16"},
        # a Linear whose sizes are no multiple of anything (feature counts as data sets have them)
        {"name": "linear_odd_tf32", "kind": "linear", "m": 333, "n": 1000, "k": 771, "precision": "tf32"},
        # two-layer MLP over 2048 tokens
        {"name": "mlp_2048_tf32", "kind": "mlp", "tokens": 2048, "d": 768, "precision": "tf32"},
        # the memory-bound modules on their own
        {"name": "layernorm", "kind": "layernorm", "rows": 2048, "d": 768, "precision": "fp32"},
        {"name": "softmax", "kind": "softmax", "heads": 12, "rows": 512, "cols": 512, "precision": "fp32"},
        {"name": "bias_gelu", "kind": "bias_gelu", "rows": 2048, "d": 3072, "precision": "fp32"},
        # a short prompt through the GPT-2-small block: latency
        {"name": "block_128_tf32", "kind": "block", "tokens": 128, "heads": 12, "precision": "tf32"},
        # a full context in the default precision
        {"name": "block_1024_fp32", "kind": "block", "tokens": 1024, "heads": 12, "precision": "fp32"},
        # a batch of prompts padded to its longest, whose length is whatever it is
        {"name": "batch_6x333_bf16", "kind": "batched_block", "batch": 6, "tokens": 333, "heads": 12, "precision": "bf16"},
        # a server's step: 64 full contexts, eight modules of eight sequences in flight
        {"name": "serve_64x1024_bf16", "kind": "serve", "modules": 8, "batch": 8, "tokens": 1024, "heads": 12, "precision": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _width(rng, lo, hi):
    """A layer width: mostly a multiple of 64, sometimes of 8, sometimes anything."""
    n, kind = _log(rng, lo, hi), rng.random()
    step = 64 if kind < 0.5 else 8 if kind < 0.75 else 1
    return max(step, n // step * step)


def draw(rng):
    kind = rng.choice(["linear", "linear", "mlp", "layernorm", "softmax", "bias_gelu", "block", "block", "batched_block", "serve"])
    c = {"kind": kind, "precision": rng.choice(PRECISIONS)}
    if kind == "linear":
        c.update(m=_log(rng, 1, 4096), n=_width(rng, 64, 4096), k=_width(rng, 64, 4096))
    elif kind == "mlp":
        c.update(tokens=_log(rng, 1, 4096), d=_width(rng, 128, 1024))
    elif kind == "layernorm":
        c.update(rows=_log(rng, 16, 16384), d=_width(rng, 64, 9000), precision="fp32")
    elif kind == "softmax":
        c.update(heads=_log(rng, 1, 16), rows=_log(rng, 16, 1024), cols=_width(rng, 16, 4096), precision="fp32")
    elif kind == "bias_gelu":
        c.update(rows=_log(rng, 16, 8192), d=_width(rng, 64, 4096), precision="fp32")
    elif kind == "block":
        c.update(tokens=_log(rng, 16, 2048), heads=rng.choice([4, 8, 12, 16]))
    elif kind == "batched_block":
        c.update(batch=rng.randint(2, 8), tokens=_log(rng, 16, 1024), heads=rng.choice([4, 8, 12]))
    else:
        c.update(modules=rng.randint(2, 4), batch=rng.randint(2, 8), tokens=_log(rng, 64, 1024), heads=rng.choice([4, 8, 12]), precision="bf16")
    return c


def _constants(shapes, rng):
    """Weights N(0, 0.02) in a block or MLP, N(0, 1 / sqrt(K)) in a Linear alone; biases small; LayerNorm
    scales about 1; the causal mask."""
    out = {}
    for name, shape in shapes.items():
        if name == "mask":
            a = np.zeros(shape, np.float32)
            a[np.triu_indices(shape[0], 1)] = -np.inf
        else:
            a = rng.standard_normal(shape, dtype=np.float32)
            if name.endswith("transpose"):
                a *= np.float32(0.02 if "." in name[:-len("weight.transpose")] else shape[0] ** -0.5)
            elif name.endswith("weight"):
                a = 1 + np.float32(0.1) * a
            else:
                a *= np.float32(0.1 if len(shapes) < 3 and "weight.transpose" not in shapes else 0.01)
        out[name] = a
    return out


def prepare(case, seed):
    plan = _plan(case)
    consts = _constants(plan.const_shapes, np.random.default_rng(seed))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    std = case["k"] ** -0.5 if case["kind"] == "linear" else 3.0 if case["kind"] == "softmax" else 1.0

    def tensor():
        return torch.randn(plan.input_shapes[0], generator=gen, device="cuda") * std

    program = program_from_plan(plan, case["precision"])
    if case["kind"] != "serve":
        return {"call": GPUExecutable(program, plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes), "x": tensor()}
    modules = [GPUExecutable(program, plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes, cuda_graphs=False)
               for _ in range(case["modules"])]
    sources = [tensor() for _ in modules]
    sinks = [torch.empty(plan.output_shapes[0], device="cuda") for _ in modules]
    return {"step": StreamedBatch(modules, concurrency=1).capture(sources, sinks), "sources": sources, "sinks": sinks}


def run(state):
    if "call" in state:
        return state["call"](state["x"])
    state["step"].run()
    return state["sinks"]


def work(case):
    """Inputs and weights read once, outputs written once; a causal score is half of the square."""
    kind = case["kind"]
    word = 2 if case["precision"] == "bf16" else 4          # weights are kept in the operand type
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 4 * (m * k + m * n + n) + word * n * k, "flops": 2 * m * n * k}
    if kind == "mlp":
        t, d = case["tokens"], case["d"]
        return {"bytes": 4 * (2 * t * d + 5 * d) + word * 8 * d * d, "flops": 16 * t * d * d}
    if kind == "layernorm":
        return {"bytes": 4 * (2 * case["rows"] * case["d"] + 2 * case["d"]), "flops": 8 * case["rows"] * case["d"]}
    if kind == "softmax":
        n = case["heads"] * case["rows"] * case["cols"]
        return {"bytes": 8 * n, "flops": 5 * n}
    if kind == "bias_gelu":
        n = case["rows"] * case["d"]
        return {"bytes": 8 * n + 4 * case["d"], "flops": 10 * n}
    t, d = case["tokens"], 64 * case["heads"]
    batch = case.get("batch", 1) * case.get("modules", 1)
    return {"bytes": 8 * batch * t * d + word * 12 * d * d, "flops": batch * (24 * t * d * d + 2 * t * t * d)}


def tolerance(case):
    """Relative error of a result whose matmul operands are rounded to the precision's type (float32
    sums in every precision)."""
    if case["kind"] in ("layernorm", "softmax", "bias_gelu"):
        return {"rel": 1e-5}
    return {"rel": {"fp32": 1e-5, "tf32": 2e-3, "bf16": 1e-2}[case["precision"]]}
