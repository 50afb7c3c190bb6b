"""Exact FP32 on float16 pairs: a producer splits its rows for one reader.  Two Linears behind the same attention, LayerNorm or bounded
Linear, each against float64."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

BOUND = 6e-7          # a matmul of this precision (see test_gpu_exact.py)


def run(plan, x, bias=0, **env):
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    with pytest.MonkeyPatch.context() as patch:
        for name, value in env.items():
            patch.setenv(name, value)
        exe = GPUExecutable(program_from_plan(plan, "fp32"), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    outs = [exe(x)[0] for _ in range(3)]
    exe.status()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    return exe, {name: torch.from_numpy(c).cuda().double() for name, c in consts.items()}, outs[0].double()


def linear(c, v, prefix):
    return v @ c[prefix + "weight.transpose"] + c[prefix + "bias"]


def norm(c, v, prefix):
    return torch.nn.functional.layer_norm(v, v.shape[-1:], c[prefix + "weight"], c[prefix + "bias"], 1e-5)


def attention(p, t, heads, batch):
    """The nodes of a block up to its merged heads."""
    d, hd, rows = 64 * heads, 64, t * (batch or 1)
    if not batch:
        h, qkv, kt = p.buffer(t, d), p.buffer(t, 3 * d), p.buffer(heads, hd, t)
        p.layernorm(p.x, "ln.", h)
        p.linear(h, "qkv.", 3 * d, qkv)
        p.copy(qkv.as_((heads, hd, t), (hd, 1, 3 * d), d), kt)
        s, w, o, merged = p.buffer(heads, t, t), p.buffer(heads, t, t), p.buffer(heads, t, hd), p.buffer(t, heads, hd)
        p.bmm(qkv.as_((heads, t, hd), (hd, 3 * d, 1)), kt, s, 0.125, p.const("mask", t, t))
        p.softmax(s, w)
        p.bmm(w, qkv.as_((heads, t, hd), (hd, 3 * d, 1), 2 * d), o)
        p.copy(o.as_((t, heads, hd), (hd, t * hd, 1)), merged)
        return merged.as_((rows, d))
    h, qkv = p.buffer(batch, t, d), p.buffer(rows, 3 * d)
    p.layernorm(p.x, "ln.", h)
    p.linear(h.as_((rows, d)), "qkv.", 3 * d, qkv)
    q, kt = p.buffer(batch, heads, t, hd), p.buffer(batch, heads, hd, t)
    p.copy(qkv.as_((batch, heads, t, hd), (t * 3 * d, hd, 3 * d, 1)), q)
    p.copy(qkv.as_((batch, heads, hd, t), (t * 3 * d, hd, 1, 3 * d), d), kt)
    s, w = p.buffer(batch * heads, t, t), p.buffer(batch, heads, t, t)
    p.bmm(q.as_((batch * heads, t, hd)), kt.as_((batch * heads, hd, t)), s)
    p.softmax(s.as_((batch, heads, t, t)), w, 0.125, p.const("mask", t, t))
    v, o, merged = p.buffer(batch, heads, t, hd), p.buffer(batch * heads, t, hd), p.buffer(batch, t, heads, hd)
    p.copy(qkv.as_((batch, heads, t, hd), (t * 3 * d, hd, 3 * d, 1), 2 * d), v)
    p.bmm(w.as_((batch * heads, t, t)), v.as_((batch * heads, t, hd)), o)
    p.copy(o.as_((batch, t, heads, hd), (heads * t * hd, hd, t * hd, 1)), merged)
    return merged.as_((rows, d))


@pytest.mark.parametrize("kernel", ["", "fma"])
@pytest.mark.parametrize("tokens,batch,n", [(1024, None, 768), (333, None, 3072), (333, 6, 768), (1024, 2, 768)])
def test_two_linears_on_the_merged_heads(tokens, batch, n, kernel):
    from perf import cases

    heads, d, rows = 12, 768, tokens * (batch or 1)
    p = cases._Plan("two_readers", (batch, tokens, d) if batch else (tokens, d), (rows, n))
    merged, a = attention(p, tokens, heads, batch), p.buffer(rows, n)
    p.linear(merged, "out.", n, a)
    p.linear(merged, "gate.", n, p.y, residual=a)
    plan = p.spec()
    x = torch.randn(plan.input_shapes[0], generator=torch.Generator(device="cuda").manual_seed(0), device="cuda")
    exe, c, got = run(plan, x, KILN_GPU_FP32_ATTENTION=kernel)
    readers = [detail for detail in exe.details if "mm_exact" in detail][-2:]
    assert len(readers) == 2 and sorted("A copied" in detail for detail in readers) == [False, True], exe.details
    q, k, v = (u.view(-1, tokens, heads, 64).transpose(1, 2) for u in linear(c, norm(c, x.double().view(-1, tokens, d), "ln."), "qkv.").split(d, -1))
    merged = torch.nn.functional.scaled_dot_product_attention(q, k, v, is_causal=True).transpose(1, 2).reshape(rows, d)
    want = linear(c, merged, "out.") + linear(c, merged, "gate.")
    assert float((got - want).norm() / want.norm()) <= 3 * BOUND          # (the projection, the attention and these)


@pytest.mark.parametrize("m,d,n", [(1024, 768, 2304), (999, 772, 3004)])
def test_two_linears_on_a_layernorm(m, d, n):
    from perf import cases

    p = cases._Plan("two_readers", (m, d), (m, n))
    h, a = p.buffer(m, d), p.buffer(m, n)
    p.layernorm(p.x, "ln.", h)
    p.linear(h, "up.", n, a)
    p.linear(h, "gate.", n, p.y, residual=a)
    x = torch.randn(m, d, generator=torch.Generator(device="cuda").manual_seed(0), device="cuda")
    exe, c, got = run(p.spec(), x)
    assert sorted("A copied" in detail for detail in exe.details if "mm_exact" in detail) == [False, True], exe.details
    h = norm(c, x.double(), "ln.")
    want = linear(c, h, "up.") + linear(c, h, "gate.")
    assert float((got - want).norm() / want.norm()) <= 2 * BOUND


@pytest.mark.parametrize("m,d,wide", [(1024, 768, 3072), (999, 772, 3004)])
def test_two_linears_on_a_bounded_linear(m, d, wide):
    from perf import cases

    p = cases._Plan("two_readers", (m, d), (m, d))
    h, f, a = p.buffer(m, d), p.buffer(m, wide), p.buffer(m, d)
    p.layernorm(p.x, "ln.", h)
    p.linear(h, "fc.", wide, f, gelu=True)
    p.linear(f, "proj.", d, a)
    p.linear(f, "gate.", d, p.y, residual=a)
    x = torch.randn(m, d, generator=torch.Generator(device="cuda").manual_seed(0), device="cuda")
    exe, c, got = run(p.spec(), x)
    readers = [detail for detail in exe.details if "mm_exact" in detail][-2:]
    assert sorted("A copied" in detail for detail in readers) == [False, True], exe.details
    f = torch.nn.functional.gelu(linear(c, norm(c, x.double(), "ln."), "fc."), approximate="tanh")
    want = linear(c, f, "proj.") + linear(c, f, "gate.")
    assert float((got - want).norm() / want.norm()) <= 3 * BOUND
