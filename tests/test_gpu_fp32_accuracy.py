"""FP32 precision on the tensor cores: as near to float64 as float32 sums are, and like them with infinities."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def linear(m, n, k, seed=0, positive=False):
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    plan = cases._plan({"kind": "linear", "m": m, "n": n, "k": k, "precision": "fp32"})
    rng = np.random.default_rng(seed)
    consts = cases._constants(plan.const_shapes, rng)
    x = (rng.standard_normal((m, k)) * k ** -0.5).astype(np.float32)
    if positive:
        consts, x = {name: np.abs(c) for name, c in consts.items()}, np.abs(x)
    build = lambda c: GPUExecutable(program_from_plan(plan, "fp32"), plan.arena_bytes, c, plan.input_shapes, plan.output_shapes)     # noqa: E731
    return build, consts, x


def exact(x, consts):
    return torch.from_numpy(x).cuda().double() @ torch.from_numpy(consts["weight.transpose"]).cuda().double() + torch.from_numpy(consts["bias"]).cuda().double()


@pytest.mark.parametrize("positive", [False, True])
@pytest.mark.parametrize("m,n,k", [(2, 64, 64), (17, 65, 67), (5, 4096, 129), (31, 1000, 100), (17, 768, 300), (2, 768, 768), (333, 1000, 771), (128, 768, 3072),
                                   (100, 3072, 768), (300, 64, 4096), (1000, 1001, 3071), (17, 128, 16384)])
def test_linears_are_as_exact_as_float32_sums(m, n, k, positive):
    """A float32 sum of k products is off by a random walk of k roundings, each of 2^-24 / sqrt(3) of a partial sum: of positive terms,
    whose partial sums grow evenly, 2^-24 sqrt(k) / 3 of the result = 2e-8 sqrt(k); as much again for the bias
    and for the last bits of the operands.  (A tensor core that truncates every accumulation is off by k / 8
    times 3e-8: 1.2e-5 at 3072.)"""
    build, consts, x = linear(m, n, k, positive=positive)
    want = exact(x, consts)
    got = build(consts)(torch.from_numpy(x).cuda())[0].double()
    assert float((got - want).norm() / want.norm()) <= 2e-8 * k ** 0.5 + 6e-8


@pytest.mark.parametrize("m,n,k", [(17, 64, 64), (9, 65, 67), (31, 100, 71), (17, 768, 768), (100, 768, 3072), (300, 64, 1023)])
def test_infinities_and_the_largest_numbers(m, n, k):
    """Where float32 arithmetic has an infinity, a NaN or a finite number, so has the tensor core's split; elsewhere nothing changes."""
    build, consts, x = linear(m, n, k)
    big = np.finfo(np.float32).max
    w = consts["weight.transpose"]
    w[3], w[7] = 1.0, 0.5 * np.sign(w[7])         # (no tails)
    w[5, ::2] = 0.0
    x[0, 3], x[1, 7], x[3, 5], x[4, 1], x[5, 1] = np.inf, -np.inf, np.inf, big, -big
    x[2, [3, 7]] = np.inf
    x[6, 2] = np.nan
    for infinite_weight in (False, True):
        if infinite_weight:
            w[4, 1], x[7, 4] = -np.inf, 0.0
        with np.errstate(invalid="ignore", over="ignore"):
            want = exact(x, consts).float().cpu().numpy()
        got = build(consts)(torch.from_numpy(x).cuda())[0].cpu().numpy()
        assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want)) \
            and np.array_equal(np.isneginf(got), np.isneginf(want))
        finite = np.isfinite(want)
        scale = np.broadcast_to(np.max(np.where(finite, np.abs(want), 0), axis=1, keepdims=True), want.shape)      # of the row
        assert np.all(np.abs(got[finite] - want[finite]) <= 1e-5 * scale[finite])


@pytest.mark.parametrize("tokens,d", [(17, 128), (100, 132)])
def test_infinities_through_every_epilogue(tokens, d):
    """Bias + GELU, and bias + residual, behind sums that are infinite."""
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    p = cases._Plan("mlp", (tokens, d), (tokens, d))
    f = p.buffer(tokens, 4 * d)
    p.linear(p.x, "0.", 4 * d, f, gelu=True)
    p.linear(f, "2.", d, p.y, residual=p.x)
    plan = p.spec()
    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    w = consts["0.weight.transpose"]
    w[3] = np.abs(w[3])
    exe = GPUExecutable(program_from_plan(plan, "fp32"), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    x = torch.randn(tokens, d, device="cuda")
    x[0, 3] = float("inf")
    got = exe(x)[0]
    c = {name: torch.from_numpy(v).cuda().double() for name, v in consts.items()}
    hidden = torch.nn.functional.gelu(x.double() @ c["0.weight.transpose"] + c["0.bias"], approximate="tanh")
    want = hidden @ c["2.weight.transpose"] + c["2.bias"] + x.double()
    assert bool(torch.isinf(hidden[0]).all())
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    assert float((got[1:].double() - want[1:]).norm() / want[1:].norm()) <= 1e-6


@pytest.mark.parametrize("batch,tokens,heads", [(4, 333, 4), (2, 1023, 4), (3, 129, 2), (1, 200, 12), (2, 256, 4)])
def test_attention_of_any_length_is_as_exact_as_float32_sums(batch, tokens, heads):
    """A score is a sum of 64 products scaled by 1/8, its partial sums at most about 1: 64 roundings of 2^-24 / sqrt(3) of half of that in the
    mean square are 2e-7, which is the relative error of an unnormalised weight; the sum over the values
    averages it.  (Truncated sums on the tensor cores: 1.3e-6 to 2.2e-6.)"""
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    d, hd = 64 * heads, 64
    if batch == 1:                                   # the chain of one sequence: scale and mask in the first matmul
        p = cases._Plan("attention", (tokens, 3 * d), (tokens, heads, hd))
        kt, s, w, o = p.buffer(heads, hd, tokens), p.buffer(heads, tokens, tokens), p.buffer(heads, tokens, tokens), p.buffer(heads, tokens, hd)
        p.copy(p.x.as_((heads, hd, tokens), (hd, 1, 3 * d), d), kt)
        p.bmm(p.x.as_((heads, tokens, hd), (hd, 3 * d, 1)), kt, s, 0.125, p.const("mask", tokens, tokens))
        p.softmax(s, w)
        p.bmm(w, p.x.as_((heads, tokens, hd), (hd, 3 * d, 1), 2 * d), o)
        p.copy(o.as_((tokens, heads, hd), (hd, tokens * hd, 1)), p.y)
    else:
        p = cases._Plan("attention", (batch * tokens, 3 * d), (batch, tokens, heads, hd))
        rows = (tokens * 3 * d, hd, 3 * d, 1)
        q, kt, v = p.buffer(batch, heads, tokens, hd), p.buffer(batch, heads, hd, tokens), p.buffer(batch, heads, tokens, hd)
        s, w, o = p.buffer(batch * heads, tokens, tokens), p.buffer(batch, heads, tokens, tokens), p.buffer(batch * heads, tokens, hd)
        p.copy(p.x.as_((batch, heads, tokens, hd), rows), q)
        p.copy(p.x.as_((batch, heads, hd, tokens), (tokens * 3 * d, hd, 1, 3 * d), d), kt)
        p.bmm(q.as_((batch * heads, tokens, hd)), kt.as_((batch * heads, hd, tokens)), s)
        p.softmax(s.as_((batch, heads, tokens, tokens)), w, 0.125, p.const("mask", tokens, tokens))
        p.copy(p.x.as_((batch, heads, tokens, hd), rows, 2 * d), v)
        p.bmm(w.as_((batch * heads, tokens, tokens)), v.as_((batch * heads, tokens, hd)), o)
        p.copy(o.as_((batch, tokens, heads, hd), (heads * tokens * hd, hd, tokens * hd, 1)), p.y)
    plan = p.spec()
    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    exe = GPUExecutable(program_from_plan(plan, "fp32"), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    assert "attention_fused" in exe.impls
    gen = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(plan.input_shapes[0], generator=gen, device="cuda")
    got = exe(x)[0].double().view(batch, tokens, heads, hd)
    q, k, v = x.double().view(batch, tokens, 3, heads, hd).permute(2, 0, 3, 1, 4)
    mask = torch.from_numpy(consts["mask"]).cuda().double()
    want = (torch.softmax(q @ k.transpose(-1, -2) * 0.125 + mask, -1) @ v).permute(0, 2, 1, 3)
    assert float((got - want).norm() / want.norm()) <= 4e-7
