"""The fused attention on bf16 operands by itself: every way it spreads its items over the SMs, sequences that end
inside a tile, and scores that outgrow the first tile's maximum many times over."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0.5, 4.0])
@pytest.mark.parametrize("batch,tokens,heads", [(2, 2, 2), (2, 127, 2), (3, 129, 2), (6, 333, 12),          # one item per CTA
                                                (2, 1024, 5), (2, 2048, 5),                                # query tiles in halves, alone and in pairs
                                                (8, 1024, 12), (5, 900, 12), (16, 128, 20)])               # several items per CTA
def test_attention_on_bf16_operands(batch, tokens, heads, scale):
    """Q, K and V are columns of x times a power of two, so they are the same bf16 numbers here and there.  What is left is
    the rounding of the probabilities to bf16 (2^-9 at most, 2^-9 / sqrt(3) = 1.1e-3 in the mean square, averaged by the sum over
    the values; a row of one key has none) and float32 sums: 2e-3."""
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    d, hd = 64 * heads, 64
    rows = (tokens * 3 * d, hd, 3 * d, 1)
    p = cases._Plan("attention", (batch * tokens, d), (batch, tokens, heads, hd))
    qkv = p.buffer(batch * tokens, 3 * d)
    p.linear(p.x, "", 3 * d, qkv)
    q, kt, v = p.buffer(batch, heads, tokens, hd), p.buffer(batch, heads, hd, tokens), p.buffer(batch, heads, tokens, hd)
    s, w, o = p.buffer(batch * heads, tokens, tokens), p.buffer(batch, heads, tokens, tokens), p.buffer(batch * heads, tokens, hd)
    p.copy(qkv.as_((batch, heads, tokens, hd), rows), q)
    p.copy(qkv.as_((batch, heads, hd, tokens), (tokens * 3 * d, hd, 1, 3 * d), d), kt)
    p.bmm(q.as_((batch * heads, tokens, hd)), kt.as_((batch * heads, hd, tokens)), s)
    p.softmax(s.as_((batch, heads, tokens, tokens)), w, 0.125, p.const("mask", tokens, tokens))
    p.copy(qkv.as_((batch, heads, tokens, hd), rows, 2 * d), v)
    p.bmm(w.as_((batch * heads, tokens, tokens)), v.as_((batch * heads, tokens, hd)), o)
    p.copy(o.as_((batch, tokens, heads, hd), (heads * tokens * hd, hd, tokens * hd, 1)), p.y)
    plan = p.spec()
    rng = np.random.default_rng(0)
    consts = cases._constants(plan.const_shapes, rng)
    weight = np.zeros((d, 3 * d), np.float32)
    weight[rng.integers(0, d, 3 * d), np.arange(3 * d)] = np.repeat([scale, scale, 1.0], d)
    consts["weight.transpose"], consts["bias"] = weight, np.zeros(3 * d, np.float32)
    exe = GPUExecutable(program_from_plan(plan, "bf16"), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    assert "attention_fused" in exe.impls
    gen = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(batch * tokens, d, generator=gen, device="cuda").bfloat16().float()
    outs = [exe(x)[0] for _ in range(3)]
    exe.status()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    mask = torch.from_numpy(consts["mask"]).cuda().double()
    qkv = (x.double() @ torch.from_numpy(weight).cuda().double()).view(batch, tokens, 3, heads, hd).permute(2, 0, 3, 1, 4)
    for b in range(batch):
        want = torch.softmax(qkv[0, b] @ qkv[1, b].transpose(-1, -2) * 0.125 + mask, -1) @ qkv[2, b]
        got = outs[0][b].permute(1, 0, 2).double()
        assert float((got - want).norm() / want.norm()) <= 2e-3
        assert float((got - want).abs().max() / want.abs().max()) <= 4e-3        # (every row: 2^-8)
