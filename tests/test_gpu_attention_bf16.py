"""The fused attention on bf16 operands by itself: every way it spreads its items over the SMs, sequences that end
inside a tile, and scores that outgrow the first tile's maximum many times over."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def attention(batch, tokens, heads, weight=None, bias=None):
    """One matmul that makes Q, K and V of x, and the attention over them -> the executable, its mask."""
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
    consts = {"mask": cases._constants({"mask": (tokens, tokens)}, None)["mask"], "weight.transpose": weight,
              "bias": np.zeros(3 * d, np.float32) if bias is None else bias}
    exe = GPUExecutable(program_from_plan(plan, "bf16"), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    assert "attention_fused" in exe.impls
    return exe, torch.from_numpy(consts["mask"]).cuda().double()


def columns_of_x(d, scale, values=1.0):
    """Q, K (times a power of two) and V as columns of x: the same bf16 numbers here and in the reference."""
    rng = np.random.default_rng(0)
    weight = np.zeros((d, 3 * d), np.float32)
    weight[rng.integers(0, d, 3 * d), np.arange(3 * d)] = np.repeat([scale, scale, values], d)
    return weight


def inputs(batch, tokens, heads):
    return torch.randn(batch * tokens, 64 * heads, generator=torch.Generator(device="cuda").manual_seed(0), device="cuda").bfloat16().float()


def exact(x, weight, mask, batch, tokens, heads):
    q, k, v = (x.double() @ torch.from_numpy(weight).cuda().double()).view(batch, tokens, 3, heads, 64).permute(2, 0, 3, 1, 4)
    for b in range(batch):
        yield torch.stack([torch.softmax(q[b, h] @ k[b, h].T * 0.125 + mask, -1) @ v[b, h] for h in range(heads)])


@pytest.mark.parametrize("scale", [0.5, 4.0])
@pytest.mark.parametrize("batch,tokens,heads", [(2, 2, 2), (2, 127, 2), (3, 129, 2), (6, 333, 12),          # one item per CTA
                                                (2, 1024, 5), (2, 2048, 5),                                # query tiles in halves, alone and in pairs
                                                (8, 1024, 12), (5, 900, 12), (16, 128, 20),                # several items per CTA
                                                (2, 2049, 2), (2, 4097, 2), (2, 2300, 40)])                # longer than a run of 16 key tiles
def test_attention_on_bf16_operands(batch, tokens, heads, scale):
    """What is left beside equal operands is the rounding of the probabilities to bf16 (2^-9 at most, 2^-9 / sqrt(3) = 1.1e-3 in the mean
    square, averaged by the sum over the values; a row of one key has none) and float32 sums: 2e-3."""
    weight = columns_of_x(64 * heads, scale)
    exe, mask = attention(batch, tokens, heads, weight)
    x = inputs(batch, tokens, heads)
    outs = [exe(x)[0] for _ in range(3)]
    exe.status()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    for b, want in enumerate(exact(x, weight, mask, batch, tokens, heads)):
        got = outs[0][b].permute(1, 0, 2).double()
        assert float((got - want).norm() / want.norm()) <= 2e-3
        assert float((got - want).abs().max() / want.abs().max()) <= 4e-3        # (every row: 2^-8)


@pytest.mark.parametrize("split", ["0", "1"])
def test_long_sums_are_not_cut_short(split, monkeypatch):
    """One value for all keys: the result is that value, but for the probabilities' rounding (over 512 rows of 8064 keys and more: 1.1e-3 / sqrt(512 *
    8064) = 6e-7) and for what the tensor core cuts off its sums, at most a unit in the last place (2^-23 to 2^-24 of the sum) per 16 keys, on average
    half of one.  In runs of 2048 keys that is 128 x 2^-24 = 7.6e-6 at most on average; 8192 in one go are 3.1e-5."""
    monkeypatch.setenv("KILN_GPU_ATTENTION_SPLIT", split)
    batch, tokens, heads = 2, 8192, 2
    d = 64 * heads
    value = float(torch.tensor(1 / 3).bfloat16())
    exe, _ = attention(batch, tokens, heads, columns_of_x(d, 0.5, 0.0), np.repeat(np.float32([0, 0, value]), d))
    got = exe(inputs(batch, tokens, heads))[0].double()[:, -128:] / value - 1
    exe.status()
    assert abs(float(got.mean())) <= 7.6e-6


@pytest.mark.parametrize("heads,split", [(12, False), (5, True)])
def test_query_tiles_are_shared_where_sms_are_idle(heads, split, monkeypatch):
    """24 heads of eight query tiles fill the SMs with whole tiles (13.6 us; halves of the long ones on two CTAs an SM 15.0); ten do not."""
    x, weight = inputs(2, 1024, heads), columns_of_x(64 * heads, 0.5)
    got = attention(2, 1024, heads, weight)[0](x)[0]
    monkeypatch.setenv("KILN_GPU_ATTENTION_SPLIT", "0")
    whole = attention(2, 1024, heads, weight)[0](x)[0]
    assert torch.equal(got, whole) != split


@pytest.mark.parametrize("batch,tokens,heads", [(2, 700, 2), (3, 1024, 6), (8, 1024, 12), (2, 2300, 2)])
def test_a_token_without_numbers(batch, tokens, heads):
    """A token that is NaN makes its own rows and all later ones of its sequence NaN, whatever the maxima drop of it; the tiles of 128 queries
    before it do not see it, nor does the next sequence."""
    weight = columns_of_x(64 * heads, 0.5)
    exe, _ = attention(batch, tokens, heads, weight)
    x = inputs(batch, tokens, heads)
    clean = exe(x)[0].clone()
    for at in (0, 130, tokens - 1):
        y = x.clone()
        y[at, 0] = float("nan")                       # (through the zeros of the matmul: all of the token's Q, K and V)
        got = exe(y)[0]
        assert bool(torch.isnan(got[0, at:]).all())
        assert torch.equal(got[0, :at // 128 * 128], clean[0, :at // 128 * 128]) and torch.equal(got[1:], clean[1:])
    exe.status()


@pytest.mark.parametrize("batch,tokens,heads", [(2, 700, 2), (3, 1024, 6), (2, 2300, 2)])
def test_one_token_far_above_the_rest(batch, tokens, heads):
    """A token of 1000s, 2e6 its own score: to each later query it is all or nothing."""
    weight = columns_of_x(64 * heads, 0.5)
    exe, mask = attention(batch, tokens, heads, weight)
    x = inputs(batch, tokens, heads)
    x[150] = 1000.0
    got = exe(x)[0]
    exe.status()
    for b, want in enumerate(exact(x, weight, mask, batch, tokens, heads)):
        want, have = want.permute(1, 0, 2), got[b].double()
        assert float((have - want).norm() / want.norm()) <= 2e-3
        assert float(((have - want).abs() / want.abs().amax(-1, keepdim=True)).max()) <= 8e-3      # (of its row's largest: 2^-8, and 2^-9 of each of the terms that make less of it)
