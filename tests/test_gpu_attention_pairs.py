"""FP32 attention on float16 pairs: any length, one or several sequences, shared query tiles, planes from the projection or from a pass, into
the out-projection or as float32, rows of NaN, and blocks whose bounds say nothing."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# What a block adds to its input, 2-norm: seven float32 kernels, the largest error the GELU's (2^-22 in its exponential and reciprocal)
BOUND = 6e-7


def block(tokens, heads, batch=None, change=None, **env):
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    c = {"kind": "batched_block" if batch else "block", "tokens": tokens, "heads": heads, "batch": batch, "precision": "fp32"}
    plan = cases._plan(c)
    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    x = torch.randn(plan.input_shapes[0], generator=torch.Generator(device="cuda").manual_seed(0), device="cuda")
    if change:
        change(consts, x)
    with pytest.MonkeyPatch.context() as patch:
        for name, value in env.items():
            patch.setenv(name, value)
        exe = GPUExecutable(program_from_plan(plan, "fp32"), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    outs = [exe(x)[0] for _ in range(3)]
    exe.status()
    assert torch.equal(outs[0].nan_to_num(), outs[1].nan_to_num()) and torch.equal(outs[0].nan_to_num(), outs[2].nan_to_num())
    return exe, consts, x, outs[0]


def reference(consts, x, heads):
    c = {name: torch.from_numpy(v).cuda().double() for name, v in consts.items()}
    shape, d = x.shape, 64 * heads
    x = x.double().view(-1, shape[-2], d)

    def norm(v, p):
        return torch.nn.functional.layer_norm(v, (d,), c[p + "weight"], c[p + "bias"], 1e-5)

    def linear(v, p):
        return v @ c[p + "weight.transpose"] + c[p + "bias"]

    q, k, v = (u.view(*u.shape[:2], heads, 64).transpose(1, 2) for u in linear(norm(x, "ln1."), "c_attn.").split(d, -1))
    a = torch.nn.functional.scaled_dot_product_attention(q, k, v, is_causal=True).transpose(1, 2).reshape(x.shape)
    y = x + linear(a, "c_proj.")
    y = y + linear(torch.nn.functional.gelu(linear(norm(y, "ln2."), "fc."), approximate="tanh"), "proj.")
    return (y - x).view(shape), y.view(shape)


@pytest.mark.parametrize("tokens,heads,batch", [(129, 12, None), (200, 12, None), (333, 4, None), (1024, 12, None), (1023, 12, None), (1500, 4, None),
                                                (2047, 16, None), (333, 12, 6), (257, 8, 3), (1024, 12, 2), (100, 12, 8)])
def test_blocks_of_any_length(tokens, heads, batch):
    exe, consts, x, got = block(tokens, heads, batch)
    added, want = reference(consts, x, heads)
    assert float((got.double() - want).norm() / added.norm()) <= (2 * BOUND if "mm_small" in "".join(exe.details) else BOUND)


@pytest.mark.parametrize("tokens,batch", [(1024, None), (777, None), (333, 6)])
def test_the_same_bits_wherever_the_pairs_are_made(tokens, batch):
    """By the projection's epilogue or by a pass; with the float32 rows stored beside them or not."""
    exe, _, _, got = block(tokens, 12, batch)
    passed, _, _, by_pass = block(tokens, 12, batch, KILN_GPU_FP32_ATTENTION="tensor")
    _, _, _, stored = block(tokens, 12, batch, KILN_GPU_MIRROR_ONLY="0")
    assert exe.device_launches == 7 and passed.device_launches == 8
    assert torch.equal(got, by_pass) and torch.equal(got, stored)


def test_a_row_of_nan():
    """Its sequence from there on is NaN (and in front of it, as far as its tile of keys is masked by a probability of 0), the other sequences are not."""
    def change(consts, x):
        x[2, 100, 5] = float("nan")

    _, consts, x, got = block(333, 12, 6, change)
    assert bool(got[2, 100:].isnan().all())
    added, want = reference(consts, x, 12)
    rest = [0, 1, 3, 4, 5]
    assert float((got.double() - want)[rest].norm() / added[rest].norm()) <= BOUND


@pytest.mark.parametrize("odd", ["heads apart", "columns apart", "infinite gain"])
def test_heads_and_columns_of_very_different_magnitudes(odd):
    """A power of two per head of Q, K and V holds heads that are 2^40 apart; columns of one head that are keep the other kernels."""
    def change(consts, x):
        w = consts["c_attn.weight.transpose"]
        if odd == "heads apart":
            w[:, 64:128] *= np.float32(2.0**-20)
            w[:, 2 * 768:2 * 768 + 64] *= np.float32(2.0**10)
        elif odd == "columns apart":
            w[:, 3] *= np.float32(2.0**20)
            w[:, 768 + 3] *= np.float32(2.0**-20)
        else:
            consts["ln1.weight"][7] = np.inf

    exe, consts, x, got = block(1024, 12, None, change)
    if odd == "infinite gain":
        assert bool(got.isnan().any())
        return
    added, want = reference(consts, x, 12)
    assert float((got.double() - want).norm() / added.norm()) <= 1e-5          # (the bound of this precision: "columns apart" keeps kernels whose
    #                                                    sums lose up to 2^-24 with each of 64 MMAs, 3.8e-6, in each of two matmuls and the attention between)
