"""Exact FP32 on float16 pairs: values far apart.  Errors by row and by column, each against its own size, so that nothing hides behind
what is large."""

import numpy as np
import pytest
import torch
from test_gpu_exact import BOUND, build, call, run_plan

pytestmark = pytest.mark.gpu


def mlp(m, d, wide, gelu=True):
    from perf import cases

    p = cases._Plan("mlp", (m, d), (m, d))
    h, f = p.buffer(m, d), p.buffer(m, wide)
    p.layernorm(p.x, "ln.", h)
    p.linear(h, "fc.", wide, f, gelu=gelu)
    p.linear(f, "proj.", d, p.y)
    plan = p.spec()
    return plan, cases._constants(plan.const_shapes, np.random.default_rng(0))


def mlp_reference(consts, x, gelu=True):
    c = {name: torch.from_numpy(v).cuda().double() for name, v in consts.items()}
    h = torch.nn.functional.layer_norm(x.double(), x.shape[-1:], c["ln.weight"], c["ln.bias"], 1e-5)
    f = h @ c["fc.weight.transpose"] + c["fc.bias"]
    f = torch.nn.functional.gelu(f, approximate="tanh") if gelu else f
    return f @ c["proj.weight.transpose"] + c["proj.bias"]


def errors(got, want, dim):
    return (got.double() - want).norm(dim=dim) / want.norm(dim=dim)


@pytest.mark.parametrize("odd", ["a unit switched off", "a unit switched off for good", "a column of zeros", "a column far above"])
def test_units_of_very_different_bounds(odd):
    """One power of two for all of a Linear's results would be that of the largest bound: the others keep their bits."""
    m, d, wide = 1024, 768, 3072
    plan, consts = mlp(m, d, wide)
    if odd == "a column of zeros":
        consts["fc.weight.transpose"][:, 5] = 0
        consts["fc.bias"][5] = 0
    elif odd == "a column far above":
        consts["fc.weight.transpose"][:, 5] *= np.float32(2.0**20)
        consts["proj.weight.transpose"][5, ::2] = 0          # half of the results do not use it
    else:
        consts["fc.bias"][5] = -1e20 if odd.endswith("good") else -1e9
    x = torch.randn(m, d, generator=torch.Generator(device="cuda").manual_seed(0), device="cuda")
    exe, got = run_plan(plan, consts, x)
    looked_at = slice(None, None, 2 if odd == "a column far above" else 1)
    assert float(errors(got[:, looked_at], mlp_reference(consts, x)[:, looked_at], 1).max()) <= 4 * BOUND
    assert all("mm_exact" in detail for detail in exe.details[1:]), exe.details
    assert ("A copied" in exe.details[2]) == (odd != "a column of zeros"), exe.details


@pytest.mark.parametrize("power", [16, 20, 24])
def test_a_feature_far_above_the_others(power):
    """Half of the results do not use it: they are sums of the small features alone."""
    m, n, k = 1024, 768, 1536
    unused = np.ones((k, n), np.float32)
    unused[7, ::2] = 0
    exe, x, c = build(m, n, k, "none", scale=unused)
    x[:, 7] = torch.exp2(torch.tensor(float(power))) * (1 + torch.rand(m, device="cuda"))
    got = call(exe, x)
    assert float(errors(got, x.double() @ c["weight.transpose"], 0).max()) <= BOUND
    assert "mm_exact" in exe.details[0], exe.details


def groups(m, n, k, powers):
    """Features in groups that are powers of two apart, the weight block-diagonal: a column uses one group."""
    of_k, of_n = np.arange(k) * len(powers) // k, np.arange(n) % len(powers)
    used = (of_k[:, None] == of_n[None, :]).astype(np.float32)
    return used, torch.exp2(torch.tensor([float(powers[g]) for g in of_k], device="cuda"))


# (down to 2^-56 and 2^-84 of the largest; a row's exponents reach below 2^-100 in the last)
@pytest.mark.parametrize("powers", [(0, 30), (0, 40), (60, 0), (0, 27, 55, 83), (-60, -100, -30)])
@pytest.mark.parametrize("m,n,k,form", [(1024, 768, 1536, "columns"), (999, 772, 2052, "2 splits"), (512, 768, 3072, "4 splits"), (3001, 3004, 516, "256 columns")])
@pytest.mark.parametrize("rows", ["all", "some"])
def test_features_in_groups_far_apart(m, n, k, form, powers, rows):
    """Elements far below their row's largest keep their bits, in tiles of such rows alone and in tiles of both kinds; the others the same bits as ever."""
    used, size = groups(m, n, k, powers)
    exe, x, c = build(m, n, k, "none", scale=used)
    assert "mm_exact" in exe.details[0] and form in exe.details[0], exe.details
    plain = call(exe, x)
    wide = torch.ones(m, dtype=torch.bool, device="cuda")
    if rows == "some":
        wide = torch.rand(m, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda") < 0.01
    x = torch.where(wide[:, None], x * size, x)
    got = call(exe, x)
    want = x.double() @ c["weight.transpose"]
    assert float(errors(got[wide], want[wide], 0).max()) <= (BOUND if rows == "all" else 2 * BOUND)          # (some: a few numbers to a column)
    assert torch.equal(got[~wide], plain[~wide])


@pytest.mark.parametrize("m,n,d", [(1024, 2304, 768), (999, 3004, 772), (1024, 1024, 4096), (512, 1024, 8196)])
def test_gains_far_apart(m, n, d):
    """The rows that a LayerNorm splits, a warp or a block to a row."""
    from perf import cases
    from test_gpu_exact import norm_linear

    used, size = groups(m, n, d, (0, 30, 60))
    plan = norm_linear(d, n, m)
    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    for name in ("ln.weight", "ln.bias"):
        consts[name] *= size.cpu().numpy()
    consts["fc.weight.transpose"] *= used
    consts["fc.bias"][:] = 0
    x = torch.randn(m, d, generator=torch.Generator(device="cuda").manual_seed(0), device="cuda")
    exe, got = run_plan(plan, consts, x)
    assert "mm_exact" in exe.details[1] and "A copied" not in exe.details[1], exe.details
    c = {name: torch.from_numpy(v).cuda().double() for name, v in consts.items()}
    h = torch.nn.functional.layer_norm(x.double(), (d,), c["ln.weight"], c["ln.bias"], 1e-5)
    assert float(errors(got, h @ c["fc.weight.transpose"], 0).max()) <= 2 * BOUND          # (the LayerNorm's own float32 sums)


def test_weights_with_elements_far_below_their_column_s_largest():
    """A weight has one power of two to a column: the kernels on TF32, which have float32's exponents, take it."""
    m, n, k = 1024, 768, 1536
    scale = np.ones((k, n), np.float32)
    scale[:k // 2, ::2] = scale[k // 2:, 1::2] = np.float32(2.0**-40)
    exe, x, c = build(m, n, k, "none", scale=scale)
    assert "mm_exact" not in exe.details[0], exe.details
    x[:, :k // 2] *= 2.0**40
    got = call(exe, x)
    assert float(errors(got, x.double() @ c["weight.transpose"], 0).max()) <= 5e-6          # (the other kernels': 2^-23 per 8 of K in one accumulator)


@pytest.mark.parametrize("gelu", [True, False])
def test_rows_of_next_to_nothing_without_biases(gelu):
    """A LayerNorm makes little of rows far below its epsilon, and a Linear without a bias nothing more: far below any bound."""
    m, d, wide = 1024, 768, 3072
    plan, consts = mlp(m, d, wide, gelu)
    for name in ("ln.bias", "fc.bias", "proj.bias"):
        consts[name][:] = 0
    x = torch.randn(m, d, generator=torch.Generator(device="cuda").manual_seed(0), device="cuda")
    x *= torch.exp2(-torch.linspace(0, 60, m, device="cuda"))[:, None]
    exe, got = run_plan(plan, consts, x)
    assert all("mm_exact" in detail for detail in exe.details[1:]) and "A copied" in exe.details[2], exe.details
    assert float(errors(got, mlp_reference(consts, x, gelu), 1).max()) <= 4 * BOUND + (4e-7 if gelu else 0)
