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


@pytest.mark.parametrize("odd", ["a unit switched off", "a unit switched off for good", "a column of zeros"])
def test_units_of_very_different_bounds(odd):
    """One power of two for all of a Linear's results would be that of the largest bound: the others keep their bits."""
    m, d, wide = 1024, 768, 3072
    plan, consts = mlp(m, d, wide)
    if odd == "a column of zeros":
        consts["fc.weight.transpose"][:, 5] = 0
        consts["fc.bias"][5] = 0
    else:
        consts["fc.bias"][5] = -1e20 if odd.endswith("good") else -1e9
    x = torch.randn(m, d, generator=torch.Generator(device="cuda").manual_seed(0), device="cuda")
    exe, got = run_plan(plan, consts, x)
    assert float(errors(got, mlp_reference(consts, x), 1).max()) <= 4 * BOUND
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
