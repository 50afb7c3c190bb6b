"""Exact FP32 on float16 pairs, short K and several rounds of tiles: a tile's sums are ready while the last tile's stores are under way."""

import pytest
import torch
from test_gpu_exact import BOUND, build, call, run_plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chain", ["none", "bias", "gelu", "residual"])
@pytest.mark.parametrize("m,n,k", [(8192, 768, 256), (8192, 1024, 192), (8191, 4092, 132), (16384, 2048, 128)])
def test_float32_results(m, n, k, chain):
    exe, x, c = build(m, n, k, chain)
    assert "mm_exact" in exe.details[0], exe.details
    want = (c["a"] if chain == "residual" else x.double()) @ c["weight.transpose"]
    if chain != "none":
        want = want + c["bias"]
    if chain == "gelu":
        want = torch.nn.functional.gelu(want, approximate="tanh")
    if chain == "residual":
        want = want + x.double()
    error = (call(exe, x).double() - want).norm(dim=1) / want.norm(dim=1)
    assert float(error.max()) <= 2 * BOUND          # (a row by itself)


@pytest.mark.parametrize("stored", ["1", "0"])
@pytest.mark.parametrize("m,d,wide", [(8192, 256, 1024), (8191, 132, 4092)])
def test_pairs_alone_and_beside_float32(m, d, wide, stored):
    """A Linear behind a LayerNorm leaves float16 pairs, and the float32 rows where they are asked for."""
    import numpy as np
    from perf import cases

    p = cases._Plan("mlp", (m, d), (m, d))
    h, f = p.buffer(m, d), p.buffer(m, wide)
    p.layernorm(p.x, "ln.", h)
    p.linear(h, "fc.", wide, f)
    p.linear(f, "proj.", d, p.y)
    plan = p.spec()
    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    x = torch.randn(m, d, generator=torch.Generator(device="cuda").manual_seed(0), device="cuda")
    exe, got = run_plan(plan, consts, x, KILN_GPU_MIRROR_ONLY=stored)
    assert all("mm_exact" in detail and "A copied" not in detail for detail in exe.details[1:]), exe.details
    c = {name: torch.from_numpy(v).cuda().double() for name, v in consts.items()}
    h = torch.nn.functional.layer_norm(x.double(), (d,), c["ln.weight"], c["ln.bias"], 1e-5)
    want = (h @ c["fc.weight.transpose"] + c["fc.bias"]) @ c["proj.weight.transpose"] + c["proj.bias"]
    error = (got.double() - want).norm(dim=1) / want.norm(dim=1)
    assert float(error.max()) <= 4 * BOUND
