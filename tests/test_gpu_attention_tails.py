"""FP32 attention on the tensor cores: the tails of Q, K and V come from the projection that writes them, or, where the kernel is
asked for by option, from a pass of their own."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("odd", ["", "infinite V", "infinite Q and K", "a NaN", "large"])
def test_tails_of_the_projection_are_those_of_the_pass(odd, monkeypatch):
    """The same bits, a launch less; also where an element has no tail (infinity minus infinity) and where the projection does a result over."""
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    plan = cases._plan({"kind": "block", "tokens": 1024, "heads": 12})
    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    x = torch.randn(plan.input_shapes[0], generator=torch.Generator(device="cuda").manual_seed(0), device="cuda")
    d = 768
    bias, weight = consts["c_attn.bias"], consts["c_attn.weight.transpose"]
    if odd == "infinite V":
        bias[2 * d + 5], bias[2 * d + 70] = np.inf, -np.inf
    elif odd == "infinite Q and K":
        weight[3, [1, d + 130]] = np.inf
    elif odd == "a NaN":
        x[700, 3] = float("nan")
    elif odd == "large":
        weight[:, 2 * d:] *= np.float32(1e30)
    outs, launches = [], []
    for choice in ("", "tensor"):
        monkeypatch.setenv("KILN_GPU_FP32_ATTENTION", choice)
        exe = GPUExecutable(program_from_plan(plan, "fp32"), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
        outs.append(exe(x)[0].clone())
        launches.append(exe.device_launches)
        exe.status()
    assert launches[1] == launches[0] + 1 and "attention_fused" in exe.impls
    assert torch.equal(torch.isnan(outs[0]), torch.isnan(outs[1]))
    assert torch.equal(torch.nan_to_num(outs[0], nan=0.0), torch.nan_to_num(outs[1], nan=0.0))
    if odd == "":
        assert not bool(torch.isnan(outs[0]).any())
