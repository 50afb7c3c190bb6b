"""LayerNorm whose scale and shift are no constants: outputs of the launch in front of it, or the caller's tensors."""

import numpy as np
import pytest
import torch

from oracle.plan_oracle import run_plan, scale_relative_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,d", [(3, 64), (200, 768), (20000, 512), (5, 771), (700, 9), (64, 4096)])
def test_affine_parameters_written_by_an_earlier_launch(rows, d):
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    p = cases._Plan("computed_affine", (rows, d), (rows, d))
    made = {}
    for name in ("weight", "bias"):
        constant, made[name] = p.const(name, d), p.buffer(d)
        p.kernel("elementwise", [("neg", [("operand", 0)], (d,))], [constant], [(0, made[name])])
    p.const = lambda name, *shape: made[name]
    p.layernorm(p.x, "", p.y)
    plan = p.spec()
    rng = np.random.default_rng(0)
    for call in range(3):
        consts = {name: rng.standard_normal(d).astype(np.float32) for name in made}
        exe = GPUExecutable(program_from_plan(plan, "fp32"), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
        exe.arena.fill_(call)
        x = rng.standard_normal((rows, d)).astype(np.float32)
        (got,) = exe(torch.from_numpy(x).cuda())
        torch.cuda.synchronize()
        exe.status()
        assert exe.impls[-1] == "row_layernorm"
        (want,) = run_plan(plan.to_json(), [x], consts, dtype=np.float64)
        assert scale_relative_error(got.cpu().numpy(), want) <= 1e-5


@pytest.mark.parametrize("rows,d", [(3, 64), (700, 771)])
def test_affine_parameters_of_the_caller(rows, d):
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    p = cases._Plan("affine_inputs", (rows, d), (rows, d))
    p.const = lambda name, *shape: cases._View(("input", 1 if name == "weight" else 2), shape)
    p.layernorm(p.x, "", p.y)
    plan = p.spec()
    plan.input_shapes = [(rows, d), (d,), (d,)]
    exe = GPUExecutable(program_from_plan(plan, "fp32"), plan.arena_bytes, {}, plan.input_shapes, plan.output_shapes)
    x = torch.randn(rows, d, device="cuda")
    for _ in range(3):
        scale, shift = torch.randn(d, device="cuda"), torch.randn(d, device="cuda")
        (got,) = exe(x, scale * 2, shift - 1)
        want = torch.nn.functional.layer_norm(x.double(), (d,), scale.double() * 2, shift.double() - 1, 1e-5)
        assert scale_relative_error(got.cpu().numpy(), want.cpu().numpy()) <= 1e-5
