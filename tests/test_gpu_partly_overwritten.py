"""Intermediates that a later kernel overwrites in part: what is left of them still holds its values."""

import numpy as np
import pytest
import torch

from oracle.plan_oracle import scale_relative_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("columns", [128, 256])
def test_a_write_with_gaps_leaves_the_rest_of_a_bf16_intermediate(columns):
    """In BF16 mode a projection read by a matmul alone is kept as bf16 only; one of whose columns some are overwritten and
    others read as float32 is not.  (All columns: every value is overwritten and the float32 store may go.)"""
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from kiln_b200.spec import KernelSpec, NodeSpec, OperandSpec, PlanSpec

    n, rows = 256, 256
    whole = OperandSpec(("arena",), 0, (rows, n), (n, 1))
    part = OperandSpec(("arena",), 0, (rows, columns), (n, 1))
    tail = OperandSpec(("arena",), n - 64, (128, 64), (n, 1))
    at = lambda base, *shape: OperandSpec(base, 0, shape, (shape[1], 1))     # noqa: E731

    def matmul(name, a, weight, out):
        return KernelSpec(name, "matmul", [NodeSpec("matmul", [("operand", 0), ("operand", 1)], (rows, n), {})], [a, at(("const", weight), n, n)], [(0, out)])

    kernels = [matmul("k0", at(("input", 0), rows, n), "w0", whole),
               matmul("k1", whole, "w1", at(("output", 0), rows, n)),
               KernelSpec("k2", "elementwise", [NodeSpec("neg", [("operand", 0)], (rows, columns), {})],
                          [OperandSpec(("input", 0), 0, (rows, columns), (n, 1))], [(0, part)]),
               KernelSpec("k3", "elementwise", [NodeSpec("neg", [("operand", 0)], (128, 64), {})], [tail], [(0, at(("output", 1), 128, 64))])]
    plan = PlanSpec("partly_overwritten", [(rows, n)], [(rows, n), (128, 64)], rows * n * 4, {"w0": (n, n), "w1": (n, n)}, kernels)
    rng = np.random.default_rng(0)
    consts = {w: (rng.standard_normal((n, n)) / 16).astype(np.float32) for w in ("w0", "w1")}
    exe = GPUExecutable(program_from_plan(plan, "bf16"), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    exe.arena.zero_()
    x = rng.standard_normal((rows, n)).astype(np.float32)
    product, rest = exe(torch.from_numpy(x).cuda())
    torch.cuda.synchronize()
    exe.status()
    f = x.astype(np.float64) @ consts["w0"]
    assert scale_relative_error(product.cpu().numpy(), f @ consts["w1"]) <= 2e-2
    want = -(f if columns < n else -x)[:128, n - 64:]
    assert scale_relative_error(rest.cpu().numpy(), want) <= 2e-2
