"""What the plans do where memory is short: weights that are not copied, and the bounds on those that are."""

import numpy as np
import pytest
import torch

from test_gpu_sizes import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "tf32", "bf16"])
@pytest.mark.parametrize("m", [1, 17, 128, 364])
@pytest.mark.parametrize("n,k", [(768, 768), (1000, 771), (3072, 96)])
def test_linear_without_copies_of_its_weight(m, n, k, precision, monkeypatch):
    """N a multiple of 32 (the weight is describable as it is) and not (it is copied to aligned rows)."""
    monkeypatch.setenv("KILN_GPU_WEIGHT_COPIES", "0")
    check({"kind": "linear", "m": m, "n": n, "k": k, "precision": precision}, calls=2)


@pytest.mark.parametrize("precision", ["fp32", "tf32"])
def test_all_copies_of_a_plan_share_a_quarter_of_the_free_memory(precision):
    """Eight Linears of 2048 x 2048 with 0.5 GB to spare: 32 MB a copy of a weight (and in FP32 as much for its tails), of which a quarter of
    what is left holds some; each Linear on its own would get a quarter of what the ones before it left."""
    from kiln_b200 import _cabi
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    layers, d, rows = 8, 2048, 256
    p = cases._Plan("stack", (rows, d), (rows, d))
    x = p.x
    for i in range(layers):
        y = p.y if i + 1 == layers else p.buffer(rows, d)
        p.linear(x, f"{i}.", d, y)
        x = y
    plan = p.spec()
    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    exe = GPUExecutable(program_from_plan(plan, precision), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    x = torch.randn(rows, d, device="cuda")
    (want,) = exe(x)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    _cabi.check(exe._lib.kb200_plan_set_option(exe._plan, _cabi.OPT_WEIGHT_COPIES, 0))
    exe._bind()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (512 << 20), dtype=torch.uint8, device="cuda")
    try:
        _cabi.check(exe._lib.kb200_plan_set_option(exe._plan, _cabi.OPT_WEIGHT_COPIES, 1))
        free = torch.cuda.mem_get_info()[0]
        exe._bind()
        taken = free - torch.cuda.mem_get_info()[0]
        (got,) = exe(x)
        torch.cuda.synchronize()
        exe.status()
    finally:
        del hold
        torch.cuda.empty_cache()
    assert free < 600 << 20
    assert 0 < taken <= free // 4 + (16 << 20)             # (allocations are rounded up to 2 MB)
    error = float((got - want).norm() / want.norm())
    assert error <= {"fp32": 1e-5, "tf32": 2e-3}[precision]      # the bounds of the precisions, as in the other tests
