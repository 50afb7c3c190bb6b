"""Exact FP32 on float16 pairs with several plans in flight: smaller grids, and modules side by side in one step, give the bits of a call."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def build(case, seed):
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    plan = cases._plan({"precision": "fp32", **case})
    consts = cases._constants(plan.const_shapes, np.random.default_rng(seed))
    exe = GPUExecutable(program_from_plan(plan, "fp32"), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes, cuda_graphs=False)
    x = torch.randn(plan.input_shapes[0], generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")
    x[..., 5, 7] = 2.0**40                               # a row of two levels
    return exe, x


# (sequences of fewer than eight query tiles: longer ones share tiles between CTAs where a module is alone)
@pytest.mark.parametrize("case", [{"kind": "linear", "m": 2048, "n": 3072, "k": 768}, {"kind": "linear", "m": 1024, "n": 768, "k": 3072},
                                  {"kind": "mlp", "tokens": 1500, "d": 768}, {"kind": "batched_block", "batch": 2, "tokens": 500, "heads": 12}])
def test_a_share_of_the_gpu(case):
    exe, x = build(case, 0)
    want = exe(x)[0].clone()
    assert "mm_exact" in "".join(exe.details), exe.details
    for plans, others in ((1, True), (2, False), (4, False), (8, False), (8, True), (1, False)):
        exe.set_concurrency(plans, others)
        assert "mm_exact" in "".join(exe.details), (plans, others, exe.details)
        assert torch.equal(exe(x)[0], want), (plans, others)
    exe.status()


@pytest.mark.parametrize("case", [{"kind": "mlp", "tokens": 1000, "d": 768}, {"kind": "block", "tokens": 333, "heads": 12}])
@pytest.mark.parametrize("concurrency", [None, 1, 4])
def test_modules_side_by_side(case, concurrency):
    from kiln_b200.runtime import StreamedBatch

    made = [build(case, seed) for seed in range(4)]
    modules, xs = [e for e, _ in made], [x for _, x in made]
    want = [e(x)[0].clone() for e, x in made]
    outs = [torch.empty_like(w) for w in want]
    step = StreamedBatch(modules, concurrency=concurrency).capture(xs, outs)
    for _ in range(3):
        for out in outs:
            out.zero_()
        step.run()
        assert all(torch.equal(a, b) for a, b in zip(outs, want))
    for e in modules:
        e.status()
