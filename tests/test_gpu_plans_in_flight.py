"""Modules that share the GPU with others: what they are told, and that it changes none of their results."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def build(p, precision, seed=0):
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    plan = p.spec()
    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    exe = GPUExecutable(program_from_plan(plan, precision), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes, cuda_graphs=False)
    return exe, torch.randn(plan.input_shapes[0], generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")


def linear(m, n, k):
    from perf import cases

    p = cases._Plan("linear", (m, k), (m, n))
    p.linear(p.x, "", n, p.y)
    return p


def test_a_module_is_alone_again_after_a_step():
    """96 tiles of 256 columns are two rounds on 74 SM pairs: that width is for modules that fill each other's rounds, and goes with them."""
    from kiln_b200.runtime import StreamedBatch

    made = [build(linear(8192, 768, 3072), "bf16", seed) for seed in (0, 1)]
    modules, xs = [e for e, _ in made], [x for _, x in made]
    alone = list(modules[0].details)
    assert "256 columns" not in alone[0], alone
    want = [e(x)[0] for e, x in made]
    outs = [torch.empty_like(w) for w in want]
    step = StreamedBatch(modules, concurrency=1).capture(xs, outs)
    assert all("256 columns" in e.details[0] for e in modules), [e.details for e in modules]
    step.run()
    assert all(torch.equal(a, b) for a, b in zip(outs, want))
    StreamedBatch(modules, concurrency=1).capture(xs, outs)            # (bound as they are: the first step's graph is still good)
    outs[0].zero_()
    step.run()
    assert all(torch.equal(a, b) for a, b in zip(outs, want))
    step.capture(xs[:1], outs[:1])                                     # one request has nobody beside it
    assert modules[0].details == alone
    step.capture(xs, outs)
    modules[0].set_concurrency(1)
    assert modules[0].details == alone
    assert torch.equal(modules[0](xs[0])[0], want[0])


def order_of_sums(detail):
    """The kernel and its K splits, of a detail string."""
    words = detail.replace(",", "").split()
    return words[0], words[words.index("splits") - 1] if "splits" in words else "1"


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("m,n,k", [(2048, 768, 3072), (600, 2048, 2048), (1793, 708, 4100),          # K in halves
                                   (9472, 160, 1024), (556, 3136, 128),                            # between two kernels
                                   (1024, 3072, 768), (700, 4096, 4096), (1000, 1000, 772)])
def test_the_order_of_sums_is_the_shape_s(m, n, k, precision):
    exe, x = build(linear(m, n, k), precision)
    want, alone = exe(x)[0], exe.details[0]
    for plans, others in ((1, True), (2, False), (4, False), (8, False), (8, True)):
        exe.set_concurrency(plans, others)
        assert order_of_sums(exe.details[0]) == order_of_sums(alone), (plans, others, exe.details, alone)
        assert torch.equal(exe(x)[0], want), (plans, others)


@pytest.mark.parametrize("concurrency", [None, 1])
def test_a_step_gives_the_bits_of_a_call(concurrency):
    """An MLP of 2048 tokens, whose second matmul takes K in halves."""
    from kiln_b200.runtime import StreamedBatch
    from perf import cases

    def mlp():
        p = cases._Plan("mlp", (2048, 768), (2048, 768))
        f = p.buffer(2048, 3072)
        p.linear(p.x, "0.", 3072, f, gelu=True)
        p.linear(f, "2.", 768, p.y)
        return p

    made = [build(mlp(), "tf32", seed) for seed in range(3)]
    assert "2 splits" in made[0][0].details[1]
    want = [e(x)[0] for e, x in made]
    outs = [torch.empty_like(w) for w in want]
    StreamedBatch([e for e, _ in made], concurrency=concurrency).capture([x for _, x in made], outs).run()
    assert all(torch.equal(a, b) for a, b in zip(outs, want))
