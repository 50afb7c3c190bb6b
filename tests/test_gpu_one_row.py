"""One row through a Linear (decoding): both row pitches the kernel reads, K on both sides of what a warp has in flight."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gelu", [False, True])
@pytest.mark.parametrize("n,k", [(4, 1), (32, 31), (36, 33), (3072, 768), (3076, 769), (260, 4099), (64, 20000), (35, 770), (4097, 1537)])
def test_one_row(n, k, gelu):
    """Within a random walk of k roundings of 2^-24 / sqrt(3) of partial sums that grow like sqrt(k): 2e-8 sqrt(k) of the result, and the
    same again for the last bits; an infinity in x stays in its products."""
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    p = cases._Plan("linear", (1, k), (1, n))
    p.linear(p.x, "", n, p.y, gelu=gelu)
    plan = p.spec()
    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    exe = GPUExecutable(program_from_plan(plan, "fp32"), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    assert exe.impls == ["mm_gemv"]
    w, b = (torch.from_numpy(consts[name]).cuda().double() for name in ("weight.transpose", "bias"))
    for seed in range(3):
        x = torch.randn(1, k, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")
        want = x.double() @ w + b
        if gelu:
            want = torch.nn.functional.gelu(want, approximate="tanh")
        got = exe(x)[0].double()
        assert float((got - want).norm() / want.norm()) <= 2e-8 * k ** 0.5 + 2e-7
    x[0, k - 1] = float("inf")
    got, want = exe(x)[0], (x.double() @ w + b)
    assert torch.equal(torch.isinf(want), torch.isinf(got)) or gelu
    assert not bool(torch.isnan(got[torch.isposinf(want)]).any())


@pytest.mark.parametrize("n", [4, 3])
def test_more_rows_than_32_bits_count(n):
    """2^31 + 4096 rows, all of them the same one (stride 0).  Every sum is a whole number of 2^-20, so those of a lane are exact to the 2^24th (n = 4: 2^24 + 32
    rows) or stop growing there (n = 3: 2^26 + 128 rows in a lane): the results are that many rows, short of the lanes' remainders."""
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    k = 2**31 + 4096
    p = cases._Plan("rows", (1, 1), (1, n))
    p.kernel("matmul", [("matmul", [("operand", 0), ("operand", 1)], (1, n))], [p.x.as_((1, k), (0, 0)), p.const("w", 1, n).as_((k, n), (0, 1))], [(0, p.y)])
    plan = p.spec()
    exe = GPUExecutable(program_from_plan(plan, "fp32"), plan.arena_bytes, {"w": np.full((1, n), 2.0**-20, np.float32)}, plan.input_shapes, plan.output_shapes)
    assert exe.impls == ["mm_gemv"]
    got = exe(torch.ones(1, 1, device="cuda"))[0].double()
    want = 32 * (4 * 2.0**24 if n == 4 else 2.0**24) * 2.0**-20
    assert float((got / want - 1).abs().max()) <= 1e-5
