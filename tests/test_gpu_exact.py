"""Exact FP32 on float16 pairs: every tile width and K in halves, ragged rows, columns and K, all four chains, rows of any magnitude,
infinities and NaN, and weights that keep the other kernels."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# Relative to the 2-norm, positive operands (every error of a sum along one sign): 2^-24 for what the terms leave of either operand and for
# the product of two tails, half of 2^-23 cut off eight times while 64 of K are summed, of what is there by then half in the mean: 2^-21
# in all, and the rounded sums over K as float32's.
BOUND = 6e-7


def build(m, n, k, chain="bias", seed=0, positive=False, scale=None, tokens=None):
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    p = cases._Plan("linear", (m, n if chain == "residual" else k), (m, n))
    x = p.x
    if chain == "residual":                         # the product of a constant and a weight, and the input added
        x = p.const("a", m, k)
    p.linear(x, "", n, p.y, gelu=chain == "gelu", residual=p.x if chain == "residual" else None)
    if chain == "none":
        kind, nodes, inputs, _ = p.kernels[0]
        p.kernels[0] = (kind, nodes[:1], inputs[:2], [(0, p.y)])
        p.consts.pop("bias")
    plan = p.spec()
    rng = np.random.default_rng(seed)
    consts = {name: rng.standard_normal(shape, dtype=np.float32) for name, shape in plan.const_shapes.items()}
    consts["weight.transpose"] *= np.float32(k ** -0.5)
    if positive:
        consts = {name: np.abs(c) for name, c in consts.items()}
    if scale is not None:
        consts["weight.transpose"] *= scale
    exe = GPUExecutable(program_from_plan(plan, "fp32"), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    x = torch.randn(plan.input_shapes[0], generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")
    return exe, x.abs() if positive else x, {name: torch.from_numpy(c).cuda().double() for name, c in consts.items()}


def call(exe, x):
    outs = [exe(x)[0] for _ in range(3)]
    exe.status()
    assert torch.equal(outs[0].nan_to_num(), outs[1].nan_to_num()) and torch.equal(outs[0].nan_to_num(), outs[2].nan_to_num())
    return outs[0]


@pytest.mark.parametrize("m,n,k,form", [(1024, 2304, 768, "128 columns"), (1000, 2300, 772, "128 columns"), (2048, 4092, 1028, "160 columns"),
                                        (700, 4096, 1024, "192 columns"), (2000, 3068, 772, "192 columns"), (513, 4096, 4096, "192 columns"),
                                        (3000, 3072, 768, "256 columns"), (3001, 3004, 516, "256 columns"),
                                        (1024, 768, 3072, "128 columns, 2 splits"), (999, 772, 2052, "128 columns, 2 splits"),
                                        (1024, 512, 2048, "128 columns, 3 splits"), (999, 508, 2052, "128 columns, 3 splits"),
                                        (512, 768, 3072, "128 columns, 4 splits"), (300, 644, 3084, "128 columns, 4 splits")])
def test_widths(m, n, k, form):
    exe, x, c = build(m, n, k, positive=True)
    assert f"mm_exact {form}" in exe.details[0], exe.details
    want = x.double() @ c["weight.transpose"] + c["bias"]
    got = call(exe, x).double()
    assert float((got - want).norm() / want.norm()) <= BOUND
    assert float(((got - want) / want).abs().max()) <= 4 * BOUND


@pytest.mark.parametrize("chain", ["none", "bias", "gelu", "residual"])
@pytest.mark.parametrize("m,n,k", [(1024, 768, 3072), (1500, 2308, 772), (999, 508, 2052), (300, 644, 3084)])
def test_chains(m, n, k, chain):
    exe, x, c = build(m, n, k, chain)
    assert "mm_exact" in exe.details[0], exe.details
    a = c["a"] if chain == "residual" else x.double()
    want = a @ c["weight.transpose"]
    if chain != "none":
        want = want + c["bias"]
    if chain == "gelu":
        want = torch.nn.functional.gelu(want, approximate="tanh")
    if chain == "residual":
        want = want + x.double()
    got = call(exe, x).double()
    # (the GELU's exponential and reciprocal are the hardware's, 2^-22 each)
    assert float((got - want).norm() / want.norm()) <= BOUND + (4e-7 if chain == "gelu" else 0)


def test_rows_of_any_magnitude():
    """Every row has a scale of its own: its result is as near as that of any other, and a row of zeros is the bias."""
    m, n, k = 1024, 768, 1536
    exe, x, c = build(m, n, k)
    assert "mm_exact" in exe.details[0], exe.details
    powers = torch.linspace(-100, 100, m, device="cuda").round()
    x = x * torch.exp2(powers)[:, None]
    x[5] = 0
    want = x.double() @ c["weight.transpose"] + c["bias"]
    got = call(exe, x).double()
    assert torch.equal(got[5], c["bias"])
    error = (got - want).norm(dim=1) / want.norm(dim=1)
    assert float(error.max()) <= BOUND


def test_infinities_and_nan_are_those_of_float32():
    m, n, k = 1024, 768, 1536
    exe, x, c = build(m, n, k, "gelu")
    assert "mm_exact" in exe.details[0], exe.details
    x[3, 7] = float("inf")
    x[70, 1535] = float("-inf")
    x[200, 0], x[200, 9] = float("inf"), float("-inf")
    x[1023, 40] = float("nan")
    x[600] = 3e38                                       # finite, and finite in 16 bits under its scale
    got = call(exe, x)
    pre = x.double() @ c["weight.transpose"] + c["bias"]
    for row in (3, 70):
        infinite = pre[row] > 0
        assert bool((got[row][infinite] == float("inf")).all()) and bool(((got[row][~infinite] == 0) | got[row][~infinite].isnan()).all())
    assert bool(got[1023].isnan().all())
    others = torch.ones(m, dtype=torch.bool, device="cuda")
    others[[3, 70, 200, 600, 1023]] = False
    want = torch.nn.functional.gelu(pre, approximate="tanh")
    assert bool(got[others].isfinite().all()) and float((got[others] - want[others]).norm() / want[others].norm()) <= BOUND + 4e-7


def test_weights_that_make_up_for_a_row_s_spread_keep_the_other_kernels():
    """Features of very different magnitudes and weights that level them: two terms under one power of two would lose the small ones."""
    m, n, k = 1024, 2304, 768
    spread = np.exp2(np.linspace(-20, 20, k)).astype(np.float32)
    exe, x, c = build(m, n, k, scale=(1 / spread)[:, None])
    assert "mm_exact" not in exe.details[0], exe.details
    x = x * torch.from_numpy(spread).cuda()
    want = x.double() @ c["weight.transpose"] + c["bias"]
    assert float((call(exe, x).double() - want).norm() / want.norm()) <= 5e-6          # (the other kernels': 2^-23 per 8 of K in one accumulator)


def norm_linear(d, n, m=1024, second_reader=False):
    """LayerNorm and a Linear behind it; a residual of the LayerNorm's output for a second reader."""
    from perf import cases

    p = cases._Plan("norm_linear", (m, d), (m, n))
    h = p.buffer(m, d)
    p.layernorm(p.x, "ln.", h)
    p.linear(h, "fc.", n, p.y, residual=h if second_reader else None)
    return p.spec()


def run_plan(plan, consts, x, **env):
    import os

    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable

    with pytest.MonkeyPatch.context() as patch:
        for name, value in env.items():
            patch.setenv(name, value)
        exe = GPUExecutable(program_from_plan(plan, "fp32"), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    return exe, call(exe, x)


@pytest.mark.parametrize("d,n,second_reader", [(768, 2304, False), (2048, 2048, True), (772, 2304, False), (128, 4096, False), (4096, 1024, False), (8196, 768, False)])
def test_a_layernorm_leaves_its_rows_split(d, n, second_reader):
    """A warp or a block per row; the same bits whether the float32 rows are stored as well or not."""
    from perf import cases

    plan = norm_linear(d, n, second_reader=second_reader)
    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    x = torch.randn(1024, d, device="cuda") * 3 + 1
    exe, got = run_plan(plan, consts, x)
    assert "mm_exact" in exe.details[1] and "A copied" not in exe.details[1] and exe.device_launches == 2, exe.details
    _, stored = run_plan(plan, consts, x, KILN_GPU_MIRROR_ONLY="0")
    assert torch.equal(got, stored)
    c = {name: torch.from_numpy(v).cuda().double() for name, v in consts.items()}
    h = torch.nn.functional.layer_norm(x.double(), (d,), c["ln.weight"], c["ln.bias"], 1e-5)
    want = h @ c["fc.weight.transpose"] + c["fc.bias"] + (h if second_reader else 0)
    assert float((got.double() - want).norm() / want.norm()) <= 2 * BOUND          # (the LayerNorm's own float32 sums)


def test_infinities_a_layernorm_makes():
    """A scale of infinity: its column is infinite in every row, which the matmul then sums from the float32 rows."""
    from perf import cases

    d, n = 768, 2304
    plan = norm_linear(d, n)
    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    consts["ln.weight"][5] = np.inf
    x = torch.randn(1024, d, device="cuda")
    x[9, 3] = float("nan")
    exe, got = run_plan(plan, consts, x)
    assert "mm_exact" in exe.details[1] and exe.device_launches == 2, exe.details
    h5 = (x[:, 5] - x.mean(1)) * float("inf")
    want = h5[:, None] * torch.from_numpy(consts["fc.weight.transpose"][5]).cuda()
    rows = torch.arange(1024, device="cuda") != 9
    assert torch.equal(got[rows], want[rows]) and bool(got[9].isnan().all())


@pytest.mark.parametrize("m,d,wide", [(1024, 768, 3072), (1000, 772, 3004), (2048, 512, 2048)])
@pytest.mark.parametrize("gelu", [True, False])
def test_a_matmul_behind_a_layernorm_leaves_its_rows_split(m, d, wide, gelu):
    """Its results have a known bound: two Linears and the LayerNorm in front are three launches, and a row of NaN stays one."""
    from perf import cases

    p = cases._Plan("mlp", (m, d), (m, d))
    h, f = p.buffer(m, d), p.buffer(m, wide)
    p.layernorm(p.x, "ln.", h)
    p.linear(h, "fc.", wide, f, gelu=gelu)
    p.linear(f, "proj.", d, p.y)
    plan = p.spec()
    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    consts["fc.bias"] += np.float32(3)
    x = torch.randn(m, d, device="cuda") * torch.exp2(torch.linspace(-20, 20, m, device="cuda"))[:, None]
    x[7, 3] = float("nan")
    exe, got = run_plan(plan, consts, x)
    assert all("mm_exact" in detail and "A copied" not in detail for detail in exe.details[1:]) and exe.device_launches == 3, exe.details
    _, stored = run_plan(plan, consts, x, KILN_GPU_MIRROR_ONLY="0")
    assert torch.equal(got.nan_to_num(), stored.nan_to_num())
    c = {name: torch.from_numpy(v).cuda().double() for name, v in consts.items()}
    h = torch.nn.functional.layer_norm(x.double(), (d,), c["ln.weight"], c["ln.bias"], 1e-5)
    f = h @ c["fc.weight.transpose"] + c["fc.bias"]
    want = (torch.nn.functional.gelu(f, approximate="tanh") if gelu else f) @ c["proj.weight.transpose"] + c["proj.bias"]
    rows = torch.arange(m, device="cuda") != 7
    assert bool(got[7].isnan().all())
    assert float((got.double() - want)[rows].norm() / want[rows].norm()) <= 3 * BOUND
