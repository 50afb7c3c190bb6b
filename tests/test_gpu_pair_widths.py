"""The matmul kernel on SM pairs at each of its tile widths: ragged last tiles of rows and columns, K off a slab,
weights along K and operands along N."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# float32 sums of operands rounded to 2^-9 (bf16) or cut to 2^-10 (TF32), relative to the 2-norm: about 0.8 of that per product
BOUND = {"tf32": 1e-3, "bf16": 3e-3}


def run(p, precision):
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    plan = p.spec()
    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    exe = GPUExecutable(program_from_plan(plan, precision), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    x = torch.randn(plan.input_shapes[0], generator=torch.Generator(device="cuda").manual_seed(0), device="cuda")
    outs = [exe(x)[0] for _ in range(3)]
    exe.status()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    return exe, x.double(), {name: torch.from_numpy(c).cuda().double() for name, c in consts.items()}, outs[0].double()


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("m,n,k,width", [(4096, 640, 640, 160), (4000, 612, 200, 160), (1024, 3072, 768, 192), (1000, 3028, 772, 192), (2432, 1568, 1536, 224),
                                         (2305, 1444, 1028, 224), (8192, 2304, 512, 256), (8190, 2304, 516, 256)])
def test_linear_at_every_width(m, n, k, width, precision):
    from perf import cases

    p = cases._Plan("linear", (m, k), (m, n))
    p.linear(p.x, "", n, p.y)
    exe, x, c, got = run(p, precision)
    assert f"mm_pair {width} columns" in exe.details[0], exe.details
    want = x @ c["weight.transpose"] + c["bias"]
    assert float((got - want).norm() / want.norm()) <= BOUND[precision]
    assert float((got - want).abs().max() / want.std()) <= 10 * BOUND[precision]


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("m,n", [(1024, 3072), (1000, 3008)])
def test_an_operand_along_n(m, n, precision):
    """B is an activation [K, N]: whole chunks of its columns only (192 columns in TF32, not in BF16)."""
    from perf import cases

    k = 512
    p = cases._Plan("product", (k, 128), (1, m, n))
    b = p.buffer(k, n)
    p.linear(p.x, "0.", n, b)
    p.bmm(p.const("a", 1, m, k), b.as_((1, k, n)), p.y)
    exe, x, c, got = run(p, precision)
    assert "mm_pair" in exe.details[1] and ("192 columns" in exe.details[1]) == (precision == "tf32"), exe.details
    want = c["a"] @ (x @ c["0.weight.transpose"] + c["0.bias"])
    assert float((got - want).norm() / want.norm()) <= 2 * BOUND[precision]


@pytest.mark.parametrize("epilogue", ["bias", "gelu", "residual", "relu"])
@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("m,n,k", [(2048, 768, 3072), (1998, 768, 3080), (1793, 708, 4100), (600, 2048, 2048)])
def test_k_in_halves(m, n, k, precision, epilogue):
    """Two pairs per tile, half of K each: ragged rows and columns (blocks of 32 columns that one of the pairs has not), steps of K that do not
    come out even, every kind of epilogue."""
    from perf import cases

    p = cases._Plan("linear", (m, k), (m, n))
    if epilogue == "relu":
        p.kernel("matmul", [("matmul", [("operand", 0), ("operand", 1)], (m, n)), ("add", [("node", 0), ("operand", 2)], (m, n)), ("relu", [("node", 1)], (m, n))],
                 [p.x, p.const("weight.transpose", k, n), p.const("bias", n)], [(2, p.y)])
    else:
        p.linear(p.x, "", n, p.y, gelu=epilogue == "gelu", residual=p.const("other", m, n) if epilogue == "residual" else None)
    exe, x, c, got = run(p, precision)
    assert "2 splits" in exe.details[0] and "mm_pair" in exe.details[0], exe.details
    want = x @ c["weight.transpose"] + c["bias"]
    want = {"bias": want, "relu": want.relu(), "gelu": torch.nn.functional.gelu(want, approximate="tanh")}.get(epilogue, want + c.get("other", 0))
    assert float((got - want).norm() / want.norm()) <= BOUND[precision]
    assert float((got - want).abs().max() / want.std()) <= 10 * BOUND[precision]


@pytest.mark.parametrize("m,n,k,precision,how", [(2048, 1024, 1024, "tf32", "128 columns"), (2048, 1000, 2048, "bf16", "128 columns"), (1024, 4096, 1000, "bf16", "256 columns"),
                                                 (4096, 4096, 4096, "tf32", "256 columns"), (2048, 768, 3072, "bf16", "192 columns, 1 slabs, 2 splits")])
def test_the_quicker_form_is_taken(m, n, k, precision, how):
    """11.9 us against 13.9 in halves of K; 15.0 against 16.9; 14.9 against 16.2 at 128 columns; 191 against 201 at 192; 17.4 against 18.6 whole at 128."""
    from perf import cases

    p = cases._Plan("linear", (m, k), (m, n))
    p.linear(p.x, "", n, p.y)
    exe, x, c, got = run(p, precision)
    assert f"mm_pair {how}" in exe.details[0] and ("splits" in how) == ("splits" in exe.details[0]), exe.details
    want = x @ c["weight.transpose"] + c["bias"]
    assert float((got - want).norm() / want.norm()) <= BOUND[precision]


@pytest.mark.parametrize("batch,m,n,k", [(2, 512, 768, 3072), (3, 300, 736, 2052)])
def test_k_in_halves_of_a_batch_and_an_operand_along_n(batch, m, n, k):
    """Batched, B an activation [K, N] in TF32: the second pair of a cluster starts in the middle of its rows."""
    from perf import cases

    p = cases._Plan("product", (batch * k, 128), (batch, m, n))
    b = p.buffer(batch * k, n)
    p.linear(p.x, "0.", n, b)
    p.bmm(p.const("a", batch, m, k), b.as_((batch, k, n)), p.y)
    exe, x, c, got = run(p, "tf32")
    assert "mm_pair" in exe.details[1] and "2 splits" in exe.details[1], exe.details
    want = c["a"] @ (x @ c["0.weight.transpose"] + c["0.bias"]).view(batch, k, n)
    assert float((got - want).norm() / want.norm()) <= 2 * BOUND["tf32"]
    assert float((got - want).abs().max() / want.std()) <= 20 * BOUND["tf32"]


@pytest.mark.parametrize("m", [2048, 1990])
def test_k_in_halves_where_only_the_bf16_copy_is_stored(m):
    from perf import cases

    p = cases._Plan("mlp", (m, 3072), (m, 768))
    f = p.buffer(m, 768)
    p.linear(p.x, "0.", 768, f)
    p.linear(f, "2.", 768, p.y)
    exe, x, c, got = run(p, "bf16")
    assert "mm_pair" in exe.details[0] and "2 splits" in exe.details[0], exe.details
    want = (x @ c["0.weight.transpose"] + c["0.bias"]) @ c["2.weight.transpose"] + c["2.bias"]
    assert float((got - want).norm() / want.norm()) <= 2 * BOUND["bf16"]


@pytest.mark.parametrize("residual,how", [(False, "128 columns"), (True, "2 splits")])
def test_a_residual_comes_under_the_exchange_of_halves(residual, how):
    """1700 x 768 x 768 TF32: with a residual behind another kernel 15.9 us at 128 columns, 15.4 in halves of K; without one (1792 rows) 10.0 and 10.4."""
    from perf import cases

    p = cases._Plan("linear", (1700, 768), (1700, 768))
    p.linear(p.x, "", 768, p.y, residual=p.x if residual else None)
    exe, x, c, got = run(p, "tf32")
    assert "mm_pair" in exe.details[0] and how in exe.details[0], exe.details
    want = x @ c["weight.transpose"] + c["bias"] + (x if residual else 0)
    assert float((got - want).norm() / want.norm()) <= BOUND["tf32"]
