"""Every form of the matmul kernel for few tiles, asked for by name: tile widths, K splits (one CTA with a ring that is used again to
eight with one step each), the three ways A comes, accumulators added up in the loop or behind it."""

import numpy as np
import pytest
import torch

from oracle.plan_oracle import run_plan, scale_relative_error
from test_gpu_sizes import BOUND

pytestmark = pytest.mark.gpu


def run(m, n, k, precision, asked=0, calls=2):
    from kiln_b200 import _cabi
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable
    from perf import cases

    plan = cases._plan({"kind": "linear", "m": m, "n": n, "k": k})
    consts = cases._constants(plan.const_shapes, np.random.default_rng(1))
    exe = GPUExecutable(program_from_plan(plan, precision), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    if asked:
        _cabi.check(exe._lib.kb200_plan_set_option(exe._plan, _cabi.OPT_FEW_TILES, asked))
        exe._bind()
    for seed in range(calls):
        x = (np.random.default_rng(2 + seed).standard_normal((m, k)) * k ** -0.5).astype(np.float32)
        (got,) = exe(torch.from_numpy(x).cuda())
        torch.cuda.synchronize()
        exe.status()
        (want,) = run_plan(plan.to_json(), [x], consts, dtype=np.float64)
        assert scale_relative_error(got.cpu().numpy(), want) <= BOUND[precision]
    return exe._lib.kb200_kernel_detail(exe._plan, 0).decode()


@pytest.mark.parametrize("precision", ["fp32", "tf32", "bf16"])
@pytest.mark.parametrize("columns", [64, 96, 128])
@pytest.mark.parametrize("splits", [1, 2, 4, 8])
def test_every_tile_and_split(columns, splits, precision):
    """Two rows of tiles, the second of one row; a last tile of 4 columns; K of 1600 in 25 to 50 steps, the last of them short."""
    detail = run(129, 3 * columns + 4, 1596, precision, columns + 1000 * splits)
    drains = precision == "fp32" and columns == 128 and splits < 8
    if drains and not detail.startswith("mm_small"):         # two accumulators, each needed again before it is drained
        return
    assert detail.startswith(f"mm_small {columns} columns, {splits} splits"), detail


@pytest.mark.parametrize("precision,columns", [("fp32", 64), ("tf32", 64), ("tf32", 96), ("tf32", 128), ("bf16", 64), ("bf16", 96), ("bf16", 128)])
@pytest.mark.parametrize("splits", [1, 4])
def test_rows_read_by_the_kernel(precision, columns, splits):
    """A on no pitch: the warps' own reads, and a copy instead of them."""
    assert ", A gathered" in run(130, 2 * columns + 4, 1031, precision, columns + 1000 * splits + 30000)
    assert ", A copied" in run(130, 2 * columns + 4, 1031, precision, columns + 1000 * splits + 10000)


@pytest.mark.parametrize("columns", [64, 96, 128])
@pytest.mark.parametrize("splits", [1, 4])
def test_float32_rows_for_bf16_products(columns, splits):
    assert ", A float32" in run(130, 2 * columns + 4, 1028, "bf16", columns + 1000 * splits + 20000)


@pytest.mark.parametrize("m,n,k", [(2, 64, 64), (17, 65, 96), (128, 768, 300), (128, 768, 768), (17, 96, 4096), (300, 64, 4096), (5, 2304, 771), (1000, 768, 3072)])
def test_exact_fp32_with_few_and_many_accumulators(m, n, k):
    """One to five accumulators of one to sixteen steps, and rings of them that are drained in the loop."""
    for columns in (64, 96, 128):
        for splits in (1, 2, 8):
            run(m, n, k, "fp32", columns + 1000 * splits, calls=1)


def test_the_estimates_choose_this_kernel_where_its_tests_need_it():
    """Sizes that the other tests give to this kernel's forms: one row of tiles, odd pitches, a few rows of tiles."""
    for precision in ("fp32", "tf32", "bf16"):
        for m, n, k in [(2, 64, 64), (128, 64, 4096), (127, 68, 1000), (128, 3072, 768), (100, 768, 3072), (5, 64, 67), (33, 768, 3071)]:
            assert run(m, n, k, precision, calls=1).startswith("mm_small"), (m, n, k, precision)
    assert ", A gathered" in run(128, 4096, 129, "tf32", calls=1)
    assert ", drains" in run(17, 4096, 771, "fp32", calls=1)
