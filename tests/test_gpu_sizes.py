"""Sizes at the edges of the kernels' tilings, for every module the performance cases describe: widths no
vector access takes, rows longer than a warp's registers, sequences that end inside a tile.  Against
the float64 evaluation of the plan, within the bounds of the other parity tests."""

import numpy as np
import pytest
import torch

from oracle.plan_oracle import run_plan, scale_relative_error

pytestmark = pytest.mark.gpu

BOUND = {"fp32": 1e-5, "tf32": 2e-3, "bf16": 2e-2}


def check(case, impls=None, calls=1):
    from perf import cases

    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable

    case = {"precision": "fp32", **case}
    plan = cases._plan(case)
    consts = cases._constants(plan.const_shapes, np.random.default_rng(1))
    exe = GPUExecutable(program_from_plan(plan, case["precision"]), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    std = case["k"] ** -0.5 if case["kind"] == "linear" else 1.0
    for seed in range(calls):
        x = (np.random.default_rng(2 + seed).standard_normal(plan.input_shapes[0]) * std).astype(np.float32)
        (got,) = exe(torch.from_numpy(x).cuda())
        torch.cuda.synchronize()
        exe.status()
        (want,) = run_plan(plan.to_json(), [x], consts, dtype=np.float64)
        assert scale_relative_error(got.cpu().numpy(), want) <= BOUND[case["precision"]]
    if impls:
        assert set(exe.impls) == set(impls), exe.impls


@pytest.mark.parametrize("rows", [1, 700])
@pytest.mark.parametrize("d", [1, 3, 31, 32, 33, 34, 35, 64, 127, 250, 255, 257, 772, 1021, 1000, 1028, 2047, 2052, 4097, 8191, 8196, 16384])
def test_rows_of_any_width(d, rows):
    check({"kind": "layernorm", "rows": rows, "d": d}, ["row_layernorm"])
    check({"kind": "softmax", "heads": 1, "rows": rows, "cols": d}, ["row_softmax"])


def test_rows_beyond_the_registers():
    check({"kind": "layernorm", "rows": 3, "d": 16388}, ["row_generic"])


@pytest.mark.parametrize("rows,d", [(1, 5), (3, 1), (7, 33), (513, 1001), (65, 2050), (2047, 255), (5, 3), (1000, 2047)])
def test_elementwise_chain_of_any_width(rows, d):
    check({"kind": "bias_gelu", "rows": rows, "d": d}, ["ew_chain"])


@pytest.mark.parametrize("precision", ["fp32", "tf32", "bf16"])
@pytest.mark.parametrize("tokens", [2, 31, 63, 65, 127, 129, 255, 333, 1025])
def test_sequences_of_any_length(tokens, precision):
    check({"kind": "block", "tokens": tokens, "heads": 4, "precision": precision}, calls=2)
    if tokens < 1000:
        check({"kind": "batched_block", "batch": 3, "tokens": tokens, "heads": 2, "precision": precision}, calls=2)


@pytest.mark.parametrize("choice", ["fma", "tensor"])
@pytest.mark.parametrize("tokens", [33, 129, 1030])
def test_both_fp32_attention_kernels_take_any_length(tokens, choice, monkeypatch):
    monkeypatch.setenv("KILN_GPU_FP32_ATTENTION", choice)
    check({"kind": "block", "tokens": tokens, "heads": 4})
    check({"kind": "batched_block", "batch": 2, "tokens": tokens, "heads": 2})


@pytest.mark.parametrize("precision", ["fp32", "tf32", "bf16"])
@pytest.mark.parametrize("m,n,k", [(2, 64, 64), (5, 65, 67), (16, 72, 200), (31, 100, 71), (128, 1001, 772), (129, 131, 770), (333, 1000, 771),
                                   (257, 132, 65), (260, 1028, 68), (1000, 200, 1030)])
def test_linear_of_any_size(m, n, k, precision):
    """Operand rows off a 16-byte pitch, widths off a 128-byte column chunk, tiles with one row or column."""
    check({"kind": "linear", "m": m, "n": n, "k": k, "precision": precision}, ["mm_tcgen05"], calls=2)


@pytest.mark.parametrize("precision", ["fp32", "tf32", "bf16"])
@pytest.mark.parametrize("m,n,k", [(2, 64, 64), (128, 64, 4096), (127, 68, 1000), (128, 3072, 768), (100, 768, 3072), (17, 2304, 96), (128, 4096, 128),
                                   (65, 1028, 3000), (512, 768, 3072), (1024, 772, 3072), (364, 2308, 768), (1020, 3072, 768)])
def test_few_tiles(m, n, k, precision):
    """One row of tiles: K split over 1 to 8 CTAs, K ranges longer and shorter than the ring, ragged last slabs."""
    check({"kind": "linear", "m": m, "n": n, "k": k, "precision": precision}, ["mm_tcgen05"], calls=2)


@pytest.mark.parametrize("n,k", [(2, 3), (33, 7), (2355, 152), (1001, 3071)])
def test_one_row_of_any_size(n, k):
    check({"kind": "linear", "m": 1, "n": n, "k": k}, ["mm_gemv"], calls=2)


@pytest.mark.parametrize("precision", ["fp32", "tf32", "bf16"])
@pytest.mark.parametrize("m,n,k", [(5, 64, 67), (2, 68, 65), (128, 4096, 129), (33, 768, 3071), (300, 128, 1023), (130, 64, 2050), (1000, 64, 4099)])
def test_few_tiles_with_rows_on_no_pitch(m, n, k, precision):
    """A read by the kernel's own warps: rows from any element on, a partial last slab, a ring that is used again."""
    check({"kind": "linear", "m": m, "n": n, "k": k, "precision": precision}, ["mm_tcgen05"], calls=2)


@pytest.mark.parametrize("precision", ["fp32", "tf32", "bf16"])
@pytest.mark.parametrize("tokens,d", [(3, 132), (64, 512), (128, 1024), (129, 260)])
def test_mlp_of_few_tokens(tokens, d, precision):
    check({"kind": "mlp", "tokens": tokens, "d": d, "precision": precision}, ["mm_tcgen05"], calls=2)
