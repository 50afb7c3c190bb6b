"""FP32 mode's fused attention: each of its kernels by option, named by the plan's details, against float64 at any length; and the TF32 form's
tails from the projection or from a pass."""

import pytest
import torch
from test_gpu_attention_pairs import block, reference

pytestmark = pytest.mark.gpu

# The TF32 form: 2^-23 cut off with each of up to 3 T / 8 MMAs of an accumulator (1030 tokens: 4.6e-5 if all were whole and of one sign; the attention's
# sums are of both signs and a third of what the block adds): within the 1e-5 that this precision promises.
BOUND = {"fma": 1e-6, "tensor": 1e-6, "tf32": 1e-5}
NAMES = {"fma": "on the CUDA cores", "tensor": "on float16 pairs", "tf32": "on TF32 pairs"}


@pytest.mark.parametrize("choice", ["fma", "tensor", "tf32"])
@pytest.mark.parametrize("tokens,heads,batch", [(129, 12, None), (1030, 4, None), (1024, 12, None), (333, 12, 6), (257, 8, 3)])
def test_every_kernel_at_any_length(tokens, heads, batch, choice):
    exe, consts, x, got = block(tokens, heads, batch, KILN_GPU_FP32_ATTENTION=choice)
    assert any(NAMES[choice] in detail for detail in exe.details), exe.details
    added, want = reference(consts, x, heads)
    assert float((got.double() - want).norm() / added.norm()) <= BOUND[choice]


@pytest.mark.parametrize("odd", ["", "a NaN"])
@pytest.mark.parametrize("tokens,batch", [(1024, None), (512, 2)])
def test_tails_of_the_projection_are_those_of_the_pass(tokens, batch, odd):
    """Columns of Q and K whose bounds are far apart keep the TF32 form."""
    def change(consts, x):
        w, b = consts["c_attn.weight.transpose"], consts["c_attn.bias"]
        w[:, 3] *= 4096
        b[3] *= 4096
        w[:, 768 + 3] /= 4096
        b[768 + 3] /= 4096
        if odd:
            x[..., tokens - 9, 3] = float("nan")

    exe, consts, x, got = block(tokens, 12, batch, change)
    passed, _, _, by_pass = block(tokens, 12, batch, change, KILN_GPU_FP32_ATTENTION="tensor")
    assert all(any("on TF32 pairs" in detail for detail in e.details) for e in (exe, passed)), (exe.details, passed.details)
    assert passed.device_launches == exe.device_launches + 1
    assert torch.equal(got.isnan(), by_pass.isnan()) and torch.equal(got.nan_to_num(), by_pass.nan_to_num())
    if not odd:
        added, want = reference(consts, x, 12)
        assert float((got.double() - want).norm() / added.norm()) <= BOUND["tf32"]


@pytest.mark.parametrize("std", [1.0, 1e-8])
@pytest.mark.parametrize("tokens,batch", [(1024, None), (333, 6)])
def test_blocks_without_biases(tokens, batch, std):
    """Rows of next to nothing come out of a LayerNorm far below the bounds of what follows."""
    from test_gpu_attention_pairs import BOUND as PAIRS

    def change(consts, x):
        for name in consts:
            if name.endswith("bias"):
                consts[name][:] = 0
        x *= std

    exe, consts, x, got = block(tokens, 12, batch, change)
    assert any("on float16 pairs" in detail for detail in exe.details), exe.details
    added, want = reference(consts, x, 12)
    assert float((got.double() - want).norm() / added.norm()) <= PAIRS
