"""What the tensor-core kernels do when a bounded wait runs out, read from their sources (no kernel is made to fail for it)."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "kiln-compiler_b200" / "csrc"
KERNELS = sorted(f.name for f in CSRC.glob("*.cu") if re.search(r"__shared__ int abort_flag", f.read_text()))


def test_the_kernels_with_bounded_waits():
    assert KERNELS == ["attention.cu", "attention_bf16.cu", "matmul_pair.cu", "matmul_small.cu", "matmul_tc.cu"]


@pytest.mark.parametrize("name", KERNELS)
def test_copies_in_flight_land_before_shared_memory_is_released(name):
    """A parity test holds for one of the two parities at any time, so asking for either is no wait."""
    text = (CSRC / name).read_text()
    assert not re.search(r"mbar_try_wait\(([^,]+), 0\) \|\| mbar_try_wait\(\1, 1\)", text)
    way_out = text.index("if (abort_flag && threadIdx.x == 0) let_copies_land();")
    assert 0 < text.index("tcgen05.dealloc") - way_out < 1000           # ... and before tensor memory is
