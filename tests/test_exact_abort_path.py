"""What the exact-FP32 kernel on float16 pairs does when a bounded wait runs out, read from its source (as for the other tensor-core kernels)."""

import re
from pathlib import Path

SOURCE = Path(__file__).resolve().parent.parent / "kiln-compiler_b200" / "csrc" / "matmul_exact.cuh"


def test_copies_in_flight_land_before_shared_memory_is_released():
    text = SOURCE.read_text()
    way_out = text.index("if (abort_flag && threadIdx.x == 0) let_copies_land();")
    assert 0 < text.index("tcgen05.dealloc") - way_out < 1000           # ... and before tensor memory is


def test_no_warp_waits_for_one_that_may_have_given_up():
    """Between the roles' start and the common exit there is no barrier of threads: a warp that gives up leaves at once."""
    text = SOURCE.read_text()
    roles = text[text.index("TMA producer ----"):text.index("common exit ----")]
    assert not re.search(r"__syncthreads|bar\.sync|cluster_wait", roles)
