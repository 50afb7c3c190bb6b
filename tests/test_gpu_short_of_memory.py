"""What the plans do where memory is short: weights that are not copied, and the bounds on those that are."""

import pytest

from test_gpu_sizes import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "tf32", "bf16"])
@pytest.mark.parametrize("m", [1, 17, 128, 364])
@pytest.mark.parametrize("n,k", [(768, 768), (1000, 771), (3072, 96)])
def test_linear_without_copies_of_its_weight(m, n, k, precision, monkeypatch):
    """N a multiple of 32 (the weight is describable as it is) and not (it is copied to aligned rows)."""
    monkeypatch.setenv("KILN_GPU_WEIGHT_COPIES", "0")
    check({"kind": "linear", "m": m, "n": n, "k": k, "precision": precision}, calls=2)
