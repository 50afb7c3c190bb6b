"""The plans that the performance cases write for themselves are the ones stored from Kiln's own passes."""

import json

import pytest

from kiln_b200.spec import PlanSpec
from kiln_b200.workloads import PLAN_DIR
from perf import cases

SAME = [({"kind": "linear", "m": 128, "n": 768, "k": 3072}, "linear_128x768x3072"), ({"kind": "linear", "m": 2048, "n": 3072, "k": 768}, "linear_2048x3072x768"),
        ({"kind": "linear", "m": 1, "n": 3072, "k": 768}, "linear_1x3072x768"), ({"kind": "mlp", "tokens": 2048, "d": 768}, "mlp_2048"),
        ({"kind": "layernorm", "rows": 2048, "d": 768}, "layernorm_2048x768"), ({"kind": "softmax", "heads": 12, "rows": 512, "cols": 512}, "softmax_12x512x512"),
        ({"kind": "bias_gelu", "rows": 2048, "d": 3072}, "bias_gelu_2048x3072"), ({"kind": "block", "tokens": 128, "heads": 12}, "gpt2_block_t128"),
        ({"kind": "block", "tokens": 1024, "heads": 12}, "gpt2_block_t1024"), ({"kind": "batched_block", "batch": 8, "tokens": 1024, "heads": 12}, "gpt2_block_b8_t1024")]


def form(plan):
    """What a plan has the backend do: everything but names."""
    d = plan.to_json()
    names = {}
    for k in d["kernels"]:
        k["name"] = ""
        for o in list(k["inputs"]) + [o for _, o in k["outputs"]]:
            if o["base"][0] == "const":
                o["base"] = ["const", names.setdefault(o["base"][1], len(names))]
    return json.loads(json.dumps({key: d[key] for key in ("input_shapes", "output_shapes", "arena_bytes", "kernels")}))


@pytest.mark.parametrize("case,stored", SAME, ids=[s for _, s in SAME])
def test_the_cases_have_the_plans_of_kilns_passes(case, stored):
    ours, kilns = cases._plan(case), PlanSpec.loads((PLAN_DIR / f"{stored}.json").read_text())
    assert form(ours) == form(kilns)
