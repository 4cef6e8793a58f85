"""Scores and weights of a routing call may be one plane: no kernel promises the compiler that they are not (no GPU: read from the source)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "recipe_dev_b200" / "csrc"


def test_planes_that_may_be_one_are_not_declared_apart():
    text = (CSRC / "rq_moe.cu").read_text()
    for name in ("route_token", "rq_route_kernel", "pick_by_warp", "rq_moe_route_plan_kernel"):
        parameters = re.search(name + r"\(([^)]*)\) \{", text).group(1)
        assert "float* scores" in parameters and "float* weights" in parameters, name
    # within one kernel the plan reads the weights that the routing wrote
    assert "float* routing" in re.search(r"plan_token\(([^)]*)\) \{", text).group(1)
