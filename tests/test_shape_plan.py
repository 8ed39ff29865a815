"""The plan of a replayed Cholesky column evaluation (ShapeGraph in csrc/gx_api.cu) is made field by field from a
column plan: every field that sets the work units and launches has to be among them, or a replay is cut and launched
by other rules than the plan it stands for (its results are the same, its speed is not)."""

from __future__ import annotations

import re
from pathlib import Path

SOURCE = (Path(__file__).resolve().parents[1] / "giaoint_gb300" / "csrc" / "gx_api.cu").read_text()


def _body(signature: str) -> str:
    start = SOURCE.index(signature)
    open_brace = SOURCE.index("{", SOURCE.index(")", start))
    depth = 0
    for i in range(open_brace, len(SOURCE)):
        depth += {"{": 1, "}": -1}.get(SOURCE[i], 0)
        if depth == 0:
            return SOURCE[open_brace:i]
    raise AssertionError(signature)


def test_shape_plans_have_what_the_unit_and_launch_rules_read():
    reads: set[str] = set()
    for signature in ("void make_units(gx_context* ctx, PlanData& plan)", "gx::QuartetClass unit_class(",
                      "bool runs_dense(", "void launch_class(", "std::vector<PlanLaunch> plan_launches("):
        reads |= set(re.findall(r"\bplan\.(\w+)", _body(signature)))
    made = {f for f in reads if f.startswith("unit")}  # by make_units itself
    start = SOURCE.index("PlanData& sp = sg->plan;")
    copied = set(re.findall(r"\bsp\.(\w+)", SOURCE[start:SOURCE.index("make_units(ctx, sp);", start)]))
    # (tuned: a shape is never tuned)
    assert reads - made - {"tuned"} <= copied, reads - made - copied
