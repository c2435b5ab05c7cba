"""Registers of the learner's ordered kernel with column copies as outputs: 32 for
conjuncts that compare and add columns without NULLs, 48 for nullable columns and
divisions, which would spill at 32, 40 for transcendental functions; computed
outputs are not held to a number.  No such kernel spills more than a few values."""
import re

import pytest

from blazingsql_gb300 import workloads as W
from blazingsql_gb300.types import TypeId as T

SCHEMA = [T.INT64] * 4 + [T.FLOAT64] * 4
SUMS = "AND(>(+($0, $1), 100000), <(*($4, 2.0), 100000.0), <($2, 100000))"
DIVISIONS = "AND(>(/($4, $5), 0.1), <(/($5, $6), 5.0), >(/($6, $4), 0.2), >($0, 100))"
LOGS = "AND(>($0, 100000), <(LN(+($4, 1.0)), 12.0), <($2, 1000))"
CASES = [(W.C4_CONDITION, False, 8), (W.C4_CONDITION, True, 5), (SUMS, False, 8), (SUMS, True, 5), (DIVISIONS, False, 5),
         (DIVISIONS, True, 5), (LOGS, False, 6), (LOGS, True, 6)]


@pytest.mark.parametrize("condition,nullable,blocks", CASES)
def test_resident_blocks(condition, nullable, blocks):
    import blazingsql_gb300 as g
    plan = g.Plan(SCHEMA, condition, ["$3", "$7"], nullable=[True] * 8)
    source = plan.kernel_source(4, [nullable] * 8)
    assert "#define GX_WARPS 8\n" in source
    assert re.search(r"GX_LB __launch_bounds__\(GX_WARPS \* 32, (\d+)\)", source).group(1) == str(blocks)
    regs, spilled, _ = plan.resources(4, [nullable] * 8)
    assert regs <= 65536 // (blocks * 256)
    assert spilled <= 256


def test_computed_outputs():
    import blazingsql_gb300 as g
    plan = g.Plan(SCHEMA, W.C4_CONDITION, ["$3", "+($7, 1.0)"], nullable=[False] * 8)
    assert "#define GX_LB __launch_bounds__(GX_WARPS * 32)\n" in plan.kernel_source(4, [False] * 8)
