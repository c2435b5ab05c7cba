"""Columns that a condition proves valid in every kept row: IS NOT NULL proves
its operand where it is a conjunct, and nothing beneath another operator, where
a kept row may hold a NULL.  In the generated kernels, and against the oracle
through copied and computed outputs, group keys and aggregates."""
import re

import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T, pack_validity
from helpers import OracleEngine, assert_tables_equal
from oracle import agg_ref
from test_aggregate import COUNT_VALID, MEAN, MIN, SUM, _compare, _run

SCHEMA = [T.INT64, T.INT32, T.INT32]
OUTPUTS = ["$0", "$1", "+($0, $1)", "CASE(IS NULL($0), $2, $1)"]
# condition: which of $0, $1 it proves valid
CONDITIONS = {
    "IS NOT NULL($0)": (True, False),
    "AND(IS NOT NULL($0), >($1, 0))": (True, True),
    "IS NOT NULL(+($0, $1))": (True, True),
    "NOT(IS NOT NULL($0))": (False, False),
    "<>(IS NOT NULL($0), true)": (False, False),
    "=(IS NOT NULL($0), IS NOT NULL($1))": (False, False),
    "IS NOT NULL(IS NOT NULL($0))": (False, False),
    "NOT(AND(IS NOT NULL($0), >($1, 5)))": (False, True),
    "AND(NOT(IS NOT NULL($0)), IS NOT NULL($1))": (False, True),
    "OR(IS NOT NULL($0), >($2, 0))": (False, False),
}


def _table(n):
    rng = np.random.default_rng(n)
    valid = [pack_validity(rng.random(n) >= 0.4), pack_validity(rng.random(n) >= 0.3), None]
    data = [rng.integers(-9, 10, n), rng.integers(-9, 10, n).astype(np.int32), rng.integers(-9, 10, n).astype(np.int32)]
    return [HostColumn(t, d, v) for t, d, v in zip(SCHEMA, data, valid)]


@pytest.mark.parametrize("kind", [1, 4, 6], ids=["filter", "ordered", "batched"])
@pytest.mark.parametrize("condition", list(CONDITIONS))
def test_masks_written_in_the_source(condition, kind):
    import blazingsql_gb300 as g
    plan = g.Plan(SCHEMA, condition, ["$0", "$1"], nullable=[True, True, False])
    source = plan.kernel_source(kind, [True, True, False])
    for j, proven in enumerate(CONDITIONS[condition]):
        writes = set(re.findall(r"(gx_put_\w+)\(a\.out_mask\[%d\]" % j, source))
        assert writes == {"gx_put_ones" if proven else "gx_put_bits"}, f"output {j}"


@pytest.mark.gpu
@pytest.mark.parametrize("condition", list(CONDITIONS))
def test_filters(condition):
    import blazingsql_gb300 as g
    for n in (1, 100, 20_011):
        cols = _table(n)
        expected = OracleEngine(2).filter_project(cols, condition, OUTPUTS)
        got = [c.to_host() for c in g.filter_project(cols, condition, OUTPUTS)]
        assert_tables_equal(got, expected, what=f"{condition} {n} rows")
        query = f"LogicalFilter(condition=[{condition}])"
        got = [c.to_host() for c in g.process_filter(cols, query)]
        assert_tables_equal(got, OracleEngine(2).process_filter(cols, query), what=f"{query} {n} rows")


@pytest.mark.gpu
@pytest.mark.parametrize("condition", list(CONDITIONS))
def test_aggregates(condition):
    cols = _table(20_011)
    aggs = [(SUM, "$0"), (COUNT_VALID, "$0"), (MEAN, "$1"), (MIN, "+($0, $1)")]
    for keys in ([], [0], [1, 0], [2]):
        _compare(_run(cols, condition, keys, aggs), agg_ref.filter_aggregate(cols, condition, keys, aggs), len(keys),
                 f"{condition} by {keys}")
