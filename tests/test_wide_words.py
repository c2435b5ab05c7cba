"""Warps of more than 32 words (more words, and rounds of kept rows, than lanes):
filters, projections and aggregations over nullable columns return what the
oracle does."""
import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T, pack_validity
from helpers import OracleEngine, assert_tables_equal
from oracle import agg_ref
from test_aggregate import COUNT_VALID, MEAN, SUM, _compare, _run

SCHEMA = [T.INT64, T.FLOAT64, T.INT32]
OUTPUTS = ["$0", "$1", "+($0, $2)", "/($1, $2)"]
CONDITIONS = ["IS NOT NULL($2)", "OR(IS NULL($1), >($2, 0))", "<($2, -40)", None]
SHAPES = [(1, 33), (1, 40), (2, 64), (4, 64)]


def _table(n):
    rng = np.random.default_rng(n)
    data = [rng.integers(-(1 << 40), 1 << 40, n), rng.normal(0, 1e3, n), rng.integers(-50, 51, n).astype(np.int32)]
    return [HostColumn(t, d, pack_validity(rng.random(n) >= p)) for t, d, p in zip(SCHEMA, data, (0.3, 0.5, 0.1))]


@pytest.mark.parametrize("kind", [0, 1, 3, 6])
def test_no_bit_is_read_from_a_lane(kind):
    import blazingsql_gb300 as g
    condition = CONDITIONS[1] if kind else None
    for words, lanes in ((32, True), (33, False)):
        plan = g.Plan(SCHEMA, condition, OUTPUTS, nullable=[True] * 3, block_threads=32, words_per_warp=words)
        source = plan.kernel_source(kind, [True] * 3).split("struct GxArgs")[1]  # past the device functions
        assert ("gx_wbit(" in source) == lanes


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("condition", CONDITIONS)
def test_plans(shape, condition):
    import blazingsql_gb300 as g
    oracle = OracleEngine(2)
    for n in (1, 1057, 2048, 40_007):
        cols = _table(n)
        plan = g.Plan(SCHEMA, condition, OUTPUTS, block_threads=shape[0] * 32, words_per_warp=shape[1])
        got, _ = plan.execute(cols)
        expected = (oracle.filter_project(cols, condition, OUTPUTS) if condition
                    else oracle.evaluate_expressions(cols, OUTPUTS))
        assert_tables_equal([c.to_host() for c in got], expected, what=f"{condition} {shape} {n} rows")


@pytest.mark.gpu
def test_aggregation(monkeypatch):
    monkeypatch.setenv("GX_WARPS", "4")
    monkeypatch.setenv("GX_WORDS", "40")
    cols = _table(40_007)
    aggs = [(SUM, "$0"), (COUNT_VALID, "$1"), (MEAN, "$1")]
    for condition in CONDITIONS:
        _compare(_run(cols, condition, [2], aggs), agg_ref.filter_aggregate(cols, condition, [2], aggs), 1, str(condition))
