"""Filters whose kept-row lists and CASE results nearly fill a block's shared memory:
large blocks that a plan asks for, and plans of many expensive CASE branches at
the shapes that large calls are tuned over."""
import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T, pack_validity
from helpers import OracleEngine, assert_tables_equal

SCHEMA = [T.INT64, T.FLOAT64, T.INT32]
SHAPES = [(32, 32), (32, 56), (32, 64), (16, 128)]
LIMIT = 227 * 1024


def _table(n):
    rng = np.random.default_rng(n)
    data = [rng.integers(-(1 << 40), 1 << 40, n), rng.normal(0, 1e3, n), rng.integers(-50, 51, n).astype(np.int32)]
    return [HostColumn(t, d, pack_validity(rng.random(n) >= 0.1)) for t, d in zip(SCHEMA, data)]


def _branches(count):
    """CASE outputs whose branches a filter evaluates apart."""
    return ["CASE(>($2, %d), ROUND(/(/($1, %d.5), $0), 3), $1)" % (k - 6, k + 3) for k in range(count)]


@pytest.mark.parametrize("kind", [1, 6], ids=["filter", "batched"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_large_blocks_compile(shape, kind):
    import blazingsql_gb300 as g
    plan = g.Plan(SCHEMA, ">($2, 0)", ["$0"], nullable=[True] * 3, block_threads=shape[0] * 32, words_per_warp=shape[1])
    assert plan.resources(kind, [True] * 3)[2] <= LIMIT


def test_branches_fit_the_tuned_shapes():
    import blazingsql_gb300 as g
    for warps, words in ((4, 8), (8, 4)):
        plan = g.Plan(SCHEMA, ">($2, 0)", _branches(24), nullable=[True] * 3, block_threads=warps * 32, words_per_warp=words)
        assert plan.resources(1, [True] * 3)[2] <= LIMIT


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_large_blocks(shape):
    import blazingsql_gb300 as g
    outputs = ["$0", "$1", "+($0, $2)"]
    for n in (1, 8191, 300_007):
        cols = _table(n)
        plan = g.Plan(SCHEMA, ">($2, -20)", outputs, block_threads=shape[0] * 32, words_per_warp=shape[1])
        got, _ = plan.execute(cols)
        assert_tables_equal([c.to_host() for c in got], OracleEngine(2).filter_project(cols, ">($2, -20)", outputs),
                            what=f"{shape} {n} rows")


@pytest.mark.gpu
@pytest.mark.parametrize("count", [2, 12])
def test_branches(count):
    import blazingsql_gb300 as g
    from blazingsql_gb300.api import DeviceColumn
    outputs = _branches(count)
    for n, calls in ((3001, 1), ((1 << 22) + 5, 6)):  # 6: the first call, the shapes' trials, the chosen shape
        cols = _table(n)
        expected = OracleEngine(8).filter_project(cols, ">($2, 40)", outputs)
        device = [DeviceColumn.from_host(c) for c in cols]
        for _ in range(calls):
            got = g.filter_project(device, ">($2, 40)", outputs)
            assert_tables_equal([c.to_host() for c in got], expected, what=f"{count} branches, {n} rows")
