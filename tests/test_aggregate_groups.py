"""Group counts at the edges of the aggregation kernel's shared-memory tables:
as many groups as a warp keeps accumulators for (32), one more, thousands (the
block's table), more than that table holds, groups that appear only late in the
table, one group, and inputs with NULLs."""
import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T, pack_validity
from oracle import agg_ref
from test_aggregate import COUNT_ALL, COUNT_VALID, MAX, MEAN, MIN, SUM, SUM0, _compare, _run

AGGREGATIONS = [(SUM, "$1"), (SUM0, "$2"), (MIN, "$1"), (MAX, "$2"), (COUNT_VALID, "$2"), (COUNT_ALL, ""), (MEAN, "$2"),
                (SUM, "*($2, 0.5)")]


def _table(n, groups, late, null_frac):
    rng = np.random.default_rng(groups)
    key = rng.integers(0, groups, n)
    if late:  # the first rows hold two groups only
        key[: n * 3 // 4] %= 2
    valid = pack_validity(rng.random(n) >= null_frac) if null_frac else None
    return [HostColumn(T.INT32, key.astype(np.int32) * 7 - 3), HostColumn(T.INT64, rng.integers(-(1 << 50), 1 << 50, n)),
            HostColumn(T.FLOAT64, rng.integers(-10**6, 10**6, n) / 8.0, valid)]


@pytest.mark.gpu
@pytest.mark.parametrize("groups", [1, 31, 32, 33, 64, 2557, 9000])
@pytest.mark.parametrize("late", [False, True])
@pytest.mark.parametrize("null_frac", [0.0, 0.3])
def test_group_counts(groups, late, null_frac):
    cols = _table(120_011, groups, late, null_frac)
    for keys, condition in (([0], None), ([0], "<($1, 0)"), ([], None)):
        got = _run(cols, condition, keys, AGGREGATIONS)
        _compare(got, agg_ref.filter_aggregate(cols, condition, keys, AGGREGATIONS), len(keys),
                 f"{groups} groups late={late} {condition} {keys}")
