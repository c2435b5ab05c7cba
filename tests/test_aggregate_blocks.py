"""The aggregation kernel in blocks of other sizes than its own 32 warps, as
GX_WARPS / GX_WORDS ask for: group counts on both sides of a one-warp block's
32 threads and of the 64 groups that have accumulators per warp, blocks whose
kept-row lists take much of the shared memory, with keys that pack into one word
and keys that do not."""
import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T
from oracle import agg_ref
from test_aggregate import COUNT_ALL, MAX, SUM, _compare, _run

AGGREGATIONS = [[(COUNT_ALL, "")], [(SUM, "$1"), (MAX, "$2")]]


def _table(n, groups):
    rng = np.random.default_rng(groups)
    key = rng.integers(0, groups, n)
    return [HostColumn(T.INT32, key.astype(np.int32) * 7 - 3), HostColumn(T.INT64, rng.integers(-(1 << 50), 1 << 50, n)),
            HostColumn(T.FLOAT64, rng.integers(-10**6, 10**6, n) / 8.0), HostColumn(T.INT64, key * (1 << 33))]


@pytest.mark.gpu
@pytest.mark.parametrize("groups", [1, 31, 32, 33, 63, 64, 65, 3000])
@pytest.mark.parametrize("shape", [(1, 4), (1, 8), (2, 4), (4, 8), (16, 8), (32, 16), (16, 32), (0, 0)], ids=str)
def test_group_counts_by_block(shape, groups, monkeypatch):
    if shape[0]:
        monkeypatch.setenv("GX_WARPS", str(shape[0]))
        monkeypatch.setenv("GX_WORDS", str(shape[1]))
    cols = _table(40_013, groups)
    for aggs in AGGREGATIONS:
        for keys, condition in (([0], None), ([3], "<($1, 0)"), ([0, 3], None)):
            got = _run(cols, condition, keys, aggs)
            _compare(got, agg_ref.filter_aggregate(cols, condition, keys, aggs), len(keys), f"{groups} {shape} {keys}")
