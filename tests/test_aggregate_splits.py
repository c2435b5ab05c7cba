"""Group counts around the splits of a warp's accumulators (few groups with many
replicas, more groups with fewer), from the first rows on or only late, with keys
that pack into one word and keys that do not."""
import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T
from oracle import agg_ref
from test_aggregate import _compare, _run
from test_aggregate_groups import AGGREGATIONS, _table


@pytest.mark.gpu
@pytest.mark.parametrize("groups", [*range(6, 26), 40])
@pytest.mark.parametrize("late", [False, True])
def test_splits(groups, late):
    cols = _table(50_021, groups, late, 0.1)
    wide = HostColumn(T.INT64, cols[0].data.astype(np.int64) * (1 << 33))
    for table, keys in ((cols, [0]), (cols + [wide], [0, 3])):
        got = _run(table, None, keys, AGGREGATIONS)
        _compare(got, agg_ref.filter_aggregate(table, None, keys, AGGREGATIONS), len(keys), f"{groups} late={late} {keys}")
