"""The aggregation kernel's own block shapes: calls on both sides of the row count
from which blocks have 32 warps, plans on both sides of the 20 accumulators from
which they have 16, key widths on both sides of 16 bits (how the shared memory is
shared out, and the groups that the first split has room for), few groups to more
than the block's table holds."""
import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T, pack_validity
from oracle import agg_ref
from test_aggregate import COUNT_ALL, MAX, MEAN, MIN, SUM, _compare, _run

LARGE = 1 << 19
INPUTS = [(k, f"${c}") for c in range(2, 9) for k in (SUM, MIN, MAX)]
AGGREGATIONS = {"few": [(SUM, "$2"), (MEAN, "$3"), (COUNT_ALL, "")], "19": INPUTS[:19], "20": INPUTS[:20],
                "21": INPUTS + [(COUNT_ALL, "")]}


@pytest.mark.gpu
@pytest.mark.parametrize("aggs,rows,groups", [
    ("few", LARGE - 1, 20), ("few", LARGE, 21), ("19", LARGE, 6), ("20", LARGE - 1, 9000), ("20", LARGE, 20),
    ("21", LARGE, 9000), ("21", LARGE - 1, 100)])
def test_shapes(aggs, rows, groups):
    rng = np.random.default_rng(groups)
    key = rng.integers(0, groups, rows)
    values = rng.integers(-(1 << 20), 1 << 20, (7, rows))
    cols = [HostColumn(T.INT16, key.astype(np.int16)), HostColumn(T.INT64, key * 0x123456789ABC)]
    cols += [HostColumn(T.INT64, v, pack_validity(rng.random(rows) >= 0.1) if i % 2 else None) for i, v in enumerate(values)]
    for keys in ([0], [1]):
        _compare(_run(cols, ">($2, -1000000)", keys, AGGREGATIONS[aggs]),
                 agg_ref.filter_aggregate(cols, ">($2, -1000000)", keys, AGGREGATIONS[aggs]), 1,
                 f"{aggs} {rows} {groups} {keys}")
