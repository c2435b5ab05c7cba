"""A single 64-bit group key, held as one word in shared memory: every value of
the type is a key of its own, NULL another, also the two values whose words are
those of an empty place and of NULL (0x9E3779B97F4A7C15 and the one that differs
from it in the last bit), beside few groups and beside more than the block's
table holds."""
import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T, np_dtype, pack_validity
from oracle import agg_ref
from test_aggregate import COUNT_ALL, MAX, MIN, SUM, _compare, _run

EDGES = np.array([0x9E3779B97F4A7C15, 0x9E3779B97F4A7C14, 0x9E3779B97F4A7C16, 0, 1, 2**63, 2**64 - 1], dtype=np.uint64)


@pytest.mark.gpu
@pytest.mark.parametrize("groups", [0, 40, 3000, 20000])
@pytest.mark.parametrize("key", [T.INT64, T.UINT64, T.TIMESTAMP_NANOSECONDS], ids=["signed", "unsigned", "time"])
def test_edge_values(key, groups):
    rng = np.random.default_rng(groups)
    n = 60_013
    values = np.concatenate([EDGES, rng.integers(0, 2**64 - 1, groups, dtype=np.uint64)])
    data = rng.choice(values, n).view(np_dtype(key))
    for mask in (None, pack_validity(rng.random(n) >= 0.1)):
        cols = [HostColumn(key, data, mask), HostColumn(T.INT64, rng.integers(-(1 << 40), 1 << 40, n))]
        aggs = [(SUM, "$1"), (MIN, "$1"), (MAX, "$1"), (COUNT_ALL, "")]
        for condition in (None, ">($1, 0)"):
            _compare(_run(cols, condition, [0], aggs), agg_ref.filter_aggregate(cols, condition, [0], aggs), 1,
                     f"{groups} {condition} {mask is not None}")
