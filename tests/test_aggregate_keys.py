"""Group keys as the aggregation kernel keeps them in shared memory: packed into
one word where the keys' widths and null bits leave room (at most 63 bits), as
separate words where they do not, over key types of each width and sign, their
smallest and largest values, NULL keys, and few groups (warp accumulators), many
(the block's table) and more than the table holds."""
import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T, np_dtype, pack_validity
from oracle import agg_ref
from test_aggregate import COUNT_ALL, MAX, MIN, SUM, _compare, _run

KEYS = {
    "one byte": [T.INT8], "unsigned": [T.UINT32], "bool": [T.BOOL8], "date": [T.TIMESTAMP_DAYS],
    "59 bits": [T.INT32, T.INT16, T.UINT8], "48 + 4 bits": [T.INT16, T.UINT16, T.INT8, T.INT8],
    "62 bits, 5 keys": [T.INT16, T.INT16, T.INT8, T.UINT8, T.BOOL8],
    "66 bits": [T.INT32, T.INT32], "64 bits": [T.INT64], "wide and narrow": [T.INT64, T.INT8],
}


def _key(rng, t, n, groups):
    dt = np_dtype(t)
    if t == T.BOOL8:
        return rng.integers(0, 2, n).astype(dt)
    info = np.iinfo(dt)
    some = rng.integers(info.min, info.max, groups, dtype=dt, endpoint=True)  # any values of the type
    some[:2] = info.min, info.max
    dense = (np.arange(groups) + 8000).astype(dt)  # consecutive ones
    return rng.choice(np.concatenate([some[: groups // 2 + 2], dense[: groups // 2 + 1]]), n)


@pytest.mark.gpu
@pytest.mark.parametrize("groups", [3, 40, 3000, 20000])
@pytest.mark.parametrize("keys", list(KEYS))
def test_group_keys(keys, groups):
    rng = np.random.default_rng(groups)
    n = 60_013
    types = KEYS[keys]
    each = max(2, int(round(groups ** (1 / len(types)))))
    for null_frac in (0.0, 0.1):
        cols = [HostColumn(t, _key(rng, t, n, each), pack_validity(rng.random(n) >= null_frac) if null_frac else None)
                for t in types]
        cols.append(HostColumn(T.INT64, rng.integers(-(1 << 40), 1 << 40, n)))
        k, v = list(range(len(types))), f"${len(types)}"
        aggs = [(SUM, v), (MIN, v), (MAX, v), (COUNT_ALL, "")]
        got = _run(cols, f">({v}, -1000000000)", k, aggs)
        _compare(got, agg_ref.filter_aggregate(cols, f">({v}, -1000000000)", k, aggs), len(k), f"{keys} {groups} {null_frac}")
