"""The kept rows' projections and validity bits at the edges of a warp's words:
block shapes up to 32 words per warp (33 mask words at an odd position), views
that start at any bit of a validity word, conditions that keep every row, few
rows or whole words, columns the condition proves valid."""
import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T, pack_validity
from helpers import OracleEngine, assert_tables_equal

SCHEMA = [T.INT64, T.FLOAT64, T.INT32, T.INT8]
OUTPUTS = ["$0", "$1", "$2", "$3", "+($0, $2)", "*($1, 2.5)", "CASE(IS NULL($1), $0, $2)"]
CONDITIONS = ["IS NOT NULL($0)", "AND(>($2, 40), IS NOT NULL($1))", "=($3, 3)", ">=($2, -1000)",
              "OR(IS NULL($1), >($2, 0))"]


def _table(n):
    rng = np.random.default_rng(n)
    word = np.repeat(rng.integers(0, 4, n // 32 + 1), 32)[:n]  # whole words of one value
    data = [rng.integers(-(1 << 40), 1 << 40, n), rng.normal(0, 1e3, n), rng.integers(-50, 51, n).astype(np.int32),
            word.astype(np.int8)]
    null = [0.001, 0.3, 0.0, 0.0]
    return [HostColumn(t, d, pack_validity(rng.random(n) >= p) if p else None) for t, d, p in zip(SCHEMA, data, null)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 32), (4, 32), (1, 16), (4, 8), (2, 1)], ids=str)
@pytest.mark.parametrize("condition", CONDITIONS)
def test_kept_rows(shape, condition):
    import blazingsql_gb300 as g
    from blazingsql_gb300.api import DeviceColumn
    oracle = OracleEngine(2)
    for n in (1, 33, 1024, 8191, 40007):
        host = _table(n)
        device = [DeviceColumn.from_host(c) for c in host]
        for off in (0, 1, 31, 32, 77):
            if off >= n:
                continue
            views = [DeviceColumn(c.type_id, c.data, c.mask, off, n - off) for c in device]
            plan = g.Plan(SCHEMA, condition, OUTPUTS, block_threads=shape[0] * 32, words_per_warp=shape[1])
            got, rows = plan.execute(views)
            expected = oracle.filter_project([HostColumn(c.type_id, c.data, c.mask, off, n - off) for c in host],
                                             condition, OUTPUTS)
            assert_tables_equal([c.to_host() for c in got], expected, what=f"{condition} {shape} {n} rows from {off}")
