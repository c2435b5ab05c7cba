"""Divisions whose divisor is past the reciprocal table or whose integer operand
has more than 53 significant bits."""
import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T
from helpers import OracleEngine, assert_tables_equal


@pytest.mark.gpu
@pytest.mark.parametrize("expression", ["/($0, $1)", "/(CAST($2):DOUBLE, $1)", "/(CAST($2):DOUBLE, CAST($1):DOUBLE)",
                                        "/(CAST($2):DOUBLE, 7.0)", "/($0, CAST($2):DOUBLE)"])
def test_large_divisors(expression):
    import blazingsql_gb300 as g
    rng = np.random.default_rng(3)
    n = 50_021
    k = np.exp(rng.uniform(0, np.log(2.0**62), n)).astype(np.int64) * rng.choice([1, -1], n)
    cols = [HostColumn(T.FLOAT64, rng.normal(0, 1, n) * 2.0 ** rng.integers(-1060, 1000, n)), HostColumn(T.INT64, k),
            HostColumn(T.INT64, rng.integers(-(1 << 63), 1 << 63, n, dtype=np.int64) | 1)]
    got = [c.to_host() for c in g.evaluate_expressions(cols, [expression])]
    assert_tables_equal(got, OracleEngine(2).evaluate_expressions(cols, [expression]), what=expression)
