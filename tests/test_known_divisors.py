"""Divisions by literals and integers, rounding, conversions, compares with
literals and DATE parts, which plans compute on the integer pipes: bit for bit
IEEE on the host, and against the oracle on the GPU at the operands where the
fast forms end (53 significant bits, the reciprocal table's last entry,
subnormals, infinities, zeros, the 32-bit ranges)."""
import os
import subprocess

import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T, pack_validity
from helpers import OracleEngine, assert_tables_equal

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("native") / "fp64emu_known_divisor")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "blazingsql_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "fp64emu_known_divisor.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("seed", [1, 2])
def test_known_divisor_routines_bit_exact(checker, seed):
    r = subprocess.run([checker, "500000", str(seed)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[-2000:]


INTEGERS = [0, 1, -1, 2, 3, 7, 997, 1023, 1024, 1025, -1024, -1025, (1 << 31) - 1, 1 << 31, -(1 << 31), (1 << 53) - 1,
            1 << 53, (1 << 53) + 1, -(1 << 53) - 1, (1 << 62) + 1, (1 << 63) - 1, -(1 << 63)]
DOUBLES = [0.0, -0.0, 0.5, -0.5, 2.5, -2.5, 1.005, 1e-310, -5e-324, 2.2250738585072014e-308, 1.7976931348623157e308,
           float("inf"), float("-inf"), float("nan"), 9007199254740993.0, 4503599627370495.5, 100.0, -300.0]
DAYS = [0, 1, -1, 59, 60, -719468, -719469, 11016, 11017, (1 << 30) - 1, 1 << 30, -(1 << 30), -(1 << 30) - 1,
        (1 << 31) - 1, -(1 << 31)]


def _table():
    pairs = [(i, k, d, t) for i in INTEGERS for k in INTEGERS for d in DOUBLES for t in DAYS[:1]]
    pairs += [(7, 3, 1.5, t) for t in DAYS]
    i, k, d, t = (np.array(c) for c in zip(*pairs))
    n = len(i)
    small = np.clip(k, -(1 << 31), (1 << 31) - 1)
    return [HostColumn(T.INT64, i.astype(np.int64)), HostColumn(T.INT64, k.astype(np.int64)),
            HostColumn(T.FLOAT64, d.astype(np.float64), pack_validity(np.arange(n) % 11 != 3)),
            HostColumn(T.INT32, small.astype(np.int32)), HostColumn(T.TIMESTAMP_DAYS, t.astype(np.int32))]


EXPRESSIONS = ["/($2, 100.0)", "/($2, -3)", "/($2, 1e300)", "/($2, 1e-300)", "/(CAST($0):DOUBLE, 10.0)", "/($2, $1)",
               "/($2, CAST($3):DOUBLE)", "/(CAST($0):DOUBLE, CAST($1):DOUBLE)", "/(CAST($0):DOUBLE, $3)",
               "/(CAST($3):DOUBLE, 7.0)", "ROUND($2, 2)", "ROUND($2)", "ROUND($2, -2)", "CAST($3):DOUBLE",
               "+($2, $0)", "*($2, MOD($0, 1000))", "MOD($3, 997)", "MOD(MOD($0, 50000), MOD($1, 1000))",
               "<($2, 0.5)", "<=($2, -0.5)", ">($2, 0.0)", ">=($2, 0.0)", "<($2, 0.0)", "<=($2, 0.0)", "=($2, 0.0)",
               "<>($2, 100.0)", ">($2, -300.0)", ">=($2, -300.0)", "BL_YEAR($4)", "BL_MONTH($4)", "BL_DAY($4)"]


@pytest.mark.gpu
@pytest.mark.parametrize("expression", EXPRESSIONS)
def test_expression_at_the_limits(expression):
    import blazingsql_gb300 as g
    cols = _table()
    got = [c.to_host() for c in g.evaluate_expressions(cols, [expression])]
    assert_tables_equal(got, OracleEngine(2).evaluate_expressions(cols, [expression]), what=expression)
