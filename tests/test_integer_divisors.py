"""Divisions by integers of any size, past the reciprocal table and past 53 bits
too, with quotients next to midpoints of two doubles: the same bits as the general
division's."""
import os
import subprocess

import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T
from helpers import OracleEngine, assert_tables_equal

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_same_bits_as_the_general_division(tmp_path, seed):
    out = str(tmp_path / "fp64emu_integer_divisor")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "blazingsql_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "fp64emu_integer_divisor.cpp"), "-o", out], check=True)
    r = subprocess.run([out, "1000000", str(seed)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[-2000:]


@pytest.mark.gpu
@pytest.mark.parametrize("expression", ["/($0, $1)", "/($0, $3)", "/(CAST($2):DOUBLE, $1)", "/(CAST($2):DOUBLE, $3)",
                                        "/(CAST($2):DOUBLE, 0.3)"])
def test_quotients(expression):
    import blazingsql_gb300 as g
    rng = np.random.default_rng(8)
    n = 40_009
    big = np.exp(rng.uniform(0, np.log(2.0**63), n)).astype(np.int64) * rng.choice([1, -1], n)
    big[:4] = [-(1 << 63), (1 << 63) - 1, (1 << 53) + 1, 1025]
    top = (1 << 63) - 1 - rng.integers(0, 4000, n)
    cols = [HostColumn(T.FLOAT64, rng.normal(0, 1, n) * 2.0 ** rng.integers(-1074, 1023, n)), HostColumn(T.INT64, big),
            HostColumn(T.INT64, np.where(rng.random(n) < 0.5, top, rng.integers(-(1 << 63), 1 << 63, n, dtype=np.int64))),
            HostColumn(T.INT32, rng.integers(1000, 1050, n).astype(np.int32))]
    got = [c.to_host() for c in g.evaluate_expressions(cols, [expression])]
    assert_tables_equal(got, OracleEngine(2).evaluate_expressions(cols, [expression]), what=expression)
    kept = [c.to_host() for c in g.filter_project(cols, "<($3, 1030)", [expression])]
    assert_tables_equal(kept, OracleEngine(2).filter_project(cols, "<($3, 1030)", [expression]), what=expression)
