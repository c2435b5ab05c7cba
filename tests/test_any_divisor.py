"""Divisions whose divisor is past the reciprocal table or whose integer operand
has more than 53 significant bits, and divisions of NaNs, whose sign and payload
the quotient keeps (MIN and MAX order doubles by their bits)."""
import os
import subprocess

import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T
from helpers import OracleEngine, assert_tables_equal

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("seed", [1, 2])
def test_same_bits_as_the_general_division(tmp_path, seed):
    out = str(tmp_path / "fp64emu_any_divisor")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "blazingsql_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "fp64emu_any_divisor.cpp"), "-o", out], check=True)
    r = subprocess.run([out, "1000000", str(seed)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[-2000:]


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


@pytest.mark.gpu
def test_a_nan_keeps_its_sign_and_payload():
    import blazingsql_gb300 as g
    nans = np.array([0x7FF8000000000000, 0xFFF8000000000000, 0x7FF8000000000123, 0xFFF0000000000001, 0xFFFFFFFFFFFFFFFF],
                    dtype=np.uint64)
    cols = [HostColumn(T.FLOAT64, nans.view(np.float64)), HostColumn(T.INT64, np.array([3, 5000, -3, -70000, 1 << 60]))]
    for expression in ("/($0, 7.0)", "/($0, -3.0)", "/($0, $1)"):
        got = g.evaluate_expressions(cols, [expression])[0].to_host().data.view(np.uint64)
        assert [hex(int(v)) for v in got] == [hex(int(v) | 1 << 51) for v in nans], expression
