"""The string builder at the edges of its pieces: 32-row words and blocks of 64
of them, words whose characters fit the shared-memory stages (2 KB) and words
that pass them, rows of up to 40 words of 16 bytes, characters that are bytes and
characters that are not, rows in the order of a filter's row map, several
columns built in one call.  Bytes and offsets are compared exactly."""
import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T
from oracle import strings_ref

KINDS = {
    "ascii": lambda rng: "".join(map(chr, rng.integers(97, 123, rng.integers(0, 18)))),
    "sixteens": lambda rng: "x" * int(rng.choice([0, 1, 3, 4, 15, 16, 17, 31, 32, 33])),
    "long": lambda rng: "".join(map(chr, rng.integers(97, 123, rng.integers(60, 640)))),
    "accents": lambda rng: "".join(rng.choice(["a", "é", "日", "𝄞", "b"], rng.integers(0, 12))),
    "one accent": lambda rng: "é" if rng.random() < 0.02 else "plain text",
}
EXPRS = ["$0", "SUBSTRING($0, 1, 10)", "SUBSTRING($0, 3, 2)", "SUBSTRING($0, 17, 40)", "SUBSTRING($0, 1, 500)",
         "CONCAT($0, '-', CAST($1):VARCHAR)", "CONCAT($0, $2, $0)", "UPPER($0)", "$2"]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("n", [1, 31, 33, 2047, 2048, 2049, 4500])
def test_string_words(kind, n):
    import blazingsql_gb300 as g
    from blazingsql_gb300.api import DeviceColumn
    rng = np.random.default_rng(n)
    strings = {c: [None if rng.random() < p else KINDS[kind](rng) for _ in range(n)] for c, p in ((0, 0.1), (2, 0.0))}
    cols = [None, HostColumn(T.INT32, rng.integers(-10**6, 10**6, n).astype(np.int32)), None]
    dev = [DeviceColumn.from_strings(strings[c]) if c in strings else DeviceColumn.from_host(cols[c]) for c in range(3)]
    exp = strings_ref.evaluate_expressions(cols, strings, EXPRS)
    got = g.evaluate_expressions(dev, EXPRS)
    _same(got, exp, "all rows")
    for condition in (">($1, 0)", ">($1, 990000)", "<($1, 0)"):
        exp, rows = strings_ref.filter_project(cols, strings, condition, EXPRS)
        got = g.filter_project(dev, condition, EXPRS)
        assert got[0].size == rows
        _same(got, exp, condition)


def _same(got, exp, what):
    for k, (c, e) in enumerate(zip(got, exp)):
        assert c.to_strings() == list(e), f"{what}: {EXPRS[k]}"
