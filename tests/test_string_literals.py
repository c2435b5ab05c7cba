"""Literals and patterns of string operators on a stream that is busy with
earlier work: their host bytes live until they have been copied, also where the
call itself returns without waiting for its results."""
import numpy as np
import pytest

from blazingsql_gb300.types import HostColumn, TypeId as T


@pytest.mark.gpu
@pytest.mark.parametrize("length", [5, 300, 20_000, 90_000])
def test_literals_on_a_busy_stream(length):
    import torch

    import blazingsql_gb300 as g
    from blazingsql_gb300.api import DeviceColumn
    words = ["ab" * (k % 7) + "q" * k for k in range(40)]
    n = HostColumn(T.INT32, np.arange(40, dtype=np.int32))
    letters = "".join(chr(97 + i % 23) for i in range(length))
    m = torch.ones((4096, 4096), device="cuda")
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    for i in range(4):
        literal = letters[i:] + letters[:i]
        table = [DeviceColumn.from_strings(words), DeviceColumn.from_host(n)]
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            for _ in range(20):
                m = m @ m * 0.0 + 1.0
        pattern = "%" + literal[:40]
        got = g.evaluate_expressions(table, [f"LIKE($0, '{pattern}')", f"LIKE($0, '%{'q' * (i + 9)}')"],
                                     stream=stream.cuda_stream)
        made = g.evaluate_expressions(table, [f"CONCAT($0, '{literal}')", f"'{literal[::-1]}'"], stream=stream.cuda_stream)
        kept = g.filter_project(table, "<($1, 30)", [f"CONCAT('{literal}', $0, '{literal[:17]}')", f"REPLACE($0, 'q', '{literal[:50]}')"],
                                stream=stream.cuda_stream)
        stream.synchronize()
        assert [bool(v) for v in got[0].to_host().data[:40]] == [w.endswith(literal[:40]) for w in words]
        assert [bool(v) for v in got[1].to_host().data[:40]] == [w.endswith("q" * (i + 9)) for w in words]
        assert made[0].to_strings() == [w + literal for w in words]
        assert made[1].to_strings() == [literal[::-1]] * 40
        assert kept[0].to_strings() == [literal + w + literal[:17] for w in words[:30]]
        assert kept[1].to_strings() == [w.replace("q", literal[:50]) for w in words[:30]]
