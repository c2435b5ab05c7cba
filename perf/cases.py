"""Work that a program has the evaluator do, as cases that can be timed.

Each case is one call (or one queue of calls) of a public entry point over
columns that are resident on the GPU, as an execution graph's Filter and
Projection steps issue them.  Tables, plans and value distributions are those
of ``blazingsql_gb300.workloads``; sizes run from one small batch to more than
a hundred million rows, most of them odd.

Kinds:

plan        a compiled plan over one small batch, into buffers that the program
            keeps (the execution graph's many small batches: latency counts)
filter      ``filter_project``: a Filter -> Projection pair in one call, on the
            C1 (light), C2 (deep, NULLs everywhere) or C5 (order-line) table
rows        ``process_filter``: every column of a table compacted (the filter
            that follows an inequality join)
project     ``evaluate_expressions``: a projection without a filter, with
            arithmetic, MOD, CASE, a date part and ROUND
batches     the batch runner over a table of log-uniform batches
learned     a queue of batches through the learner that orders the conjuncts
aggregate   filter + group-by in one call: a few groups (two flag columns) or
            thousands (a date column); the groups are then ordered by their
            keys, as ORDER BY does, because they come in no order of their own
strings     filter + projection over a table with two string columns
"""
from __future__ import annotations

import math

import numpy as np
import torch

import blazingsql_gb300 as g
from blazingsql_gb300 import _native as N
from blazingsql_gb300 import workloads as W
from blazingsql_gb300.api import DeviceColumn
from blazingsql_gb300.types import TypeId as T, np_dtype

DAY0 = W.DAY_1992_01_01
DAYS = W.DAYS_7Y


def listed():
    return [
        # one small batch of a streaming query: launch and host latency
        {"name": "plan_tiny", "kind": "plan", "table": "c1", "rows": 1031, "cut": 500000},
        # an ordinary partition of a selective scan
        {"name": "plan_small", "kind": "plan", "table": "c5", "rows": 100003, "cut": 2436},
        # a light plan over one ordinary batch
        {"name": "filter_light", "kind": "filter", "table": "c1", "rows": 1 << 24, "cut": 500000},
        # a deep expression over nullable columns, exact binary64 arithmetic
        {"name": "filter_deep", "kind": "filter", "table": "c2", "rows": (1 << 26) + 7, "cut": 1826},
        # a wide scan of an order-line table that keeps nearly every row
        {"name": "filter_orderline", "kind": "filter", "table": "c5", "rows": (1 << 27) - 5, "cut": 2436},
        # compaction of a joined batch's columns, NULLs included
        {"name": "rows_join", "kind": "rows", "table": "c2", "rows": (1 << 23) + 77},
        # a projection of every row
        {"name": "project_every", "kind": "project", "table": "c2", "rows": (1 << 25) + 1},
        # the batched graph: small and large batches of one plan
        {"name": "batches_deep", "kind": "batches", "table": "c2", "count": 96, "most": 1 << 22, "cut": 1826},
        # conjuncts whose selectivity moves from batch to batch
        {"name": "learned_queue", "kind": "learned", "count": 8, "rows": (1 << 23) - 3},
        # pricing summary: few groups, nine aggregations
        {"name": "aggregate_flags", "kind": "aggregate", "keys": "flags", "rows": (1 << 26) + 3, "cut": 2436},
        # a daily report: thousands of groups
        {"name": "aggregate_dates", "kind": "aggregate", "keys": "dates", "rows": (1 << 24) + 1, "cut": 2557},
        # a text predicate and string outputs
        {"name": "strings_comment", "kind": "strings", "rows": (1 << 23) + 9, "cut": 2436},
    ]


def draw(rng):
    def rows(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kind = rng.choice(["plan", "filter", "filter", "filter", "rows", "project", "batches", "learned", "aggregate",
                       "aggregate", "strings"])
    if kind == "plan":
        table = rng.choice(["c1", "c2", "c5"])
        cut = rng.randrange(100000, 900001) if table == "c1" else rng.randrange(256, DAYS + 1)
        return {"kind": kind, "table": table, "rows": rows(1, 1 << 20), "cut": cut}
    if kind == "filter":
        table = rng.choice(["c1", "c2", "c5"])
        cut = rng.randrange(100000, 900001) if table == "c1" else rng.randrange(256, DAYS + 1)
        return {"kind": kind, "table": table, "rows": rows(1 << 20, {"c1": 1 << 25, "c2": 1 << 26, "c5": 1 << 27}[table]),
                "cut": cut}
    if kind == "rows":
        return {"kind": kind, "table": "c2", "rows": rows(1 << 18, 1 << 25)}
    if kind == "project":
        return {"kind": kind, "table": "c2", "rows": rows(1 << 18, 1 << 25)}
    if kind == "batches":
        return {"kind": kind, "table": "c2", "count": rng.randrange(16, 97), "most": rows(1 << 14, 1 << 22),
                "cut": rng.randrange(256, DAYS + 1)}
    if kind == "learned":
        return {"kind": kind, "count": rng.randrange(5, 9), "rows": rows(1 << 19, 1 << 23)}
    if kind == "aggregate":
        keys = rng.choice(["flags", "dates"])
        return {"kind": kind, "keys": keys, "rows": rows(1 << 16, 1 << 26 if keys == "flags" else 1 << 24),
                "cut": rng.randrange(256, DAYS + 1)}
    return {"kind": kind, "rows": rows(1 << 16, 1 << 23), "cut": rng.randrange(256, DAYS + 1)}


# ------------------------------------------------------------------ the plans
def _date(cut):
    return str(np.datetime64("1992-01-01") + np.timedelta64(cut, "D"))


def _condition(case):
    table = case.get("table", "c5")
    if table == "c1":
        return "AND(>($0, %d), <($1, 0.5))" % case["cut"]
    if table == "c2":
        return "AND(IS NOT NULL($2), <=($4, %s))" % _date(case["cut"])
    return "<=($4, %s)" % _date(case["cut"])


PROJECTIONS = {"c1": W.C1_PROJECTIONS, "c2": W.C2_PROJECTIONS, "c5": W.C5_PROJECTIONS}
ROWS_QUERY = "LogicalFilter(condition=[>($1, $0)])"
PROJECT = ["+(*($2, 0.9), $3)", "MOD($0, 1000)", "CASE(>($5, 2), $2, $3)", "BL_YEAR($4)", "ROUND($2, 2)"]
LEARNED_OUT = ["$3", "$7"]  # the carried columns, which no conjunct tests
# (kind, input): 0 SUM, 5 COUNT(*), 6 MEAN
DATE_AGGREGATIONS = [(0, "$1"), (5, ""), (6, "/(CAST($2):DOUBLE, 100.0)"), (0, "/(CAST($1):DOUBLE, CAST($0):DOUBLE)")]
STRING_PROJECTIONS = ["$7", "SUBSTRING($8, 1, 10)", "CONCAT($7, '-', CAST($0):VARCHAR)",
                      "*(*($1, -(100, $2)), +(100, $3))"]


def _batch_sizes(case):
    """Log-uniform sizes from 1K rows, the same for every seed."""
    return W.c3_batch_sizes(seed=case["count"], nbatches=case["count"], lo=1024, hi=case["most"])


# ------------------------------------------------------------------ inputs
# The rows that a condition keeps are as many for every seed: the columns that
# it reads hold one table's values (drawn once per case) in an order of the
# seed's, and the other columns hold the seed's own values.
TABLE_SEED = 11
CONDITION_COLUMNS = {"c1": (0, 1), "c2": (0, 1, 2, 4), "c5": (4,)}


def _bits(mask, count):
    words = mask.view(torch.int32)
    bit = (words[:, None] >> torch.arange(32, device="cuda", dtype=torch.int32)[None, :]) & 1
    return bit.reshape(-1)[:count].bool()


def _packed(valid):
    words = max(16, ((valid.numel() + 31) // 32 + 15) // 16 * 16)
    room = torch.zeros(words * 32, dtype=torch.bool, device="cuda")
    room[:valid.numel()] = valid
    byte = (room.view(-1, 8) * torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], dtype=torch.uint8, device="cuda")).sum(1)
    return byte.to(torch.uint8)


def _reordered(col, order):
    data = col.data.view(_TORCH[int(col.type_id)])[order].view(torch.uint8)
    mask = None if col.mask is None else _packed(_bits(col.mask, col.size)[order])
    return DeviceColumn(col.type_id, data, mask, 0, col.size)


def _order(rows, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return torch.randperm(rows, generator=gen, device="cuda")


def _numbers(name, rows, seed):
    cols = W.device_columns(name, rows, seed=seed)
    order = _order(rows, seed)
    base = W.device_columns(name, rows, seed=TABLE_SEED)
    for i in CONDITION_COLUMNS[name]:
        cols[i] = _reordered(base[i], order)
    return cols


def _skewed(rows, seed, batch):
    base = W.c4_batch_device(rows, TABLE_SEED, batch)
    order = _order(rows, seed * 1000 + batch)
    cols = [_reordered(c, order) for c in base]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 1000 + batch)
    carried = torch.randint(0, 1 << 30, (rows,), generator=gen, device="cuda")
    cols[3] = DeviceColumn(T.INT64, carried.view(torch.uint8), None, 0, rows)
    carried = torch.rand(rows, generator=gen, device="cuda", dtype=torch.float64) * 1e6
    cols[7] = DeviceColumn(T.FLOAT64, carried.view(torch.uint8), None, 0, rows)
    return cols


def _text_column(ids, phrases):
    width = max(len(p) for p in phrases)
    tab = torch.zeros((len(phrases), width), dtype=torch.uint8)
    for i, p in enumerate(phrases):
        tab[i, :len(p)] = torch.tensor(list(p.encode()), dtype=torch.uint8)
    tab = tab.to("cuda")
    lens = torch.tensor([len(p) for p in phrases], dtype=torch.int32, device="cuda")[ids]
    offs = torch.zeros(ids.numel() + 1, dtype=torch.int32, device="cuda")
    offs[1:] = torch.cumsum(lens, 0, dtype=torch.int32)
    keep = torch.arange(width, device="cuda", dtype=torch.int32)[None, :] < lens[:, None]
    return DeviceColumn(T.STRING, torch.masked_select(tab[ids], keep), None, 0, ids.numel(), offs)


def _texts(rows, seed):
    """The order-line columns, a mode column (7 short tokens) and a comment
    column (10 to 43 characters of random words); every column is reordered, so
    the outputs have as many characters for every seed."""
    rng = np.random.default_rng(TABLE_SEED)
    letters = np.array(list("abcdefghijklmnopqrstuvwxyz"))
    words = ["".join(rng.choice(letters, int(rng.integers(3, 10)))) for _ in range(200)]
    comments = []
    while len(comments) < 512:
        phrase, target = "", int(rng.integers(10, 44))
        while len(phrase) < target:
            phrase = (phrase + " " + words[int(rng.integers(0, len(words)))]).strip()
        comments.append(phrase[:target].strip() or "x")
    modes = ["".join(rng.choice(letters, int(rng.integers(3, 8)))).upper() for _ in range(7)]
    order = _order(rows, seed)
    cols = [_reordered(c, order) for c in W.device_columns("c5", rows, seed=TABLE_SEED)]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(TABLE_SEED)
    for phrases in (modes, comments):
        ids = torch.randint(0, len(phrases), (rows,), generator=gen, device="cuda")
        cols.append(_text_column(ids[order], phrases))
    return cols


def _table(case, seed):
    kind = case["kind"]
    if kind == "learned":
        return [_skewed(case["rows"], seed, b) for b in range(case["count"])]
    if kind == "strings":
        return _texts(case["rows"], seed)
    if kind in ("batches", "aggregate", "project"):  # their outputs have one shape whatever the values
        rows = sum(_batch_sizes(case)) if kind == "batches" else case["rows"]
        return W.device_columns(case.get("table", "c5"), rows, seed=seed)
    return _numbers(case["table"], case["rows"], seed)


def _buffers(types, rows):
    """Output buffers: (data tensor, mask tensor) per column, room for `rows` rows."""
    words = max(16, ((rows + 31) // 32 + 15) // 16 * 16)
    return [(torch.zeros(max(rows, 1), dtype=_TORCH[int(t)], device="cuda"),
             torch.zeros(words, dtype=torch.int32, device="cuda")) for t in types]


def prepare(case, seed):
    kind = case["kind"]
    cols = _table(case, seed)
    state = {"case": case, "cols": cols}
    if kind == "plan":
        w = W.workload(case["table"])
        state["plan"] = g.Plan(w.schema, _condition(case), PROJECTIONS[case["table"]], nullable=w.nullable)
        state["buffers"] = _buffers(state["plan"].output_types(), case["rows"])
        state["out"] = [N.Column(int(t), 0, d.data_ptr(), m.data_ptr(), 0, case["rows"])
                        for t, (d, m) in zip(state["plan"].output_types(), state["buffers"])]
    elif kind == "batches":
        w = W.workload("c2")
        sizes = _batch_sizes(case)
        plan = g.Plan(w.schema, _condition(case), PROJECTIONS["c2"], nullable=w.nullable)
        state["plan"] = plan
        state["runner"] = g.BatchRunner(plan, max_batches=len(sizes), max_total_rows=sum(sizes))
        state["bound"] = state["runner"].bind(W.slice_batches(cols, sizes))
        # every batch writes its own slot of one buffer per column; slots start at multiples of 512 rows
        types = plan.output_types()
        starts = np.concatenate([[0], np.cumsum([(n + 511) // 512 * 512 for n in sizes])])
        state["buffers"] = _buffers(types, int(starts[-1]))
        state["out"] = [N.Column(int(t), 0, d.data_ptr() + int(s) * d.element_size(), m.data_ptr() + int(s) // 8, 0, n)
                        for s, n in zip(starts, sizes) for t, (d, m) in zip(types, state["buffers"])]
    elif kind == "learned":
        state["plan"] = g.Plan([T.INT64] * 4 + [T.FLOAT64] * 4, W.C4_CONDITION, LEARNED_OUT, nullable=[False] * 8)
        state["learner"] = g.Learner(state["plan"], warmup_batches=4, relabel_every=0, fast_words_per_warp=8,
                                     size_outputs=0)
        state["queue"] = state["learner"].queue_args(cols)
    return state


# ------------------------------------------------------------------ outputs
_TORCH = {int(T.INT8): torch.int8, int(T.INT16): torch.int16, int(T.INT32): torch.int32, int(T.INT64): torch.int64,
          int(T.FLOAT32): torch.float32, int(T.FLOAT64): torch.float64, int(T.BOOL8): torch.uint8,
          int(T.TIMESTAMP_DAYS): torch.int32}


class _Memory:
    """Device memory of an output column, as torch reads it (no copy); it keeps the column."""

    def __init__(self, column, pointer, count, typestr):
        self.column = column
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (pointer, False), "version": 2}


def _tensor(column, pointer, count, typestr):
    return torch.as_tensor(_Memory(column, pointer, count, typestr), device="cuda")


def _columns(columns):
    """[data, validity words] of each column; a string column's data are its offsets and characters."""
    out = []
    for c in columns:
        n = c.size
        mask = _tensor(c, c.mask_ptr, (n + 31) // 32, "<i4")
        if c.type_id == T.STRING:
            out.append([_tensor(c, c.view().string_offsets, n + 1, "<i4"),
                        _tensor(c, c.data_ptr, int(c._c.string_bytes), "|u1"), mask])
        else:
            out.append([_tensor(c, c.data_ptr, n, np_dtype(c.type_id).str), mask])
    return out


def _ordered(columns, keys):
    """Groups ordered by their keys (none of the columns holds a NULL)."""
    out = _columns(columns)
    order = out[0][0].to(torch.int64)
    if keys == "flags":
        order = order * 2 + out[1][0]
    order = torch.argsort(order)
    return [[data[order], mask] for data, mask in out]


def run(state):
    case, cols = state["case"], state["cols"]
    kind = case["kind"]
    if kind == "plan":
        _, rows = state["plan"].execute(cols, out=state["out"])
        return [[d[:rows], m[:(rows + 31) // 32]] for d, m in state["buffers"]]
    if kind == "filter":
        return _columns(g.filter_project(cols, _condition(case), PROJECTIONS[case["table"]]))
    if kind == "rows":
        return _columns(g.process_filter(cols, ROWS_QUERY))
    if kind == "project":
        return _columns(g.evaluate_expressions(cols, PROJECT))
    if kind == "batches":
        _, rows = state["runner"].run(state["bound"], out=state["out"], raw=True)
        return [state["buffers"], np.array(rows)]
    if kind == "learned":
        state["learner"].run_queue(state["queue"])
        return [_columns(c) for c, _, _ in state["learner"].queue_results(state["queue"])]
    if kind == "aggregate":
        keys, aggs = ([5, 6], W.C5_AGGREGATIONS) if case["keys"] == "flags" else ([4], DATE_AGGREGATIONS)
        return _ordered(g.filter_aggregate(cols, _condition(case), keys, aggs)[0], case["keys"])
    condition = "AND(<=($4, %s), NOT(LIKE($8, '%%ke%%q%%')))" % _date(case["cut"])
    return _columns(g.filter_project(cols, condition, STRING_PROJECTIONS))


# ------------------------------------------------------------------ compulsory work
def _width(name):
    return W.workload(name).in_bytes_per_row


def work(case):
    kind = case["kind"]
    share = min(1.0, (case.get("cut", 0) + 1) / DAYS)
    if kind in ("plan", "filter"):
        w = W.workload(case["table"])
        kept = {"c1": (1 - case["cut"] / 1e6) * 0.6915, "c2": 0.9025 * share, "c5": share}[case["table"]]
        per_row = {"c1": 4, "c2": 24, "c5": 8}[case["table"]]
        return {"bytes": case["rows"] * (w.in_bytes_per_row + kept * w.out_bytes_per_row), "flops": case["rows"] * per_row}
    if kind == "rows":
        return {"bytes": case["rows"] * _width("c2") * 1.45, "flops": case["rows"]}
    if kind == "project":
        return {"bytes": case["rows"] * (_width("c2") - 8 - 1 / 8 + 40 + 5 / 8), "flops": case["rows"] * 20}
    if kind == "batches":
        rows = sum(_batch_sizes(case))
        return {"bytes": rows * (_width("c2") + 0.9025 * share * (16 + 1 / 4)), "flops": rows * 24}
    if kind == "learned":
        return {"bytes": case["count"] * case["rows"] * 48.0, "flops": case["count"] * case["rows"] * 6}
    if kind == "aggregate":
        return {"bytes": case["rows"] * (_width("c5") if case["keys"] == "flags" else 24.0), "flops": case["rows"] * 12}
    # 28 fixed bytes, 8 of offsets and about 32 characters in; about 40 bytes a kept row out
    return {"bytes": case["rows"] * (28 + 8 + 32 + 40 * share), "flops": case["rows"] * 40}


# ------------------------------------------------------------------ 64-bit results
def _value(col):
    return col.data.view(_TORCH[int(col.type_id)])[col.offset:col.offset + col.size]


def _valid(col):
    if col.mask is None:
        return torch.ones(col.size, dtype=torch.bool, device="cuda")
    return _bits(col.mask, col.offset + col.size)[col.offset:]


# Data under a NULL are what the operators make of the data under their
# operands' NULLs, except that a NULL branch of a CASE reads as 0.
def _light(cols, cut):
    a, b, c = (_value(x) for x in cols)
    keep = (a > cut) & (b < 0.5)
    return [[None, None], [b[keep] / c[keep].double(), None]]


def _deep(cols, cut):
    keep = _valid(cols[2]) & _valid(cols[4]) & (_value(cols[4]) <= DAY0 + cut)
    d0, d1, d2, d3, _, d5 = (_value(c)[keep] for c in cols)
    v0, v1, _, v3, _, v5 = (_valid(c)[keep] for c in cols)
    log = torch.floor(torch.log(d2.abs() + 1.0))
    left = torch.fmod(torch.where(v0, d0, d1), 997).double()
    near = torch.where(v0 & v1, d3 - torch.fmod((d1 - d0).abs(), 1000).double(), 0.0)
    rest = left + torch.floor(torch.where(v3, near, d2) / 10.0) * d5.double()
    zero = torch.where(v3, torch.exp(d3 / 1000.0), 0.0)
    return [[torch.where(~v5, log, torch.where(d5 == 0, zero, rest)), None], [None, None]]


def _orderline(cols, cut):
    q, price, disc, _, ship = (_value(c) for c in cols[:5])
    keep = ship <= DAY0 + cut
    return [[None, None], [price[keep].double() / q[keep].double(), None], [disc[keep].double() / 100.0, None],
            [None, None], [None, None]]


def _groups(cols, case):
    q, price, disc, _, ship, f1, f2 = (_value(c) for c in cols[:7])
    keep = ship <= DAY0 + case["cut"]
    key = (f1.long() * 2 + f2.long() if case["keys"] == "flags" else ship.long())[keep]
    _, where = torch.unique(key, return_inverse=True)
    groups = int(where.max()) + 1
    count = torch.bincount(where, minlength=groups).double()
    unit = price[keep].double() / q[keep].double()
    rate = disc[keep].double() / 100.0

    def total(v):
        # by parts, so that the sums of a few large groups do not lose digits
        parts = torch.zeros((groups, 4096 if groups < 64 else 16), dtype=torch.float64, device="cuda")
        lane = torch.arange(v.numel(), device="cuda") % parts.shape[1]
        parts.view(-1).index_add_(0, where * parts.shape[1] + lane, v)
        return parts.sum(1)

    none = [None, None]
    if case["keys"] == "flags":
        top = torch.full((groups,), -math.inf, dtype=torch.float64, device="cuda").scatter_reduce(0, where, unit, "amax")
        return [none, none, none, none, none, [total(unit), None], [total(q[keep].double()) / count, None],
                [total(rate) / count, None], none, none, [top, None]]
    return [none, none, none, [total(rate) / count, None], [total(unit), None]]


def _conjuncts(cols):
    v = [_value(c) for c in cols]
    keep = (v[0] > 100000) & (v[1] == 1000) & (v[2] < 1000) & (v[4] < 1000.0) & (v[5] > 5000.0) & (v[6] < 100.0)
    return [[None, None], [v[7][keep], None]]


def exact(case, seed):
    cols, kind = _table(case, seed), case["kind"]
    if kind in ("plan", "filter"):
        return {"c1": _light, "c2": _deep, "c5": _orderline}[case["table"]](cols, case["cut"])
    if kind == "rows":
        keep = _valid(cols[0]) & _valid(cols[1]) & (_value(cols[1]) > _value(cols[0]))
        return [[_value(c)[keep] if c.type_id == T.FLOAT64 else None, None] for c in cols]
    if kind == "project":
        d2, d3 = _value(cols[2]), _value(cols[3])
        scaled = d2 * 100.0
        near = torch.trunc(scaled) + torch.where((scaled - torch.trunc(scaled)).abs() >= 0.5, torch.sign(scaled), 0.0)
        return [[d2 * 0.9 + d3, None], [None, None], [None, None], [None, None], [near / 100.0, None]]
    if kind == "batches":
        outs, start = None, 0
        for n in _batch_sizes(case):
            part = [DeviceColumn(c.type_id, c.data, c.mask, start, n) for c in cols]
            value = _deep(part, case["cut"])[0][0]
            room = torch.zeros((n + 511) // 512 * 512, dtype=torch.float64, device="cuda")
            room[:value.numel()] = value
            outs = [room] if outs is None else outs + [room]
            start += n
        return [[[torch.cat(outs), None], [None, None]], None]
    if kind == "learned":
        return [_conjuncts(c) for c in cols]
    if kind == "aggregate":
        return _groups(cols, case)
    return None  # strings and whole numbers only
