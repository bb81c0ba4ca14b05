"""The work whose speed is measured: operator plans as TQP-Inmem's executor runs them, each through
the drop-in operators of ``tqpk.operators`` over columns resident on the GPU.

A case is one plan over seeded tables of TPC-H's shapes and value distributions: int64 keys (sparse
order keys, eight of every 32, as TPC-H has them), int32 dates, float64 decimals with two digits,
uint8 flags, zero-padded int8 [N, w] text.  Every pass runs the whole plan, host work included.

  report         filter + eight aggregates over two flags + sort (the pricing summary)
  order_totals   two aggregates per order (one to seven lines each), then a filter over the groups
  part_supplier  one year's lines summed by (part, supplier): a sparse two-column key
  text_groups    text predicates, then groups by two text columns and a size, ordered by four keys
  join_orders    filtered orders x filtered lines on the order key, payload columns gathered
  join_two_key   lines x part suppliers: a repeated key and a second key as the join's condition
  join_exists    orders with a late line: the semi-join over a build side of repeated keys
  sort_full      a whole table ordered by price descending, then date
  take_top       two computed columns, then the 100 largest rows with an int64 tie-breaker
  fused_orders   filter, filter, join, aggregate, top 10 handed over as one run (try_fused)
  fused_star     the star plan, three joins, handed over as one run (try_fused)
"""
import math
import sys
from pathlib import Path

import torch

_ROOT = Path(__file__).resolve().parent.parent
if str(_ROOT / "tqp-inmem_gb300") not in sys.path:
    sys.path.insert(0, str(_ROOT / "tqp-inmem_gb300"))

DAYS = 2557                       # order and ship dates: days of seven years


# ---------------------------------------------------------------------------- the cases
def listed():
    return [
        # a small table (scale factor 0.01): launches, host work and synchronisations are the time
        {"name": "report_small", "kind": "report", "rows": 60175},
        # the pricing summary at scale factor 1: few groups, many aggregates
        {"name": "report_sf1", "kind": "report", "rows": 6001215},
        # as many groups as orders, from lines stored in order-key order
        {"name": "order_totals_sf1", "kind": "order_totals", "rows": 6001215, "orders": 1500000, "stored": True},
        # a key space far larger than the rows: the sparse group-by
        {"name": "part_supplier_sf1", "kind": "part_supplier", "rows": 6001215, "parts": 200000},
        # text filters, text group keys, text sort keys
        {"name": "text_groups_sf1", "kind": "text_groups", "rows": 800000},
        # primary-key join of the two largest tables, both filtered
        {"name": "join_orders_sf1", "kind": "join_orders", "rows": 6001215, "orders": 1500000, "stored": True,
         "type": "inner"},
        # a join whose build key repeats four times and whose second key is a condition
        {"name": "join_two_key_sf1", "kind": "join_two_key", "rows": 6001215, "parts": 200000},
        # exists(): a semi-join whose build side is the large table
        {"name": "join_exists_sf1", "kind": "join_exists", "rows": 6001215, "orders": 1500000},
        # order by without a limit
        {"name": "sort_full_sf1", "kind": "sort_full", "rows": 1500000},
        # order by with a limit, over computed columns
        {"name": "take_top_sf1", "kind": "take_top", "rows": 6001215, "limit": 100},
        # the fused join plan at the benchmark's size
        {"name": "fused_orders_sf1", "kind": "fused_orders", "rows": 6001215, "orders": 1500000, "limit": 10},
        # the fused star plan at the benchmark's size: the largest call
        {"name": "fused_star_sf10", "kind": "fused_star", "rows": 59986052, "limit": 100},
    ]


def _log_size(rng, lo, hi):
    """A size spread evenly over its logarithm, odd ones among them."""
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(sorted(_KINDS))
    n = _log_size(rng, 2000, 59986052 if kind == "fused_star" else 800000 if kind == "text_groups"
                  else 1500000 if kind == "sort_full" else 6001215)
    c = {"kind": kind, "rows": n}
    if kind in ("order_totals", "join_orders", "join_exists", "fused_orders"):
        c["orders"] = max(500, int(n / rng.uniform(2.0, 8.0)))
    if kind in ("order_totals", "join_orders"):
        c["stored"] = rng.random() < 0.5
    if kind == "join_orders":
        c["type"] = rng.choice(["inner", "inner", "right-semi", "right-anti", "right-outer"])
    if kind in ("part_supplier", "join_two_key"):
        c["parts"] = max(100, int(n / rng.uniform(10.0, 60.0)))
    if kind in ("take_top", "fused_orders", "fused_star"):
        c["limit"] = rng.choice([1, 10, 20, 100])
    return c


# ---------------------------------------------------------------------------- seeded columns
# The columns that decide how many rows a plan returns (keys, filtered dates) come from the case alone
# and are put in an order of the seed's; every other column comes from the seed.  So two seeds give
# other tables whose results have the same number of rows.
class _Gen:
    """Seeded columns on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed) * 1000003 + 17)

    def ints(self, lo, hi, n, dtype=torch.int64):
        return torch.randint(lo, hi, (n,), generator=self.g, device="cuda", dtype=torch.int64).to(dtype)

    def decimals(self, lo, hi, n):
        """Two-digit decimals lo/100 .. (hi-1)/100."""
        return self.ints(lo, hi, n).double() / 100.0

    def perm(self, n):
        return torch.randperm(n, generator=self.g, device="cuda")

    def price(self, n):
        return self.decimals(90000, 10495001, n)

    def discount(self, n):
        return self.decimals(0, 11, n)

    def tax(self, n):
        return self.decimals(0, 9, n)

    def quantity(self, n):
        return self.ints(1, 51, n).double()

    def dates(self, n):
        return self.ints(0, DAYS, n, torch.int32)


def _order_key(i):
    """TPC-H's sparse order keys: the first eight of every 32."""
    return (i // 8) * 32 + i % 8 + 1


def _text(words, width):
    t = torch.zeros(len(words), width, dtype=torch.int8)
    for i, w in enumerate(words):
        t[i, :len(w)] = torch.tensor(list(w.encode()), dtype=torch.int8)
    return t.cuda()


_SIZES = ("49", "14", "23", "45", "19", "3", "36", "9")
_TYPES = [" ".join((a, b, c)) for a in ("STANDARD", "SMALL", "MEDIUM", "LARGE", "ECONOMY", "PROMO")
          for b in ("ANODIZED", "BURNISHED", "PLATED", "POLISHED", "BRUSHED")
          for c in ("TIN", "NICKEL", "BRASS", "STEEL", "COPPER")]
_BRANDS = ["BRAND-%d%d" % (i, j) for i in range(1, 6) for j in range(1, 6)]
_PRIORITIES = ["1-URGENT", "2-HIGH", "3-MEDIUM", "4-NOT SPECIFIED", "5-LOW"]


def _suppliers(parts):
    return max(4, parts // 20)


def _supplier_of(part, j, parts):
    """TPC-H's four suppliers of a part, spread over the supplier keys."""
    s = _suppliers(parts)
    return (part + j * (s // 4 + part // s)) % s + 1


def _star_dims(n):
    """Dimension sizes of a star over n fact rows, in the benchmark's proportions (60 M : 2 M : 15 M : 1.5 M)."""
    return max(50, n // 30), max(400, n // 4), max(40, n // 40)


# ---------------------------------------------------------------------------- plans
def _sum(tree, i, out):
    return [[["sum", [tree]], "#", str(i)], "AS", "a#%d" % out]


_REVENUE = ["price#2", "*", ["1.0", "-", "discount#3"]]


def _report(case, g):
    n = case["rows"]
    cols = {1: g.quantity(n), 2: g.price(n), 3: g.discount(n), 4: g.tax(n), 5: g.ints(0, 3, n, torch.uint8),
            6: g.ints(0, 2, n, torch.uint8), 7: g.dates(n)}
    ids = [1, 2, 3, 4, 5, 6]
    aggs = ["flag#5", "status#6", _sum("quantity#1", 101, 201), _sum("price#2", 102, 202), _sum(_REVENUE, 103, 203),
            _sum([_REVENUE, "*", ["1.0", "+", "tax#4"]], 104, 204),
            [[["avg", ["quantity#1"]], "#", "105"], "AS", "a#205"],
            [[["avg", ["price#2"]], "#", "106"], "AS", "a#206"],
            [[["avg", ["discount#3"]], "#", "107"], "AS", "a#207"],
            [[["count", ["1"]], "#", "108L"], "AS", "a#208"]]
    outs = [5, 6] + list(range(201, 209))
    plan = [("filter", {"filter tree": [[["isnotnull", ["d#7"]], "AND", ["d#7", "<=", "2470"]]],
                        "materialized in": [7], "out mask id": 900}),
            ("aggregate", {"is partial": False, "keys": ["flag#5", "status#6"], "input ids": ids, "results": aggs,
                           "out agg ids": outs[2:], "mask map": {c: 900 for c in ids}}),
            ("sort", {"input ids": outs, "key ids": [5, 6], "key orders": [False, False]})]
    return cols, plan, outs


def _order_totals(case, g):
    n, m = case["rows"], case["orders"]
    o = _Gen(0).ints(0, m, n)
    o = torch.sort(o)[0] if case["stored"] else o[g.perm(n)]      # stored: in the order of the order key
    cols = {1: g.quantity(n), 2: g.price(n), 3: _order_key(o)}
    plan = [("aggregate", {"is partial": False, "keys": ["o#3"], "input ids": [1, 2, 3],
                           "results": ["o#3", _sum("quantity#1", 101, 201), _sum("price#2", 102, 202)],
                           "out agg ids": [201, 202]}),
            ("filter", {"filter tree": [["q#201", ">", "150.0"]], "materialized in": [201], "out mask id": 901})]
    return cols, plan, [3, 201, 202, 901]


def _part_supplier(case, g):
    n, p = case["rows"], case["parts"]
    s, at = _Gen(0), g.perm(n)
    part, j, date = s.ints(0, p, n)[at], s.ints(0, 4, n)[at], s.dates(n)[at]
    cols = {1: g.quantity(n), 2: part + 1, 3: _supplier_of(part, j, p), 7: date}
    plan = [("filter", {"filter tree": [[["d#7", ">=", "1994-01-01"], "AND", ["d#7", "<", "1995-01-01"]]],
                        "materialized in": [7], "out mask id": 900}),
            ("aggregate", {"is partial": False, "keys": ["p#2", "s#3"], "input ids": [1, 2, 3],
                           "results": ["p#2", "s#3", _sum("quantity#1", 101, 201),
                                       [[["count", ["1"]], "#", "102L"], "AS", "a#202"]],
                           "out agg ids": [201, 202], "mask map": {1: 900, 2: 900, 3: 900}})]
    return cols, plan, [2, 3, 201, 202]


def _text_groups(case, g):
    n = case["rows"]
    s, at = _Gen(0), g.perm(n)
    cols = {1: _text(_TYPES, 25)[s.ints(0, len(_TYPES), n)[at]], 2: _text(_BRANDS, 10)[s.ints(0, len(_BRANDS), n)[at]],
            3: s.ints(1, 51, n)[at], 4: g.decimals(100, 100001, n)}
    plan = [("filter", {"filter tree": [[["NOT", [["StartsWith", ["t#1", "MEDIUM POLISHED"]]]], "AND",
                                         [["NOT", [["t#1", "LIKE", "%ECONOMY%TIN%"]]], "AND",
                                          ["s#3", "IN", list(_SIZES)]]]],
                        "materialized in": [1, 3], "out mask id": 900}),
            ("aggregate", {"is partial": False, "keys": ["b#2", "t#1", "s#3"], "input ids": [1, 2, 3, 4],
                           "results": ["b#2", "t#1", "s#3", [[["count", ["1"]], "#", "101L"], "AS", "a#201"],
                                       _sum("c#4", 102, 202)],
                           "out agg ids": [201, 202], "mask map": {c: 900 for c in (1, 2, 3, 4)}}),
            ("sort", {"input ids": [2, 1, 3, 201, 202], "key ids": [201, 2, 1, 3],
                      "key orders": [True, False, False, False]})]
    return cols, plan, [2, 1, 3, 201, 202]


def _join_orders(case, g):
    n, m = case["rows"], case["orders"]
    s = _Gen(0)
    o, date, line_date = s.ints(0, m, n), s.dates(m), s.dates(n)
    if case["stored"]:
        o, b = torch.sort(o)[0], torch.arange(m, device="cuda")
    else:
        at, b = g.perm(n), g.perm(m)
        o, line_date = o[at], line_date[at]
    cols = {11: _order_key(b), 12: date[b], 13: g.ints(0, 5, m), 21: _order_key(o), 22: line_date, 23: g.price(n),
            24: g.discount(n)}
    plan = [("filter", {"filter tree": [["d#12", "<", "1170"]], "materialized in": [12], "out mask id": 901}),
            ("filter", {"filter tree": [["d#22", ">", "1170"]], "materialized in": [22], "out mask id": 902}),
            ("join", {"left group": [11, 12, 13], "right group": [21, 22, 23, 24],
                      "materialized in": [11, 12, 13, 21, 23, 24],
                      "mask map": {11: 901, 12: 901, 13: 901, 21: 902, 23: 902, 24: 902}}, 11, 21, [], case["type"])]
    return cols, plan, [11, 12, 13, 21, 23, 24]


def _join_two_key(case, g):
    n, p = case["rows"], case["parts"]
    part = torch.arange(p, device="cuda").repeat_interleave(4)
    j = torch.arange(4 * p, device="cuda") % 4
    lp = g.ints(0, p, n)
    cols = {11: part + 1, 12: _supplier_of(part, j, p), 13: g.decimals(100, 100001, 4 * p),
            21: lp + 1, 22: _supplier_of(lp, g.ints(0, 4, n), p), 23: g.quantity(n), 24: g.price(n)}
    plan = [("join", {"left group": [11, 12, 13], "right group": [21, 22, 23, 24],
                      "materialized in": [11, 12, 13, 21, 22, 23, 24]}, 11, 21, [["s#12", "=", "s#22"]], "inner")]
    return cols, plan, [11, 12, 13, 21, 22, 23, 24]


def _join_exists(case, g):
    n, m = case["rows"], case["orders"]
    s = _Gen(0)
    commit = g.ints(30, DAYS - 30, n, torch.int32)
    cols = {11: _order_key(torch.sort(s.ints(0, m, n))[0]), 12: commit,
            13: commit + s.ints(-20, 31, n, torch.int32),
            21: _order_key(torch.arange(m, device="cuda")), 22: s.dates(m),
            23: _text(_PRIORITIES, 15)[g.ints(0, 5, m)], 24: g.price(m)}
    plan = [("filter", {"filter tree": [["c#12", "<", "r#13"]], "materialized in": [12, 13], "out mask id": 901}),
            ("filter", {"filter tree": [[["d#22", ">=", "1993-01-01"], "AND", ["d#22", "<", "1994-01-01"]]],
                        "materialized in": [22], "out mask id": 902}),
            ("join", {"left group": [11, 12, 13], "right group": [21, 22, 23, 24], "materialized in": [21, 23, 24],
                      "mask map": {11: 901, 21: 902, 23: 902, 24: 902}}, 11, 21, [], "right-semi")]
    return cols, plan, [21, 23, 24]


def _sort_full(case, g):
    n = case["rows"]
    cols = {1: g.price(n), 2: g.dates(n), 3: _order_key(g.perm(n)), 4: _text(_PRIORITIES, 15)[g.ints(0, 5, n)],
            5: g.ints(0, 150000, n)}
    plan = [("sort", {"input ids": [3, 1, 2, 4, 5], "key ids": [1, 2], "key orders": [True, False]})]
    return cols, plan, [3, 1, 2, 4, 5]


def _take_top(case, g):
    n = case["rows"]
    cols = {1: _order_key(g.perm(n)), 2: g.price(n), 3: g.discount(n), 7: g.dates(n)}
    plan = [("project", {"rename map": {}, "materialized in": [2, 3, 7],
                         "used expr": [[_REVENUE, "AS", "rev#20"], [["year", ["d#7"]], "AS", "y#21"]],
                         "materialized out": [20, 21]}),
            ("top", {"limit": case["limit"], "input ids": [1, 20, 21], "key ids": [20, 1],
                     "key orders": [True, False]})]
    return cols, plan, [1, 20, 21]


def _fused_orders(case, g):
    n, m = case["rows"], case["orders"]
    cols = {11: (g.perm(m) + 1).int(), 12: g.dates(m), 21: g.ints(1, m + 1, n, torch.int32), 22: g.dates(n),
            2: g.price(n), 3: g.discount(n)}
    args = [{"name": "Filter", "filter tree": [["d#12", "<", "1170"]], "materialized in": [12], "out mask id": 901},
            {"name": "Filter", "filter tree": [["d#22", ">", "1170"]], "materialized in": [22], "out mask id": 902},
            {"name": "Join", "left keys": [11], "right keys": [21], "join type": "Inner", "left group": [11, 12],
             "right group": [21, 22, 2, 3], "materialized in": [11, 21, 2, 3],
             "mask map": {11: 901, 21: 902, 2: 902, 3: 902}},
            {"name": "Aggregate", "is partial": False, "keys": ["k#11"], "input ids": [11, 2, 3],
             "results": ["k#11", _sum(_REVENUE, 301, 302)], "out agg ids": [302]},
            {"name": "take ordered", "limit": case["limit"], "input ids": [11, 302], "key ids": [302],
             "key orders": [True]}]
    return cols, [("fused", args)], [11, 302]


def _fused_star(case, g):
    n = case["rows"]
    na, nb, nc = _star_dims(n)
    i32 = torch.int32
    cols = {31: (g.perm(na) + 1).int(), 32: g.ints(1, 6, na, torch.uint8), 41: g.ints(1, na + 1, n, i32),
            42: g.ints(1, nb + 1, n, i32), 2: g.price(n), 3: g.discount(n), 51: (g.perm(nb) + 1).int(),
            52: g.ints(1, nc + 1, nb, i32), 61: (g.perm(nc) + 1).int()}
    args = [{"name": "Filter", "filter tree": [["cat#32", "=", "1"]], "materialized in": [32], "out mask id": 901},
            {"name": "Join", "left keys": [31], "right keys": [41], "join type": "Inner", "left group": [31, 32],
             "right group": [41, 42, 2, 3], "materialized in": [31, 41, 42, 2, 3], "mask map": {31: 901}},
            {"name": "Join", "left keys": [51], "right keys": [42], "join type": "Inner", "left group": [51, 52],
             "right group": [31, 41, 42, 2, 3], "materialized in": [51, 52, 42, 2, 3]},
            {"name": "Join", "left keys": [61], "right keys": [52], "join type": "Inner", "left group": [61],
             "right group": [51, 52, 42, 2, 3], "materialized in": [61, 52, 2, 3]},
            {"name": "Aggregate", "is partial": False, "keys": ["c#61"], "input ids": [61, 2, 3],
             "results": ["c#61", _sum(_REVENUE, 71, 72), [[["count", ["1"]], "#", "73L"], "AS", "a#74"]],
             "out agg ids": [72, 74]},
            {"name": "take ordered", "limit": case["limit"], "input ids": [61, 72, 74], "key ids": [72],
             "key orders": [True]}]
    return cols, [("fused", args)], [61, 72, 74]


_KINDS = {"report": _report, "order_totals": _order_totals, "part_supplier": _part_supplier,
          "text_groups": _text_groups, "join_orders": _join_orders, "join_two_key": _join_two_key,
          "join_exists": _join_exists, "sort_full": _sort_full, "take_top": _take_top,
          "fused_orders": _fused_orders, "fused_star": _fused_star}


# ---------------------------------------------------------------------------- running a plan
def _column_type(t):
    return {torch.float64: "float", torch.int64: "int", torch.int32: "date"}.get(t.dtype, "string")


def prepare(case, seed):
    """The tables of a program and the parsed plan that its executor holds."""
    from tqpk.variable import Variable
    cols, plan, outs = _KINDS[case["kind"]](case, _Gen(seed))
    return {"columns": {c: Variable(t, _column_type(t)) for c, t in cols.items()}, "plan": plan, "outs": outs}


def _own(args):
    """The operators write to their argument dicts: each call gets its own."""
    return {k: dict(v) if isinstance(v, dict) else list(v) if isinstance(v, list) else v for k, v in args.items()}


def run(state):
    """One pass of the plan, as the executor's loop calls the operators."""
    from tqpk import operators as ops
    tg = dict(state["columns"])
    for step in state["plan"]:
        op, args = step[0], step[1]
        if op == "filter":
            ops.tqp_filter(True, tg, _own(args), None, None, None, "filter")
        elif op == "join":
            left, right, conditions, jtype = step[2:]
            ops.join_vortex(True, tg, _own(args), left, right, conditions, jtype, None, None, "join")
        elif op == "aggregate":
            ops.tqp_hash_aggregate(True, tg, _own(args), None, None, "aggregate")
        elif op == "project":
            ops.tqp_project(True, tg, _own(args), None, None, "project")
        elif op in ("sort", "top"):
            ops.tqp_sort(True, tg, _own(args), op == "top", op)
        else:
            done = ops.try_fused(True, tg, list(range(len(args))), {i: _own(a) for i, a in enumerate(args)}, 0)
            if done != len(args):
                raise RuntimeError("the plan did not run as one fused run")
    return [tg[c].tensor for c in state["outs"]]


# ---------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes of the columns read and of the outputs written, once each; the arithmetic of the aggregates."""
    k, n = case["kind"], case["rows"]
    m = case.get("orders", 0)
    late = 1.0 - 1171 / DAYS                     # lines after day 1170
    early = 1170 / DAYS                          # orders before it
    if k == "report":
        return {"bytes": n * (4 * 8 + 2 + 4), "flops": 9 * n}
    if k == "order_totals":
        return {"bytes": n * 24 + min(m, n) * 25, "flops": 2 * n}
    if k == "part_supplier":
        rows = n * 365 / DAYS
        return {"bytes": n * 28 + min(rows, 4 * case["parts"]) * 32, "flops": rows}
    if k == "text_groups":
        rows = n * 8 / 50 * 0.92
        return {"bytes": n * (25 + 10 + 8 + 8) + min(rows, 30000) * 59, "flops": rows}
    if k == "join_orders":
        hit = n * late * (early if case["type"] in ("inner", "right-semi") else 1.0)
        width = 24 if case["type"] in ("right-semi", "right-anti") else 44
        return {"bytes": m * 24 + n * 28 + hit * width, "flops": 0}
    if k == "join_two_key":
        return {"bytes": 4 * case["parts"] * 24 + n * 32 + n * 56, "flops": 0}
    if k == "join_exists":
        return {"bytes": n * 16 + m * 35 + m * 0.14 * 31, "flops": 0}
    if k == "sort_full":
        return {"bytes": 2 * n * (8 + 4 + 8 + 15 + 8), "flops": 0}
    if k == "take_top":
        return {"bytes": n * 28, "flops": 2 * n}
    if k == "fused_orders":
        return {"bytes": m * 8 + n * 24, "flops": 3 * n * late * early}
    na, nb, nc = _star_dims(n)
    return {"bytes": n * 24 + na * 5 + nb * 8 + nc * 4, "flops": 3 * n * 0.2}


# ---------------------------------------------------------------------------- the same values in 64 bits and more
def _two_prod(a, b):
    """a * b as an unevaluated sum of two float64 (Dekker's product with Veltkamp's split)."""
    def split(x):
        t = x * 134217729.0
        h = t - (t - x)
        return h, x - h
    p = a * b
    ah, al = split(a)
    bh, bl = split(b)
    return p, ((ah * bh - p) + ah * bl + al * bh) + al * bl


def _one_and(x, sign):
    """1 + sign * x as an unevaluated sum of two float64 (|x| < 1)."""
    s = 1.0 + sign * x
    return s, sign * x - (s - 1.0)


def _times(hi, lo, bh, bl):
    p, e = _two_prod(hi, bh)
    return p, e + (hi * bl + lo * bh)


def _revenue(price, discount):
    h, low = _one_and(discount, -1.0)
    return _times(price, torch.zeros_like(price), h, low)


def _group_sum(group, hi, lo, groups):
    """Sums of hi + lo by group: the multiples of 2^-20 added as integers, the rest as float64."""
    step = 1048576.0
    whole = torch.round(hi * step)
    w = torch.zeros(groups, dtype=torch.int64, device=hi.device).index_add_(0, group, whole.long())
    r = torch.zeros(groups, dtype=torch.float64, device=hi.device).index_add_(0, group, (hi - whole / step) + lo)
    return w.double() / step + r


def _plain_sum(group, x, groups):
    return _group_sum(group, x, torch.zeros_like(x), groups)


def exact(case, seed):
    """What run() returns, in plain torch; None where rows are only moved (joins, orders) or in the place of
    columns that are not computed."""
    k = case["kind"]
    if k.startswith("join") or k == "sort_full":
        return None
    c, _, _ = _KINDS[k](case, _Gen(seed))
    if k == "report":
        keep = c[7] <= 2470
        q, p, d, t = (c[i][keep] for i in (1, 2, 3, 4))
        group = c[5][keep].long() * 2 + c[6][keep].long()
        cnt = torch.bincount(group, minlength=6)
        hi, lo = _revenue(p, d)
        ch, cl = _times(hi, lo, *_one_and(t, 1.0))
        sums = [_plain_sum(group, x, 6) for x in (q, p, d)]
        cols = [sums[0], sums[1], _group_sum(group, hi, lo, 6), _group_sum(group, ch, cl, 6)]
        cols += [s / cnt.double() for s in sums] + [cnt]
        return [None, None] + [x[cnt > 0] for x in cols]
    if k == "order_totals":
        groups = int(c[3].max()) + 1
        some = torch.bincount(c[3], minlength=groups) > 0
        return [None, _plain_sum(c[3], c[1], groups)[some], _plain_sum(c[3], c[2], groups)[some], None]
    if k == "part_supplier":
        keep = (c[7] >= 1461) & (c[7] < 1826)
        wide = int(c[3].max()) + 1
        _, group = torch.unique(c[2][keep] * wide + c[3][keep], return_inverse=True)
        groups = int(group.max()) + 1 if group.numel() else 0
        return [None, None, _plain_sum(group, c[1][keep], groups), torch.bincount(group, minlength=groups)]
    if k == "text_groups":
        words, t = torch.unique(c[1], dim=0, return_inverse=True)      # in the order of their bytes
        _, b = torch.unique(c[2], dim=0, return_inverse=True)
        words = [bytes(w).rstrip(b"\0").decode() for w in words.cpu().numpy().view("uint8")]
        fits = torch.tensor([not w.startswith("MEDIUM POLISHED") and not (w.startswith("ECONOMY") and w.endswith("TIN"))
                             for w in words], device="cuda")
        keep = fits[t] & torch.isin(c[3], torch.tensor([int(x) for x in _SIZES], device="cuda"))
        _, group = torch.unique((b[keep] * len(words) + t[keep]) * 64 + c[3][keep], return_inverse=True)
        groups = int(group.max()) + 1 if group.numel() else 0
        cnt = torch.bincount(group, minlength=groups)
        order = torch.sort(cnt, descending=True, stable=True)[1]
        return [None, None, None, cnt[order], _plain_sum(group, c[4][keep], groups)[order]]
    if k == "take_top":
        rev = c[2] * (1.0 - c[3])
        limit = min(case["limit"], rev.numel())
        return [None, torch.topk(rev, limit, sorted=True)[0], None]
    if k == "fused_orders":
        m = case["orders"]
        early = torch.zeros(m + 1, dtype=torch.bool, device="cuda")
        early[c[11].long()] = c[12] < 1170
        group = c[21].long()
        keep = (c[22] > 1170) & early[group]
        group = group[keep]
        hi, lo = _revenue(c[2][keep], c[3][keep])
        groups = m + 1
    else:
        na, nb, nc = _star_dims(case["rows"])
        cat = torch.zeros(na + 1, dtype=torch.bool, device="cuda")
        cat[c[31].long()] = c[32] == 1
        to_c = torch.zeros(nb + 1, dtype=torch.int64, device="cuda")
        to_c[c[51].long()] = c[52].long()
        keep = cat[c[41].long()]
        group = to_c[c[42][keep].long()]
        hi, lo = _revenue(c[2][keep], c[3][keep])
        groups = nc + 1
    total = _group_sum(group, hi, lo, groups)
    cnt = torch.bincount(group, minlength=groups)
    total[cnt == 0] = -math.inf
    limit = min(case["limit"], int((cnt > 0).sum()))
    top, at = torch.topk(total, limit, sorted=True)
    return [None, top] if k == "fused_orders" else [None, top, cnt[at]]
