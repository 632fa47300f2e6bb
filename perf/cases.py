"""The work whose speed is measured: what a program that uses this engine has it do.

Twelve listed cases, one per kind of work or per end of its range, and draw(), which gives
others of the same ranges. A case is a plain dict; prepare() makes its tables on the GPU from
a seed, run() is one pass through the engine's public calls, work() the bytes that pass cannot
do without (every column that the query has to read in full, read once; columns read only for
the rows that a predicate keeps are counted for those rows).

Every output is a whole number (sums of fixed-point integers, counts, keys), so two versions of
the engine agree when they are equal, and no floating-point reference is given.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from gpudbmetalbenchmark_b200 import capi
from gpudbmetalbenchmark_b200.engine import Engine, Q1_COLS, Q12_LI_COLS

M = 1_000_000
MODES = {"global": capi.JOIN_GLOBAL, "radix": capi.JOIN_RADIX, "direct": capi.JOIN_DIRECT, "auto": capi.JOIN_AUTO}
Q3_COLS = ("order_key", "ship_date", "ext_price", "discount")
Q9_COLS = ("part_key", "supp_key", "order_key", "ext_price", "discount", "quantity")
NATION_COLS = ("order_key", "part_key", "supp_key", "ship_date", "flag", "ext_price", "discount")

_engine = None


def engine():
    """One engine for the process, as a program that keeps its tables resident has."""
    global _engine
    if _engine is None:
        _engine = Engine(0)
    return _engine


class State:
    """What a program holds before the call; its tables are freed with it."""

    def __init__(self, kind):
        self.kind, self.tables = kind, []

    def gen(self, *a, **kw):
        t = engine().generate(*a, **kw)
        self.tables.append(t)
        return t

    def __del__(self):
        for t in self.tables:
            if _engine is not None and _engine.ctx:
                _engine.free(t)


def listed():
    return [
        # The smallest table of the served stream: both scans, where launches and the call itself count.
        {"name": "scans_1m", "kind": "scans", "rows": M, "first": 0, "ship_le": 2436, "ship_lo": 365, "days": 365},
        # The benchmark's step: filtered sum and 6-group aggregate over 60M resident rows.
        {"name": "scans_60m", "kind": "scans", "rows": 60 * M, "first": 0, "ship_le": 2436, "ship_lo": 365, "days": 365},
        # The same two scans over a table in pinned host memory, streamed to the GPU.
        {"name": "scans_streamed_8m", "kind": "streamed", "rows": 8 * M, "ship_le": 2436, "ship_lo": 365, "days": 365},
        # Hash join, per-order aggregate and top 10 in the engine's default join mode (one hash table).
        {"name": "q3_6m_global", "kind": "q3", "rows": 6 * M, "mode": "global", "segment": 1, "date": 1170, "k": 10},
        # The same at ten times the rows, in the mode the engine chooses by itself.
        {"name": "q3_60m_auto", "kind": "q3", "rows": 60 * M, "mode": "auto", "segment": 1, "date": 1170, "k": 10},
        # Star join of five tables, grouped by nation and year.
        {"name": "q9_60m", "kind": "q9", "rows": 60 * M},
        # LIKE over the orders' comments and a count of counts.
        {"name": "q13_15m", "kind": "q13", "rows": 15 * M},
        # Two semi-join counts (late orders by priority, ship modes by priority), ordinary size.
        {"name": "q4_q12_6m", "kind": "q4q12", "rows": 6 * M, "from_day": 547},
        # Four revenue reports by nation or customer (Q5, Q7, Q8, Q10) over large tables.
        {"name": "nations_60m", "kind": "nations", "rows": 60 * M, "from_day": 731},
        # Join count with both sides radix-partitioned; half of the orders are on the build side.
        {"name": "join_count_60m_radix", "kind": "join_count", "rows": 60 * M, "mode": "radix"},
        # Stable radix partition of keys with a payload; a size that fills no tile evenly.
        {"name": "partition_20m", "kind": "partition", "rows": 20 * M + 3, "bits": 8},
        # A served batch: 32 requests of four pipelines over tables of three sizes, in one call.
        {"name": "batch_32", "kind": "batch", "rows": 60 * M, "requests": 32},
    ]


def draw(rng):
    def rows(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | rng.randrange(2)

    kind = rng.choice(["scans", "scans", "streamed", "q3", "q3", "q9", "q13", "q4q12", "nations", "join_count",
                       "partition", "batch"])
    case = {"kind": kind}
    if kind in ("scans", "streamed"):
        case["rows"] = rows(50_000, 59 * M) if kind == "scans" else rows(500_000, 8 * M)
        if kind == "scans":
            case["first"] = rng.choice([0, 0, 4, 1, 3])   # a shard may begin at any row of the table
        case.update(ship_le=rng.randrange(300, 2527), ship_lo=rng.randrange(0, 2000), days=rng.randrange(7, 731))
    elif kind == "q3":
        case.update(rows=rows(200_000, 59 * M), mode=rng.choice(["global", "radix", "direct", "auto"]),
                    segment=rng.randrange(5), date=rng.randrange(600, 1800), k=rng.choice([10, 10, 20, 64]))
    elif kind in ("q4q12", "nations"):
        case.update(rows=rows(200_000, 59 * M), from_day=rng.randrange(200, 1400))
    elif kind == "join_count":
        case.update(rows=rows(200_000, 59 * M), mode=rng.choice(["global", "radix", "direct"]))
    elif kind == "partition":
        case.update(rows=rows(100_000, 20 * M), bits=rng.randrange(4, 11))
    elif kind == "q13":
        case["rows"] = rows(50_000, 14 * M)
    elif kind == "batch":
        case.update(rows=rows(2 * M, 59 * M), requests=rng.choice([4, 8, 16, 24, 32]))
    else:
        case["rows"] = rows(200_000, 59 * M)
    return case


def _sizes(rows):
    """Row counts beside a fact table of `rows` rows, in the benchmark's proportions."""
    orders = max(1000, rows // 4)
    return {"orders": orders, "customer": max(100, orders // 10), "part": max(200, rows // 30),
            "supplier": max(8, rows // 600 // 4 * 4)}


def prepare(case, seed):
    s = State(case["kind"])
    s.case = dict(case)
    rows, n = case["rows"], _sizes(case["rows"])
    getattr(s_prepare, case["kind"])(s, rows, n, seed)
    torch.cuda.synchronize()
    return s


class s_prepare:
    @staticmethod
    def scans(s, rows, n, seed):
        t = s.gen("lineitem", rows + s.case["first"], seed=seed, columns=Q1_COLS)
        s.li = t.lineitem(n_rows=rows, row_offset=s.case["first"])

    @staticmethod
    def streamed(s, rows, n, seed):
        s.li = s.gen("lineitem", rows, seed=seed, columns=Q1_COLS, location=capi.MEM_HOST).lineitem()

    @staticmethod
    def q3(s, rows, n, seed):
        s.cu = s.gen("customer", n["customer"], seed=seed, columns=("cust_key", "segment"))
        s.od = s.gen("orders", n["orders"], seed=seed, columns=("order_key", "cust_key", "order_date"),
                     n_cust=n["customer"])
        s.li = s.gen("lineitem", rows, seed=seed, columns=Q3_COLS, n_orders=n["orders"],
                     order_mode=capi.ORDERS_CLUSTERED)

    @staticmethod
    def q9(s, rows, n, seed):
        s.pa = s.gen("part", n["part"], seed=seed, columns=("part_key", "flag"))
        s.su = s.gen("supplier", n["supplier"], seed=seed)
        s.ps = s.gen("partsupp", 4 * n["part"], seed=seed, n_supp=n["supplier"])
        s.od = s.gen("orders", n["orders"], seed=seed, columns=("order_key", "order_date"))
        s.li = s.gen("lineitem", rows, seed=seed, columns=Q9_COLS, n_orders=n["orders"], n_parts=n["part"],
                     n_supp=n["supplier"], order_mode=capi.ORDERS_UNIFORM)

    @staticmethod
    def q13(s, rows, n, seed):
        s.cu = s.gen("customer", max(100, rows // 10), seed=seed, columns=("cust_key",))
        s.od = s.gen("orders", rows, seed=seed, columns=("cust_key", "comment"), n_cust=max(100, rows // 10))

    @staticmethod
    def q4q12(s, rows, n, seed):
        s.od = s.gen("orders", n["orders"], seed=seed, columns=("order_key", "order_date", "priority"))
        s.li = s.gen("lineitem", rows, seed=seed, columns=Q12_LI_COLS, n_orders=n["orders"],
                     order_mode=capi.ORDERS_CLUSTERED)

    @staticmethod
    def nations(s, rows, n, seed):
        s.cu = s.gen("customer", n["customer"], seed=seed, columns=("cust_key", "nation"))
        s.su = s.gen("supplier", n["supplier"], seed=seed)
        s.pa = s.gen("part", n["part"], seed=seed, columns=("part_key", "type"))
        s.od = s.gen("orders", n["orders"], seed=seed, columns=("order_key", "cust_key", "order_date"),
                     n_cust=n["customer"])
        s.li = s.gen("lineitem", rows, seed=seed, columns=NATION_COLS, n_orders=n["orders"], n_parts=n["part"],
                     n_supp=n["supplier"], order_mode=capi.ORDERS_CLUSTERED)

    @staticmethod
    def join_count(s, rows, n, seed):
        g = torch.Generator("cuda").manual_seed(seed)
        keep = torch.rand(n["orders"], device="cuda", generator=g) < 0.5
        s.build = (torch.nonzero(keep).view(-1) * 4 + 1).to(torch.int32)
        s.probe = s.gen("lineitem", rows, seed=seed, columns=("order_key",), n_orders=n["orders"],
                        order_mode=capi.ORDERS_CLUSTERED)

    @staticmethod
    def partition(s, rows, n, seed):
        g = torch.Generator("cuda").manual_seed(seed)
        s.keys = torch.randint(0, 1 << 30, (rows,), device="cuda", generator=g, dtype=torch.int32)
        s.payload = torch.arange(rows, device="cuda", dtype=torch.int32)
        s.out = [torch.empty_like(s.keys), torch.empty_like(s.keys),
                 torch.empty((1 << s.case["bits"]) + 1, device="cuda", dtype=torch.int32)]

    @staticmethod
    def batch(s, rows, n, seed):
        """Requests in turn from the four pipelines, their constants from the seed."""
        rng = random.Random(seed)
        scans = [s.gen("lineitem", r, seed=seed, columns=Q1_COLS).lineitem()
                 for r in (max(1, rows // 60), max(1, rows // 10), rows)]
        tenth = max(1000, rows // 10)
        k = _sizes(tenth)
        parts = State("batch")
        s_prepare.q3(parts, tenth, k, seed)
        s.q3 = capi.Q3Tables(parts.cu.struct(), parts.od.struct(), parts.li.lineitem())
        s_prepare.q9(parts, tenth, k, seed + 1)
        s.q9 = capi.Q9Tables(parts.pa.struct(), parts.su.struct(), parts.ps.struct(), parts.od.struct(),
                             parts.li.lineitem())
        s.parts = parts
        s.scans = scans
        count = s.case["requests"]
        s.reqs = (capi.Request * count)()
        each = (count + 3) // 4
        s.q6_out, s.q1_out = (capi.Q6Result * each)(), (capi.Q1Result * each)()
        s.q3_out, s.q9_out = (capi.Q3Result * each)(), ((capi.Q9Group * 256) * each)()
        for i, r in enumerate(s.reqs):
            j = i // 4
            r.pipeline = (capi.PIPE_Q6, capi.PIPE_Q1, capi.PIPE_Q3, capi.PIPE_Q9)[i % 4]
            r.li = C.pointer(scans[j % 3])
            lo, d = rng.randrange(0, 2000), rng.randrange(0, 11)
            r.q6 = capi.Q6Params(lo, lo + rng.randrange(30, 731), d, min(10, d + rng.randrange(0, 4)),
                                 rng.randrange(1, 52))
            r.q1 = capi.Q1Params(rng.randrange(300, 2527), 0)
            r.q3 = C.pointer(s.q3)
            r.q3p = capi.Q3Params(rng.randrange(5), rng.randrange(200, 2406), rng.randrange(200, 2400), 10,
                                  capi.JOIN_GLOBAL, 0)
            r.q9 = C.pointer(s.q9)
            r.q6_out = C.pointer(s.q6_out[j])
            r.q1_out = C.pointer(s.q1_out[j])
            r.q3_out = C.pointer(s.q3_out[j])
            r.q9_out = C.cast(s.q9_out[j], C.POINTER(capi.Q9Group))
            r.q9_capacity = 256


def run(s):
    return getattr(s_run, s.kind)(s, s.case, engine())


class s_run:
    @staticmethod
    def scans(s, c, e):
        return {"q6": e.q6(s.li, ship_lo=c["ship_lo"], ship_hi=c["ship_lo"] + c["days"]),
                "q1": e.q1(s.li, ship_le=c["ship_le"])}

    streamed = scans

    @staticmethod
    def q3(s, c, e):
        return _table(e.q3(s.cu, s.od, s.li, segment=c["segment"], order_date_lt=c["date"], ship_date_gt=c["date"],
                           k=c["k"], join_mode=MODES[c["mode"]]), c["k"], 3)

    @staticmethod
    def q9(s, c, e):
        return _table(e.q9(s.pa, s.su, s.ps, s.od, s.li), 200, 3)

    @staticmethod
    def q13(s, c, e):
        return _rows(e.q13(s.cu, s.od), 128, 2)

    @staticmethod
    def q4q12(s, c, e):
        d = c["from_day"]
        return {"q4": e.q4(s.od, s.li, date_lo=d, date_hi=d + 92),
                "q12": e.q12(s.od, s.li, receipt_lo=d, receipt_hi=d + 365)}

    @staticmethod
    def nations(s, c, e):
        d = c["from_day"]
        return {"q5": _rows(e.q5(s.cu, s.su, s.od, s.li, date_lo=d, date_hi=d + 365), 5, 2),
                "q7": _rows(e.q7(s.cu, s.su, s.od, s.li, ship_lo=d, ship_hi=d + 730), 16, 4),
                "q8": _rows(e.q8(s.cu, s.su, s.pa, s.od, s.li, date_lo=d, date_hi=d + 730), 8, 3),
                "q10": _table(e.q10(s.cu, s.od, s.li, date_lo=d, date_hi=d + 92), 20, 2)}

    @staticmethod
    def join_count(s, c, e):
        return e.hash_join_count(s.build.data_ptr(), s.build.numel(), s.probe.ptr("order_key"), c["rows"],
                                 mode=MODES[c["mode"]])

    @staticmethod
    def partition(s, c, e):
        k, p, o = s.out
        e.radix_partition(s.keys.data_ptr(), s.payload.data_ptr(), c["rows"], c["bits"], k.data_ptr(), p.data_ptr(),
                          o.data_ptr())
        return s.out

    @staticmethod
    def batch(s, c, e):
        e._check(e.lib.gpudb_batch_run(e.ctx, s.reqs, c["requests"], None, None))
        return {"status": [r.status for r in s.reqs[:4]], "q6": _words(s.q6_out), "q1": _words(s.q1_out),
                "q3": _words(s.q3_out), "q9": _words(s.q9_out)}


def _rows(rows, most, width):
    """An answer's rows as one array of a fixed shape: how many there are depends on the data."""
    a = np.zeros((most, width), dtype=np.int64)
    if rows:
        a[:len(rows)] = rows
    return a


def _table(answer, most, width):
    rows, n = answer
    return {"rows": _rows(rows, most, width), "n": n}


def _words(structs):
    """The result structs as one array of 64-bit words, without a copy."""
    return np.frombuffer(structs, dtype=np.int64)


def work(case):
    kind, rows = case["kind"], case["rows"]
    n = _sizes(rows)
    if kind in ("scans", "streamed"):
        b = 46 * rows                      # Q6 reads 20 bytes a row, Q1 26
    elif kind == "q3":
        joined = case["date"] / 2406 / 5 * max(0, 2527 - case["date"]) / 2527
        b = 5 * n["customer"] + 12 * n["orders"] + 8 * rows + 12 * rows * joined
    elif kind == "q9":
        b = 5 * n["part"] + 5 * n["supplier"] + 16 * 4 * n["part"] + 8 * n["orders"] + 4 * rows + 24 * 0.055 * rows
    elif kind == "q13":
        b = 84 * rows + 4 * max(100, rows // 10)
    elif kind == "q4q12":
        b = 29 * rows + 14 * n["orders"]
    elif kind == "nations":
        b = (8 + 12 + 4 + 5) * rows + (12 + 8 + 12 + 12) * n["orders"] + 19 * n["customer"] + 5 * n["part"]
    elif kind == "join_count":
        b = 4 * rows + 4 * n["orders"] // 2
    elif kind == "partition":
        b = 16 * rows
    else:
        t = _sizes(max(1000, rows // 10))
        b = 26 * (rows + rows // 10 + rows // 60) + rows // 10 * (8 + 4) + 12 * t["orders"] + 64 * t["part"]
    return {"bytes": float(b), "flops": 0.0}
