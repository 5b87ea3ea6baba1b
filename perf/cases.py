"""The engine's work as its callers have it done, one case per pipeline and size.

Every case goes through a public entry point (``engine.Engine``, ``learned.JoinSizer``,
``batching.Batch`` or the C ABI that the drop-in driver calls) over device-resident columns.  The inputs follow
the seeded generators of the package: TPC-H-like values, uniform foreign keys, Zipf-distributed ids.  All
results are whole numbers (counts, fixed-point sums, row lists), so they are the same bit for bit or wrong.

``listed`` gives the sizes the package itself names, ``draw`` any size of the same ranges:

==================  =====================================================================================
scan_agg            Q1 over the wide fact layout (38 B per row); 10 thousand to 60 million rows: the smallest
                    instances of a batch, the declared 6 million rows, the served fact table
lineitem_q1         Q1 over the storage-plan columns (15 B per row) that the drop-in driver keeps
join                the filtered join with the sizing network in the call, asynchronous
join_partitioned    the radix-partitioned join: build sides whose table is far beyond L2
join_multi          what a server does with several waiting joins: one pass for all of them
groupby             the skewed three-way join, group-by and top 10, table sized from an estimate
groupby_partitioned the same with flat keys and a broad filter: millions of groups
tpch_q3, tpch_q18   the two queries of the driver with a join or a group-by per order and sorted rows
batch               many unequal pipelines in one launch of the persistent kernel
==================  =====================================================================================
"""
import ctypes as C
import functools
import math
import types

import numpy as np
import torch

from bespokeolap_artifacts_b200 import batching as B
from bespokeolap_artifacts_b200 import learned as L
from bespokeolap_artifacts_b200 import native as N
from bespokeolap_artifacts_b200.datagen import DATE_HI, DATE_LO, Q1_CUTOFF, days_from_civil, join_date_cutoff
from bespokeolap_artifacts_b200.engine import Engine

SEGMENTS = 5
CATEGORIES = 113
Q3_DATE = days_from_civil(1995, 3, 17) - DATE_LO
Q18_QUANTITY = 250 * 100
FACT = ("ship_date", "quantity", "ext_price", "discount", "tax", "flag_a", "flag_b")


def listed():
    return [
        # The smallest pipeline a batch or a test hands over: launch and latency.
        {"name": "scan_agg_10k", "kind": "scan_agg", "rows": 10_007},
        # The declared scan configuration: 6M rows, 228 MB.
        {"name": "scan_agg_6m", "kind": "scan_agg", "rows": 6_000_000},
        # The served fact table, a ragged number of rows.
        {"name": "scan_agg_60m", "kind": "scan_agg", "rows": 59_999_987},
        # Q1 at scale factor 1 in the driver's own column layout.
        {"name": "lineitem_q1_6m", "kind": "lineitem_q1", "rows": 6_001_215},
        # The headline join: 4% of a 1.5M-row build side, 6M probe rows.
        {"name": "join_6m", "kind": "join", "build": 1_500_000, "probe": 6_000_000, "date_share": 0.2},
        # A build side of 30M qualifying keys: the table is many times L2.
        {"name": "join_partitioned_150m", "kind": "join_partitioned", "build": 150_000_000, "probe": 150_000_000},
        # A full slot of the server: 16 waiting joins over the served tables.
        {"name": "join_multi_60m", "kind": "join_multi", "build": 15_000_000, "probe": 60_000_000, "queries": 16},
        # The declared group-by: A 2.5M, B 36M, C 4M, 8 categories, 21 years.
        {"name": "groupby_36m", "kind": "groupby", "rows": 36_000_000, "years": 21},
        # Flat keys and half of C: 17M groups.
        {"name": "groupby_partitioned_60m", "kind": "groupby_partitioned", "rows": 60_000_000},
        # The driver's Q3 and Q18 at scale factor 1, rows into pinned memory.
        {"name": "tpch_q3_1.5m", "kind": "tpch_q3", "orders": 1_500_000},
        {"name": "tpch_q18_1.5m", "kind": "tpch_q18", "orders": 1_500_000},
        # The declared batch: 64 instances of 10 thousand to 60 million rows.
        {"name": "batch_64", "kind": "batch", "instances": 64, "most": 60_000_000, "mix": 2024},
    ]


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kind = rng.choice(["scan_agg", "lineitem_q1", "join", "join", "join_partitioned", "join_multi", "groupby",
                       "groupby", "groupby_partitioned", "tpch_q3", "tpch_q18", "batch"])
    case = {"kind": kind}
    if kind in ("scan_agg", "lineitem_q1"):
        case["rows"] = size(10_000, 60_000_000)
    elif kind == "join":
        probe = size(10_000, 60_000_000)
        case |= {"build": max(1, int(probe * rng.uniform(0.05, 0.5))), "probe": probe,
                 "date_share": round(rng.uniform(0.04, 1.0), 3)}
    elif kind == "join_partitioned":
        build = size(15_000_000, 150_000_000)
        case |= {"build": build, "probe": min(150_000_000, int(build * rng.uniform(0.7, 4.0)))}
    elif kind == "join_multi":
        probe = size(100_000, 60_000_000)
        case |= {"build": max(1, probe // 4), "probe": probe, "queries": rng.randint(2, N.JOIN_MULTI_MAX)}
    elif kind == "groupby":
        case |= {"rows": size(10_000, 60_000_000), "years": rng.randint(5, 30)}
    elif kind == "groupby_partitioned":
        case["rows"] = size(10_000_000, 60_000_000)
    elif kind in ("tpch_q3", "tpch_q18"):
        case["orders"] = size(15_000, 1_500_000)
    else:
        case |= {"instances": rng.randint(8, 64), "most": size(1_000_000, 50_000_000), "mix": rng.randint(0, 10_000)}
    return case


@functools.lru_cache(maxsize=None)
def _engine():
    """A program makes one engine context and keeps it."""
    return Engine(torch.cuda.current_device())


# ------------------------------------------------------------ preparation --
def _scan_agg(case, seed):
    inst = B.fact_instance(case["rows"], seed, cutoff=Q1_CUTOFF)
    out = torch.empty(6 * C.sizeof(N.Q1Agg), dtype=torch.uint8, device="cuda")
    return {"cols": [inst.cols[k] for k in FACT], "out": out}


def _lineitem_q1(case, seed):
    f = B.fact_instance(case["rows"], seed, cutoff=Q1_CUTOFF).cols
    li = {
        "shipdate": (f["ship_date"] - DATE_LO).to(torch.int16),
        "returnflag_linestatus": f["flag_a"] * 2 + f["flag_b"],
        "extendedprice": f["ext_price"].to(torch.int32),
        "discounted_price": (f["ext_price"] * (100 - f["discount"]) // 100).to(torch.int32),
        "discount": f["discount"].to(torch.uint8),
        "tax": f["tax"].to(torch.uint8),
        "quantity": f["quantity"].to(torch.int16),
        "n_rows": case["rows"],
    }
    out = torch.empty(6 * C.sizeof(N.Q1Agg), dtype=torch.uint8, device="cuda")
    return {"li": li, "out": out}


def _join_columns(case, seed):
    c = B.join_instance(case["probe"], seed, n_build=case["build"], date_lt=0, seg_eq=0).cols
    return (c["b_key"], c["b_date"], c["b_seg"]), (c["p_fk"], c["p_price"], c["p_disc"])


def _join(case, seed):
    build, probe = _join_columns(case, seed)
    rng = np.random.default_rng(seed)
    date_lt, seg = join_date_cutoff(case["date_share"]), int(rng.integers(0, SEGMENTS))
    sizer = L.JoinSizer(_engine(), seed=5)
    # A network that has learnt this filter: the count with the usual margin of 1.7.
    w = sizer.mlp.get_params()
    w[-65:-1] = 0.0
    w[-1] = math.log1p(1.7 * case["build"] * case["date_share"] / SEGMENTS)
    sizer.mlp.set_params(w)
    st = L.join_table_stats(_engine().ctx, *build, case["build"])
    out = torch.empty(C.sizeof(N.JoinResult), dtype=torch.uint8, device="cuda")
    return {"sizer": sizer, "features": L.join_features(st, date_lt, seg), "build": build, "probe": probe,
            "n": (case["build"], case["probe"]), "where": (date_lt, seg), "out": out}


def _join_partitioned(case, seed):
    build, probe = _join_columns(case, seed)
    return {"build": build, "probe": probe, "n": (case["build"], case["probe"]),
            "where": (DATE_HI + 1, seed % SEGMENTS), "fanout": L.JoinSizer.fanout(case["build"] / SEGMENTS)}


def _join_multi_queries(case, seed):
    rng = np.random.default_rng(seed)
    return [(int(rng.integers(DATE_LO + 100, DATE_HI)), int(rng.integers(0, SEGMENTS)))
            for _ in range(case["queries"])]


def _join_multi(case, seed):
    build, probe = _join_columns(case, seed)
    return {"build": build, "probe": probe, "n": (case["build"], case["probe"]),
            "queries": _join_multi_queries(case, seed),
            "out": torch.empty(case["queries"], C.sizeof(N.JoinResult), dtype=torch.uint8, device="cuda")}


def _a_mask(tables):
    """The id bitmap over A that a program builds when it loads the table."""
    n_a = int(tables["a_ids"].numel())
    mask = torch.zeros((tables["a_id_max"] + 32) // 32, dtype=torch.int32, device="cuda")
    _engine().ctx.call("bo_groupby_a_mask_device", C.byref(N.GbACols(N.ptr(tables["a_ids"]), n_a)),
                       tables["a_id_max"], C.c_void_p(mask.data_ptr()))
    tables["a_mask"] = mask


def _gb_sizes(case):
    if case["kind"] == "groupby":
        return max(16, case["rows"] * 25 // 360), max(16, case["rows"] // 9)
    return max(16, case["rows"] * 25 // 60), max(16, case["rows"] // 15)


def _groupby(case, seed):
    n_a, n_c = _gb_sizes(case)
    t = B.groupby_tables_device(n_a, case["rows"], n_c, seed)
    _a_mask(t)
    cats = np.sort(np.random.default_rng(seed).choice(CATEGORIES, size=8, replace=False))
    q = types.SimpleNamespace(cat_set=[int(v) for v in cats], year_lo=1990, year_hi=1989 + case["years"], k=10)
    st = L.groupby_table_stats(_engine().ctx, t, n_a, case["rows"], n_c)
    groups, _ = L.groupby_naive(st, q.cat_set, q.year_lo, q.year_hi)
    return {"tables": t, "query": q, "groups": torch.tensor([groups], dtype=torch.float32, device="cuda")}


def _groupby_partitioned(case, seed):
    n_a, n_c = _gb_sizes(case)
    t = B.groupby_tables_device(n_a, case["rows"], n_c, seed, s_a=0.3, s_c=0.3)
    _a_mask(t)
    q = types.SimpleNamespace(cat_set=list(range(0, CATEGORIES, 2)), year_lo=1900, year_hi=2020, k=10)
    st = L.groupby_table_stats(_engine().ctx, t, n_a, case["rows"], n_c)
    groups, joined = L.groupby_naive(st, q.cat_set, q.year_lo, q.year_hi)
    return {"tables": t, "query": q, "fanout": L.GroupBySizer.fanout(groups), "joined": joined}


def _orders(case, seed):
    """Orders sorted by date, each with 1 to 7 lineitems; lineitems in orderkey order, 8 of every 32 keys used."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n, n_cust = case["orders"], max(5, case["orders"] // 10)

    def ints(lo, hi, size, dtype):
        return torch.randint(lo, hi + 1, (size,), generator=g, device="cuda").to(dtype)

    i = torch.arange(n, device="cuda")
    key = i // 8 * 32 + i % 8 + 1
    date, lines = ints(0, 2404, n, torch.int64), ints(1, 7, n, torch.int64)
    by_date = torch.sort(date, stable=True).indices
    l_key, l_date = torch.repeat_interleave(key, lines), torch.repeat_interleave(date, lines)
    n_line = int(l_key.numel())
    order_row = torch.full((int(key[-1]) + 1,), -1, dtype=torch.int32, device="cuda")
    order_row[key[by_date]] = i.to(torch.int32)
    cust = torch.randperm(n_cust, generator=g, device="cuda")
    cust_row = torch.full((n_cust + 1,), -1, dtype=torch.int32, device="cuda")
    cust_row[cust + 1] = torch.arange(n_cust, dtype=torch.int32, device="cuda")
    return {
        "c_custkey": (cust + 1).to(torch.int32), "c_mktsegment": ints(0, SEGMENTS - 1, n_cust, torch.int16),
        "o_orderkey": key[by_date].to(torch.int32), "o_custkey": ints(1, n_cust, n, torch.int32),
        "o_orderdate": date[by_date].to(torch.int16),
        "o_shippriority": torch.zeros(n, dtype=torch.int32, device="cuda"),
        "o_totalprice": ints(100_000, 50_000_000, n, torch.int32),
        "l_orderkey": l_key.to(torch.int32),
        "l_shipdate": (l_date + ints(1, 121, n_line, torch.int64)).to(torch.int16),
        "l_discounted_price": ints(90_000, 10_500_000, n_line, torch.int32),
        "l_quantity": ints(1, 50, n_line, torch.int16) * 100,
        "orderkey_to_row": order_row, "custkey_to_row": cust_row,
    }


def _filled(table, cols, **scalars):
    """A column struct of the C ABI: device pointers by field name, then the row counts and bounds."""
    for name, _ in table._fields_:
        if name in cols:
            setattr(table, name, cols[name].data_ptr())
    for name, v in scalars.items():
        setattr(table, name, v)
    return table


def _rows_buffer(row, orders):
    """Pinned memory for the result rows: a fortieth of the orders is several times what either query returns."""
    n = max(256, orders // 40)
    return {"max_rows": n, "rows": torch.zeros(n, C.sizeof(row), dtype=torch.uint8, pin_memory=True)}


def _tpch_q3(case, seed):
    c, n = _orders(case, seed), case["orders"]
    n_cust = int(c["c_custkey"].numel())
    tables = _filled(N.TpchQ3Tables(), c, n_customer=n_cust, custkey_bound=n_cust + 1, n_orders=n,
                     n_orderkey_map=int(c["orderkey_to_row"].numel()), n_lineitem=int(c["l_orderkey"].numel()))
    return {"cols": c, "tables": tables, **_rows_buffer(N.TpchQ3Row, n)}


def _tpch_q18(case, seed):
    c, n = _orders(case, seed), case["orders"]
    tables = _filled(N.TpchQ18Tables(), c, n_orders=n, n_lineitem=int(c["l_orderkey"].numel()),
                     n_custkey_map=int(c["custkey_to_row"].numel()), n_customer=int(c["c_custkey"].numel()),
                     orderkey_bound=int(c["orderkey_to_row"].numel()), dense_orderkeys=0, dense_custkeys=0)
    return {"cols": c, "tables": tables, **_rows_buffer(N.TpchQ18Row, n)}


def _batch_mix(case):
    """(kind, rows) of the instances: every kind as often, rows log-uniform from 10 thousand."""
    rng = np.random.default_rng(case["mix"])
    return [(int(rng.integers(0, 3)), int(math.exp(rng.uniform(math.log(1e4), math.log(case["most"])))))
            for _ in range(case["instances"])]


def _batch_instances(case, seed):
    make = {N.BATCH_SCAN_AGG: B.fact_instance, N.BATCH_JOIN: B.join_instance, N.BATCH_GROUPBY: B.groupby_instance}
    insts = [make[kind](rows, 1000 * seed + i) for i, (kind, rows) in enumerate(_batch_mix(case))]
    B.load_tile_table().apply(insts)
    for q in insts:  # what a sizer would say: independence estimates, with a margin
        p = q.params
        if q.kind == N.BATCH_JOIN:
            n = int(q.cols["b_key"].numel())
            q.predicted = 64 + 1.5 * n * (p["date_lt"] - DATE_LO) / (DATE_HI + 1 - DATE_LO) / SEGMENTS
        elif q.kind == N.BATCH_GROUPBY:
            f = 8 / CATEGORIES * (p["year_hi"] - p["year_lo"] + 1) / 121
            q.predicted = 64 + p["a_id_max"] * (1 - (1 - f) ** (q.rows / p["a_id_max"]))
    return insts


def _batch(case, seed):
    insts = _batch_instances(case, seed)
    return {"batch": B.Batch(_engine(), insts, B.load_tile_table().workers_per_sm)}


_PREPARE = {"scan_agg": _scan_agg, "lineitem_q1": _lineitem_q1, "join": _join, "join_partitioned": _join_partitioned,
            "join_multi": _join_multi, "groupby": _groupby, "groupby_partitioned": _groupby_partitioned,
            "tpch_q3": _tpch_q3, "tpch_q18": _tpch_q18, "batch": _batch}


def prepare(case, seed):
    return {"kind": case["kind"], "case": case, **_PREPARE[case["kind"]](case, seed)}


# --------------------------------------------------------------- one pass --
def _rows_of(state, call, row, *args):
    n = C.c_int64()
    buf = C.cast(state["rows"].data_ptr(), C.POINTER(row))
    _engine().ctx.call(call, C.byref(state["tables"]), *args, buf, state["max_rows"], C.byref(n))
    return {"rows": state["rows"], "n_rows": n.value}


def _top(r, k=10):
    """A group-by's answer with its (up to k) rows as one array; rows that do not exist are -1."""
    rows = np.full((k, 3), -1, np.int64)
    for i, row in enumerate(zip(r["keys"], r["counts"], r["min_years"])):
        rows[i] = row
    return {**{f: v for f, v in r.items() if f not in ("keys", "counts", "min_years")}, "rows": rows}


def _batch_answers(results):
    """Every instance's answer, one row each: the eight sums of six groups, a join's five fields, or a group-by's
    counts and rows, with zeros behind."""
    out = np.zeros((len(results), 48), np.int64)
    for i, r in enumerate(results):
        if r["kind"] == "scan_agg":
            v = [x for g in r["groups"] for x in g.values()]
        elif r["kind"] == "join":
            v = [r[f] for f in B.ANSWER_FIELDS["join"]]
        else:
            t = _top(r)
            v = [t["n_groups"], t["joined_rows"], t["c_qualifying"], *t["rows"].ravel()]
        out[i, :len(v)] = v
    return out


def run(state):
    eng, kind = _engine(), state["kind"]
    if kind == "scan_agg":
        eng.q1_fact_device(state["cols"], state["case"]["rows"], Q1_CUTOFF, 3, 2, state["out"])
        return state["out"]
    if kind == "lineitem_q1":
        eng.q1_lineitem_device(state["li"], Q1_CUTOFF - DATE_LO, 6, state["out"])
        return state["out"]
    if kind == "join":
        state["sizer"].join_device(state["features"], state["build"], state["probe"], *state["n"], *state["where"],
                                   state["out"])
        return state["out"]
    if kind == "join_partitioned":
        return eng.join_partitioned(state["build"], state["probe"], *state["n"], *state["where"], state["fanout"])
    if kind == "join_multi":
        eng.join_multi_device(state["build"], state["probe"], *state["n"], state["queries"], state["out"])
        return state["out"]
    if kind == "groupby":
        return _top(eng.groupby_presized(state["tables"], state["query"], state["groups"]))
    if kind == "groupby_partitioned":
        return _top(eng.groupby_partitioned(state["tables"], state["query"], state["fanout"], state["joined"]))
    if kind == "tpch_q3":
        return _rows_of(state, "bo_tpch_q3", N.TpchQ3Row, Q3_DATE, 1)
    if kind == "tpch_q18":
        return _rows_of(state, "bo_tpch_q18", N.TpchQ18Row, Q18_QUANTITY)
    return _batch_answers(state["batch"].run())


# ------------------------------------------------------------------- work --
def _join_bytes(build, probe, share):
    """Build columns and foreign keys once, price and discount of the matching share."""
    return 9 * build + 4 * probe + 16 * share * probe


def _share_any(queries):
    """Share of the build keys that some query of a shared join selects."""
    latest = [max([d for d, s in queries if s == seg], default=DATE_LO) for seg in range(SEGMENTS)]
    return sum(d - DATE_LO for d in latest) / (DATE_HI + 1 - DATE_LO) / SEGMENTS


def work(case):
    """Bytes of the columns a pass has to read and of the rows it writes; integer work, no floating-point
    operations worth a count."""
    kind = case["kind"]
    if kind == "scan_agg":
        b = 38 * case["rows"]
    elif kind == "lineitem_q1":
        b = 15 * case["rows"]
    elif kind == "join":
        b = _join_bytes(case["build"], case["probe"], case["date_share"] / SEGMENTS)
    elif kind == "join_partitioned":
        b = _join_bytes(case["build"], case["probe"], 1 / SEGMENTS)
    elif kind == "join_multi":
        b = _join_bytes(case["build"], case["probe"], _share_any(_join_multi_queries(case, 0)))
    elif kind in ("groupby", "groupby_partitioned"):
        n_a, n_c = _gb_sizes(case)
        b = 8 * case["rows"] + 6 * n_c + n_a // 8
    elif kind == "tpch_q3":  # customer 6 B, orders 10 B, about 4 lineitems of 10 B each
        b = case["orders"] * (0.6 + 10 + 4 * 10)
    elif kind == "tpch_q18":  # about 4 lineitems of 6 B, the order's key
        b = case["orders"] * (4 * 6 + 4)
    else:
        b = _batch_bytes(case)
    return {"bytes": int(b), "flops": 0}


def _batch_bytes(case):
    """Per row of the scanned table: a fact row; a fourth of a build row, a foreign key and a tenth of the payload;
    a B row with its share of C and of A's bitmap."""
    per_row = {N.BATCH_SCAN_AGG: 38, N.BATCH_JOIN: 9 / 4 + 4 + 1.6, N.BATCH_GROUPBY: 8 + 6 / 9 + 25 / 360 / 8}
    return sum(per_row[kind] * rows for kind, rows in _batch_mix(case))


def exact(case, seed):
    """Every output is a whole number that has one right value, the same in any arithmetic: there is nothing
    that 64-bit floating point would give more exactly."""
    return None
