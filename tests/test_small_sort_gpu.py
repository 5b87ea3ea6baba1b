"""TPC-H Q18 result sizes at the edges of the two-launch result sort (chunks of
256 items, 24,576 items at most; larger results are sorted after a read-back)
against numpy, with all rows tied on totalprice and date so that only the
orderkey orders them, and with none tied."""
import ctypes as C

import numpy as np
import pytest

from bespokeolap_artifacts_b200 import native as N

pytestmark = pytest.mark.gpu

ROW = np.dtype([("sum", "<i8"), ("cust", "<i4"), ("crow", "<i4"), ("okey", "<i4"), ("total", "<i4"), ("date", "<i2"),
                ("p0", "<i2"), ("p1", "<i4")])


@pytest.mark.parametrize("want", [0, 1, 31, 32, 33, 255, 256, 257, 5000, 24_575, 24_576, 24_577, 60_000])
@pytest.mark.parametrize("tied", [False, True])
def test_q18_result_sizes(engine, torch_cuda, want, tied):
    torch = torch_cuda
    n = 70_001
    rng = np.random.default_rng(want + tied)
    okey = rng.permutation(np.arange(1, n + 1, dtype=np.int32) * 3)
    qty = np.full(n, 100, np.int16)
    keep = rng.permutation(n)[:want]
    qty[keep] = 200
    total = np.full(n, 7, np.int32) if tied else rng.integers(-2**31, 2**31, n).astype(np.int32)
    date = np.full(n, 5, np.int16) if tied else rng.integers(-2**15, 2**15, n).astype(np.int16)
    cust = rng.integers(1, 100, n).astype(np.int32)
    order = np.argsort(okey)  # lineitems in orderkey order, one per order
    t = {"ok": okey, "cu": cust, "da": date, "to": total, "lk": okey[order], "lq": qty[order],
         "cm": np.arange(100, dtype=np.int32)}
    g = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in t.items()}
    tb = N.TpchQ18Tables()
    tb.o_orderkey, tb.o_custkey, tb.o_orderdate = g["ok"].data_ptr(), g["cu"].data_ptr(), g["da"].data_ptr()
    tb.o_totalprice, tb.n_orders = g["to"].data_ptr(), n
    tb.l_orderkey, tb.l_quantity, tb.n_lineitem = g["lk"].data_ptr(), g["lq"].data_ptr(), n
    tb.custkey_to_row, tb.n_custkey_map, tb.n_customer = g["cm"].data_ptr(), 100, 100
    tb.orderkey_bound = 3 * n + 1
    out, cnt = (N.TpchQ18Row * n)(), C.c_int64(-1)
    engine.ctx.call("bo_tpch_q18", C.byref(tb), 150, out, n, C.byref(cnt))
    rows = np.frombuffer(out, dtype=ROW)[: cnt.value]
    by = np.lexsort((okey[keep], date[keep], -total[keep].astype(np.int64)))
    assert cnt.value == want
    assert np.array_equal(rows["okey"], okey[keep][by])
    assert np.array_equal(rows["total"], total[keep][by]) and np.array_equal(rows["date"], date[keep][by])
