"""The grid rule and the block flush of the Q1 scans: row counts around a full
block of chunks and a full resident grid, and every row at the ends of its value
range in the first, the last and a single group, bit-exact against the oracle."""
import numpy as np
import pytest

from bespokeolap_artifacts_b200 import datagen as dg
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# A block takes 256 chunks of four (fact) or eight (storage plan) rows; 148 SMs x 2 blocks.
FACT, LINE, SMS = 1024, 2048, 148


@pytest.mark.parametrize("n", [FACT - 1, FACT, FACT + 1, 3 * FACT + 3, 2 * SMS * FACT + 5, 256 * 2 * SMS * 256 + 7])
def test_fact_grid_edges(engine, n):
    t = dg.gen_fact(n, 41)
    assert engine.q1_fact_host(t, dg.Q1_CUTOFF) == O.q1_fact(t, dg.Q1_CUTOFF)[0]


@pytest.mark.parametrize("n", [LINE - 1, LINE, LINE + 1, 5 * LINE + 7, 2 * SMS * LINE + 9])
def test_storage_plan_grid_edges(engine, n):
    li = dg.fact_to_storage_plan(dg.gen_fact(n, 42))
    cut = dg.Q1_CUTOFF - 8035
    assert engine.q1_lineitem_host(li, cut, 6) == O.q1_lineitem(li, cut, 6)[0]


@pytest.mark.parametrize("n_fa,n_fb", [(3, 2), (4, 2), (1, 1)])
@pytest.mark.parametrize("high", [False, True])
def test_fact_extreme_values(engine, n_fa, n_fb, high):
    n = 2 * SMS * 256 * 64 + 3
    t = dg.gen_fact(n, 43)
    t.n_flag_a, t.n_flag_b = n_fa, n_fb
    for col, lo, hi in ((t.quantity, 0, 2**31 - 1), (t.ext_price, 0, 2**31 - 1), (t.discount, 0, 100), (t.tax, 0, 100)):
        col[:] = hi if high else lo
    if high:
        t.discount[::2] = 0
    t.flag_a[:] = n_fa - 1
    t.flag_b[:] = n_fb - 1
    want, rc = O.q1_fact(t, dg.DATE_HI)
    assert rc == 0
    assert engine.q1_fact_host(t, dg.DATE_HI) == want


@pytest.mark.parametrize("n_groups", [1, 6, 7, 8])
@pytest.mark.parametrize("price,qty,disc,tax", [(2**31 - 1, 32767, 0, 255), (-2**31, -32768, 255, 255)])
def test_storage_plan_extreme_values(engine, n_groups, price, qty, disc, tax):
    n = 2 * SMS * 256 * 64 + 3
    li = dg.fact_to_storage_plan(dg.gen_fact(n, 44))
    for name, v in (("extendedprice", price), ("discounted_price", price), ("quantity", qty), ("discount", disc), ("tax", tax),
                    ("returnflag_linestatus", n_groups - 1), ("shipdate", 0)):
        li[name][:] = v
    want, rc = O.q1_lineitem(li, 1, n_groups)
    assert rc == 0
    assert engine.q1_lineitem_host(li, 1, n_groups) == want
