"""The dense form of the presized and partitioned group-by (one entry per
a_id) against the oracle's restatement of the reference's dense-count, min and
ordering patterns (bespoke_ceb/query_q1a.cpp, query_q10a.cpp:843-856,
bespoke_tpch/query_q10.cpp:318-372): with and without the filter in shared
memory, at tile edges of A, with ids no table holds, ties, every k, year ranges
at the byte's limit and past it (hash form), and A without a prebuilt mask."""
import numpy as np
import pytest

from bespokeolap_artifacts_b200 import datagen as dg
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("n_groups", "joined_rows", "keys", "counts", "min_years")


def check(engine, torch, g, mask, log2p=None, groups=None, rerun=0):
    o = O.groupby_topk(g)
    dev = engine.groupby_to_device(g, prebuild_a_mask=mask)
    if log2p is None:
        pred = torch.tensor([float(o["n_groups"] if groups is None else groups)], dtype=torch.float32, device="cuda")
        r = engine.groupby_presized(dev, g, pred)
    else:
        r = engine.groupby_partitioned(dev, g, log2p, float(o["joined_rows"]))
    assert tuple(r[f] for f in FIELDS) == tuple(o[f] for f in FIELDS)
    c = np.isin(g.c_cat, g.cat_set) & (g.c_year >= g.year_lo) & (g.c_year <= g.year_hi)
    assert (r["c_qualifying"], r["reruns"], r["overflowed"]) == (int(c.sum()), rerun, 0)
    return r


# B rows on both sides of the filter's line (2^20), C filters that pass 1% (the filter is used) and nearly all
# (it is not), A sizes at the edges of a collecting block's tile of 2048 ids.
@pytest.mark.parametrize("n_a,n_b,n_c,cats,k", [
    (2047, 1_048_575, 5000, 8, 10), (2048, 1_048_577, 500_000, 8, 64), (2049, 1_300_003, 700_001, 64, 1),
    (65_535, 9, 33, 64, 3), (1, 5000, 31, 64, 10), (600_000, 2_000_001, 1_600_000, 64, 10), (16, 0, 100, 8, 5),
    (500, 4096, 1, 64, 10)])
@pytest.mark.parametrize("mask", [True, False])
def test_dense_sizes(engine, torch_cuda, n_a, n_b, n_c, cats, k, mask):
    g = dg.gen_groupby(n_a, n_b, n_c, seed=n_a % 97 + n_b % 89, n_cat_set=cats, year_lo=1950, k=k)
    check(engine, torch_cuda, g, mask)
    check(engine, torch_cuda, g, mask, log2p=8)


@pytest.mark.parametrize("n_b", [300_000, 2_500_000])
def test_dense_ids_no_table_holds(engine, torch_cuda, n_b):
    g = dg.groupby_with_bad_ids(dg.gen_groupby(50_000, n_b, 60_000, seed=3, n_cat_set=40))
    g.a_ids = g.a_ids[::3].copy()  # two thirds of B's a_ids are no ids of A
    g.a_ids[5] = -9
    g.b_a[3::101] = -1
    check(engine, torch_cuda, g, True)
    check(engine, torch_cuda, g, False, log2p=6)


@pytest.mark.parametrize("year_hi", [1990 + 253, 1990 + 254, 1989])
def test_dense_year_ranges(engine, torch_cuda, year_hi):
    """Codes 1 .. 254 fit a byte; one year more takes the hash form; an empty range joins nothing."""
    g = dg.gen_groupby(3000, 1_200_000, 9000, seed=4, n_cat_set=30, year_lo=1990, year_hi=year_hi)
    g.c_year[:] = 1990 + np.arange(9000) % 300 - 20
    check(engine, torch_cuda, g, True)


def test_dense_equal_counts_keep_id_order(engine, torch_cuda):
    """Every id as often: the top k is the k smallest ids, spread over many blocks' candidates."""
    g = dg.gen_groupby(400_000, 1_200_000, 1000, seed=5, n_cat_set=64, year_lo=0, year_hi=240, k=64)
    g.c_cat[:] = g.cat_set[0]
    g.c_year[:] = np.arange(1000) % 200
    g.b_a = np.random.default_rng(6).permutation(np.arange(1_200_000) % 400_000 + 1).astype(np.int32)
    r = check(engine, torch_cuda, g, True)
    assert r["keys"] == list(range(1, 65)) and set(r["counts"]) == {3}


def test_dense_counts_ascending_with_id(engine, torch_cuda):
    """The best groups come last in every block: each step's candidates beat all before."""
    reps = 1 + np.arange(20_000) // 100
    g = dg.gen_groupby(20_000, int(reps.sum()), 1000, seed=7, n_cat_set=64, year_lo=0, year_hi=240, k=37)
    g.c_cat[:] = g.cat_set[1]
    g.c_year[:] = np.arange(1000) % 200
    g.b_a = np.repeat(np.arange(1, 20_001), reps).astype(np.int32)
    check(engine, torch_cuda, g, True)
    check(engine, torch_cuda, g, True, log2p=4)


def test_dense_under_predicted_reruns(engine, torch_cuda):
    g = dg.gen_groupby(100_000, 1_500_000, 5000, seed=8, n_cat_set=64, year_lo=1900, year_hi=2020)
    check(engine, torch_cuda, g, True, groups=500, rerun=1)
    check(engine, torch_cuda, g, True, log2p=1, rerun=1)


@pytest.mark.parametrize("n_cat,year_lo,k", [(8, 1990, 10), (64, 1900, 64), (64, 1900, 0)])
def test_dense_counts_alone(engine, torch_cuda, n_cat, year_lo, k):
    """More ids than pairs are kept for (2^23): entries are counts, years come from a second pass over B."""
    n_a = (1 << 23) + 1001
    g = dg.gen_groupby(1000, 17_000_003, 200_000, seed=9, n_cat_set=n_cat, year_lo=year_lo, year_hi=2020, k=k)
    rng = np.random.default_rng(10)
    g.a_ids = rng.permutation(np.arange(1, n_a, dtype=np.int32))[: n_a - 5000]
    g.a_ids[0] = n_a
    heavy = rng.integers(1, 40, 17_000_003)
    g.b_a = np.where(rng.random(17_000_003) < 0.01, heavy, rng.integers(-3, n_a + 5, 17_000_003)).astype(np.int32)
    check(engine, torch_cuda, g, True)
    check(engine, torch_cuda, g, False, log2p=13)
