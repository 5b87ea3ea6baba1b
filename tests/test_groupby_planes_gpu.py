"""The group-by's counts from bit planes (partitioned form, B of a million rows
and more, most of C passing) against the oracle: C's bitmap in one to four parts
and beyond, at the parts' edges, rows that miss C or A, ragged B, one heavy id."""
import numpy as np
import pytest

from bespokeolap_artifacts_b200 import datagen as dg
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("n_groups", "joined_rows", "keys", "counts", "min_years")
PART = 1600 * 1024  # C rows whose bits one block holds


def check(engine, g, log2p=10):
    o = O.groupby_topk(g)
    r = engine.groupby_partitioned(engine.groupby_to_device(g, prebuild_a_mask=True), g, log2p, float(o["joined_rows"]))
    assert tuple(r[f] for f in FIELDS) == tuple(o[f] for f in FIELDS)
    assert (r["reruns"], r["overflowed"]) == (0, 0)


@pytest.mark.parametrize("n_c", [1, 127, 300_001, PART, PART + 1, 2 * PART - 1, 2 * PART + 33, 3 * PART + 129,
                                 4 * PART, 4 * PART + 1])
@pytest.mark.parametrize("n_b", [(1 << 20) + 7, 2_300_001])
def test_parts_of_the_bitmap(engine, n_c, n_b):
    g = dg.gen_groupby(700_000, n_b, n_c, seed=n_c % 101, n_cat_set=60, year_lo=1900, year_hi=2020)
    edges = np.array([x for p in range(5) for x in (p * PART - 1, p * PART, p * PART + 1)] + [n_c - 1, n_c, -1, 2**31 - 1])
    g.b_c[::7] = np.resize(edges, len(g.b_c[::7])).astype(np.int32)  # the parts' edges, C's end, ids beyond
    g.b_a[::11] = -5
    g.c_year[::2] = 1930  # most of C passes
    g.c_cat[::2] = g.cat_set[0]
    check(engine, g)


def test_one_heavy_id_and_ids_in_two_passes(engine):
    g = dg.gen_groupby(17_500_000, 1_500_003, 400_000, seed=6, n_cat_set=60, year_lo=1900, year_hi=2020)
    g.b_a[::3] = g.a_ids.max()  # the last id: a third of the rows
    check(engine, g, 14)
