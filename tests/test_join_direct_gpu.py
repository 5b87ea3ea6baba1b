"""The direct form of the partitioned join (large calls: one bit per 32-bit
key instead of partitions) against the oracle's restatement of run_q3's
filtered join (bespoke_tpch/query_q3.cpp:182-260): ragged sizes, empty sides,
keys over the whole int32 range, repeated keys (a few, and every key several
times), and calls in a row whose keys share no page of the bit table."""
import numpy as np
import pytest

from bespokeolap_artifacts_b200 import datagen as dg
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("build_rows", "distinct_keys", "match_count", "sum_exact", "sum_trunc")
ROWS = 1 << 22  # both sides together: from here on calls take the direct form


def check(engine, torch, j, log2p, rerun=0):
    b = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (j.b_key, j.b_date, j.b_seg)]
    p = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (j.p_fk, j.p_price, j.p_disc)]
    r = engine.join_partitioned(b, p, j.n_build, j.n_probe, j.date_lt, j.seg_eq, log2p)
    o = O.join_agg(j)
    distinct = len(np.unique(j.b_key[(j.b_date < j.date_lt) & (j.b_seg == j.seg_eq)]))
    assert tuple(r[f] for f in FIELDS) == (o["build_count"], distinct, o["match_count"], o["sum_exact"], o["sum_trunc"])
    assert (r["mode"], r["reruns"], r["overflowed"]) == (2, rerun, 0)


def with_keys(j, key, fk, date_lt=dg.DATE_HI + 1):
    return dg.JoinInput(key.astype(np.int32), j.b_date, j.b_seg, fk.astype(np.int32), j.p_price, j.p_disc, date_lt,
                        j.seg_eq, j.seed)


@pytest.mark.parametrize("nb,npr,log2p", [(1_000_003, ROWS - 1_000_003, 9), (999_937, 5_000_011, 14), (ROWS + 5, 0, 10),
                                          (0, ROWS, 3), (1, ROWS, 0), (ROWS, 1, 10)])
def test_direct_sizes(engine, torch_cuda, nb, npr, log2p):
    check(engine, torch_cuda, dg.gen_join(nb, npr, seed=nb % 1000 + log2p), log2p)


def test_direct_keys_of_the_whole_range_then_dense(engine, torch_cuda):
    j = dg.gen_join(1_200_000, 3_300_000, seed=5)
    rng = np.random.default_rng(6)
    key = np.unique(rng.integers(-2**31, 2**31, 1_500_000))
    key = np.unique(np.concatenate([[-2**31, 2**31 - 1, 0, -1], key[:1_199_990]]))
    fk = np.where(rng.random(3_300_000) < 0.5, rng.choice(key, 3_300_000), rng.integers(-2**31, 2**31, 3_300_000))
    j1 = with_keys(j, rng.permutation(np.resize(key, 1_200_000)), fk)
    check(engine, torch_cuda, j1, 10)
    check(engine, torch_cuda, j, 10)  # no bit of the first call is left
    check(engine, torch_cuda, j1, 12)


@pytest.mark.parametrize("distinct", [1_199_900, 300_000, 1])
def test_direct_repeated_keys(engine, torch_cuda, distinct):
    j = dg.gen_join(1_200_000, 3_300_000, seed=8)
    rng = np.random.default_rng(distinct)
    key = rng.permutation(np.arange(1_200_000) % distinct) * 7 + 1
    fk = rng.choice(key, 3_300_000) + (rng.random(3_300_000) < 0.3)
    if distinct == 1:
        fk = np.where(rng.random(3_300_000) < 0.001, key[0], 5)  # few matches of one key on 240K build rows
    check(engine, torch_cuda, with_keys(j, key, fk), 10)
    check(engine, torch_cuda, j, 10)


def test_direct_too_few_partitions_reruns(engine, torch_cuda):
    check(engine, torch_cuda, dg.gen_join(1_200_000, 3_300_000, seed=9, date_lt=dg.DATE_HI + 1), 2, rerun=1)
