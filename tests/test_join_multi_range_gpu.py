"""How the shared joins choose their form, against the oracle: the range of all
keys decides, then that of the keys of rows with a class, then the hash table;
with the same counts and capacity whichever pass counted the rows."""
import numpy as np
import pytest

from bespokeolap_artifacts_b200 import datagen as dg
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("build_rows", "distinct_keys", "match_count", "sum_exact", "sum_trunc")
PARAMS = [(9000, 1), (dg.DATE_HI + 1, 1), (dg.DATE_HI + 1, 2), (9500, 1), (dg.DATE_LO, 3)]


@pytest.mark.parametrize("nb", [1, 7, 100_003])
@pytest.mark.parametrize("kind", ["dense", "negative", "outliers without a class", "outliers", "spread", "no class"])
def test_forms(engine, torch_cuda, nb, kind):
    rng = np.random.default_rng(nb)
    j = dg.gen_join(nb, 300_007, seed=nb % 97)
    key, seg = rng.permutation(nb) + 1, j.b_seg.copy()
    ends = [0, -1][:nb]
    if kind == "negative":
        key = key - nb // 2 - 5
    elif kind == "spread":
        key = key.astype(np.int64) * (2**32 // (nb + 1)) - 2**31
    elif kind.startswith("outliers"):
        key[ends] = [-2**31, 2**31 - 1][:len(ends)]
        seg[ends] = 9 if kind.endswith("class") else 1
    elif kind == "no class":
        seg[:] = 9
    fk = np.where(rng.random(j.n_probe) < 0.7, rng.choice(key, j.n_probe), rng.integers(-2**31, 2**31, j.n_probe))
    j = dg.JoinInput(key.astype(np.int32), j.b_date, seg.astype(np.uint8), fk.astype(np.int32), j.p_price, j.p_disc,
                     j.date_lt, j.seg_eq, j.seed)
    b = [torch_cuda.from_numpy(np.ascontiguousarray(x)).cuda() for x in (j.b_key, j.b_date, j.b_seg)]
    p = [torch_cuda.from_numpy(np.ascontiguousarray(x)).cuda() for x in (j.p_fk, j.p_price, j.p_disc)]
    got = engine.join_multi(b, p, nb, j.n_probe, PARAMS)
    union = int(np.any([(j.b_date < d) & (j.b_seg == s) for d, s in PARAMS], axis=0).sum())
    top = max(10, (2 * nb - 1).bit_length())
    cap = next(c for c in range(10, top + 1) if c == top or 1 << c >= 2 * union)
    for g, (d, s) in zip(got, PARAMS):
        jj = dg.JoinInput(j.b_key, j.b_date, j.b_seg, j.p_fk, j.p_price, j.p_disc, d, s, j.seed)
        o = O.join_agg(jj)
        rows = int(((j.b_date < d) & (j.b_seg == s)).sum())
        assert tuple(g[f] for f in FIELDS) == (rows, rows, o["match_count"], o["sum_exact"], o["sum_trunc"])
        assert (o["build_count"], g["capacity_log2"], g["reruns"], g["overflowed"]) == (rows, cap, 0, 0)
