"""The key bits of the single join against the oracle, in the probe's shared
memory (build sides of up to 1.536M rows) and in device memory (larger ones,
from 524 thousand expected keys on): keys within the bits' range, beyond it and
negative, repeated keys, ragged sizes, a table probed twice, predictions on both
sides of the rules, and a hashed call after one with bits."""
import numpy as np
import pytest

from bespokeolap_artifacts_b200 import datagen as dg
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("build_rows", "distinct_keys", "match_count", "sum_exact", "sum_trunc")
SMEM_ROWS = 1_536_000  # build rows up to which the bits are in shared memory
BITS_KEYS = (1 << 19) + 1  # predicted rows from which keys are bits


def columns(torch, j):
    return ([torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (j.b_key, j.b_date, j.b_seg)],
            [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (j.p_fk, j.p_price, j.p_disc)])


def want(j):
    o = O.join_agg(j)
    distinct = len(np.unique(j.b_key[(j.b_date < j.date_lt) & (j.b_seg == j.seg_eq)]))
    return o["build_count"], distinct, o["match_count"], o["sum_exact"], o["sum_trunc"]


def fields(r):
    return tuple(r[f] for f in FIELDS)


def check(engine, torch, j):
    b, p = columns(torch, j)
    args = (b, p, j.n_build, j.n_probe, j.date_lt, j.seg_eq)
    w = want(j)
    r = engine.join_plain(*args)
    assert fields(r) == w and r["overflowed"] == 0
    for rows in (BITS_KEYS - 1, BITS_KEYS, max(BITS_KEYS, w[0])):
        r = engine.join_presized(*args, torch.full((1,), float(rows), device="cuda"))
        assert fields(r) == w and r["overflowed"] == 0


def with_keys(j, key, fk):
    return dg.JoinInput(key.astype(np.int32), j.b_date, j.b_seg, fk.astype(np.int32), j.p_price, j.p_disc,
                        dg.DATE_HI + 1, j.seg_eq, j.seed)


@pytest.mark.parametrize("nb,npr", [((1 << 20) + 1, 0), (1_100_003, 1), (1_200_001, 4095), (4_000_000, 2_000_003),
                                    (2_700_001, 1_000_033), (1, 1), (2, 40_000), (33, 257),
                                    (5_000, 0), (30_011, 33_000), (200_000, 1_999_999), (383_999, 700_003),
                                    (1_536_000, 300_000), (1_536_001, 300_000)])
def test_sizes(engine, torch_cuda, nb, npr):
    check(engine, torch_cuda, dg.gen_join(nb, npr, seed=nb % 1000, date_lt=dg.DATE_HI + 1))


@pytest.mark.parametrize("nb", [4_000_000, 1_500_000, 20_000])
@pytest.mark.parametrize("kind", ["dense", "edge", "negative", "sparse", "repeated", "every key five times", "one key"])
def test_keys(engine, torch_cuda, nb, kind):
    npr = 1_500_007
    j = dg.gen_join(nb, npr, seed=3)
    rng = np.random.default_rng(4)
    edge = nb * 16 if nb > SMEM_ROWS else min(4 * nb, SMEM_ROWS)  # the first key without a bit
    key = {"dense": lambda: np.arange(nb), "edge": lambda: edge - nb // 2 + np.arange(nb),
           "negative": lambda: np.arange(nb) - nb // 2, "sparse": lambda: rng.integers(-2**31, 2**31, nb),
           "repeated": lambda: np.where(rng.random(nb) < 0.01, 7, np.arange(nb)),
           "every key five times": lambda: np.arange(nb) // 25 * 3, "one key": lambda: np.full(nb, 11)}[kind]()
    fk = np.where(rng.random(npr) < 0.6, rng.choice(key, npr), rng.integers(-2**31, 2**31, npr))
    if kind == "one key":
        fk = np.where(rng.random(npr) < 0.001, 11, fk + 1)
    check(engine, torch_cuda, with_keys(j, rng.permutation(key), fk))


@pytest.mark.parametrize("nb", [3_300_000, 900_000])
def test_probed_twice_and_hashed_after(engine, torch_cuda, nb):
    from bespokeolap_artifacts_b200 import native as N
    import ctypes as C

    torch = torch_cuda
    j = dg.gen_join(nb, 700_001, seed=5, date_lt=dg.DATE_HI + 1)
    small = dg.gen_join(30_000, 90_001, seed=6, date_lt=dg.DATE_HI + 1)
    b, p = columns(torch, j)
    out = torch.zeros(C.sizeof(N.JoinResult), dtype=torch.uint8, device="cuda")

    def result():
        engine.synchronize()
        return N.JoinResult.from_buffer_copy(out.cpu().numpy().tobytes()).as_dict()

    pred = torch.full((1,), 600_000.0, device="cuda")
    engine.join_presized_device(b, p, j.n_build, j.n_probe, j.date_lt, j.seg_eq, pred, out)
    assert fields(result()) == want(j)
    half = dg.JoinInput(j.b_key, j.b_date, j.b_seg, *[x[::2].copy() for x in (j.p_fk, j.p_price, j.p_disc)], j.date_lt,
                        j.seg_eq, j.seed)
    hb, hp = columns(torch, half)
    engine.join_probe_device(hp, half.n_probe, out)
    assert fields(result()) == want(half)
    sb, sp = columns(torch, small)
    assert fields(engine.join_plain(sb, sp, small.n_build, small.n_probe, small.date_lt, small.seg_eq)) == want(small)
    engine.join_probe_device(p, j.n_probe, out)
    cross = dg.JoinInput(small.b_key, small.b_date, small.b_seg, j.p_fk, j.p_price, j.p_disc, small.date_lt,
                         small.seg_eq, j.seed)
    assert fields(result()) == want(cross)


def test_few_matches_queue_over_many_steps(engine, torch_cuda):
    j = dg.gen_join(1_000, 80_000_003, seed=9, date_lt=dg.DATE_HI + 1)
    fk = np.full(j.n_probe, 999_999)
    fk[::300_007] = 1 + np.arange(len(fk[::300_007])) % 1_000
    check(engine, torch_cuda, with_keys(j, 1 + np.arange(1_000), fk))


def test_low_prediction_overflows_and_reruns(engine, torch_cuda):
    j = dg.gen_join(8_000_000, 500_000, seed=7, date_lt=dg.DATE_HI + 1)  # 1.6 million keys
    b, p = columns(torch_cuda, j)
    pred = torch_cuda.full((1,), float(BITS_KEYS), device="cuda")  # a table of 2^22 slots: 1.6 million fit
    r = engine.join_presized(b, p, j.n_build, j.n_probe, j.date_lt, j.seg_eq, pred)
    assert fields(r) == want(j) and r["reruns"] == 0
    j = dg.gen_join(20_000_000, 500_000, seed=8, date_lt=dg.DATE_HI + 1)  # 4 million keys: too many
    b, p = columns(torch_cuda, j)
    r = engine.join_presized(b, p, j.n_build, j.n_probe, j.date_lt, j.seg_eq, pred)
    assert fields(r) == want(j) and r["reruns"] == 1
