"""Joins of a batch in each of their table forms -- one bit per key value,
hashed slots where the key values do not fit, and the hashed build after a
dense one that met repeated keys -- must give the solo plain join's answer (in
turn checked against the oracle by the join's own tests)."""
import pytest

from bespokeolap_artifacts_b200 import batching as B

pytestmark = pytest.mark.gpu


def with_keys(inst, f):
    inst.cols["b_key"] = f(inst.cols["b_key"].long()).int()
    inst.cols["p_fk"] = f(inst.cols["p_fk"].long()).int()
    return inst


def joins(torch):
    n_probe, n_build = 130_003, 30_001
    insts = []
    for seed, f in enumerate([
            lambda k: k,                                            # dense
            lambda k: k - n_build // 2,                             # dense, negative keys too
            lambda k: k * 65_537,                                   # hashed: far beyond one bit per value
            lambda k: (k * 0x9E3779B1 % 2**32) - 2**31,             # hashed, the whole int32 range
            lambda k: (k + 1) // 2,                                 # every key on two build rows
            lambda k: torch.where(k == 7, torch.full_like(k, 8), k),  # one repeated key
            lambda k: (k + 1) // 2 * 65_537,                        # hashed, repeated keys
            lambda k: torch.full_like(k, 5)]):                      # one key on every build row
        inst = with_keys(B.join_instance(n_probe if seed < 7 else 500, 50 + seed, n_build=n_build, seg_eq=2), f)
        inst.params["date_lt"] = 10_600  # every date: a fifth of the build rows
        inst.predicted = 7000.0
        insts.append(inst)
    return insts


@pytest.mark.parametrize("workers", [0, 1])
def test_join_forms_match_solo(engine, torch_cuda, workers):
    insts = joins(torch_cuda) + [B.fact_instance(20_001, 3), B.groupby_instance(60_000, 4)]
    b = B.Batch(engine, insts, workers_per_sm=workers)
    for _ in range(2):
        for inst, r in zip(insts, b.run()):
            assert B.same_answer(r, B.solo_result(engine, inst)), inst.params
            assert r["reruns"] == 0 if "reruns" in r else True
    b.close()


@pytest.mark.parametrize("extra", [0, 1])
def test_join_key_range_at_the_tables_bits(engine, torch_cuda, extra):
    """A table of 2^10 slots holds a bit for each of 65,536 key values, and one value more takes the hashed form."""
    inst = B.join_instance(40_000, 71, n_build=900, seg_eq=1)
    inst.params["date_lt"] = 10_600
    inst.cols["b_key"][0] = 1
    inst.cols["b_key"][1:] = torch_cuda.arange(2, 901, device="cuda")
    inst.cols["b_key"][-1] = 65_536 + extra
    inst.cols["b_seg"][-1] = 1
    inst.cols["p_fk"][:100] = 65_536 + extra
    inst.cols["p_fk"][100:200] = 65_535
    inst.predicted = 200.0
    b = B.Batch(engine, [inst])
    r = b.run()[0]
    assert B.same_answer(r, B.solo_result(engine, inst)) and r["capacity_log2"] == 10 and r["reruns"] == 0
    b.close()


def test_join_limit_on_items_is_what_it_was(engine, torch_cuda):
    """A pool for exactly the items a footprint names takes those instances, repeated keys included."""
    insts = joins(torch_cuda)
    b = B.Batch.pool(engine, len(insts), sum(B.footprint(i)[1] for i in insts), sum(B.footprint(i)[0] for i in insts))
    b.update(insts)
    for inst, r in zip(insts, b.run()):
        assert B.same_answer(r, B.solo_result(engine, inst))
    b.close()
