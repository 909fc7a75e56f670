"""The bounded waits between the two blocks of a paired chain (N = 2048): with a
short limit and one block leaving before a step, the call fails with
DNSPIR_ERR_TIMEOUT (5), the device stays usable, and the same call without the
hook answers as the oracle does.  No block waits longer than the limit, so the
hook's step may be any: the first, where nothing was exchanged yet, an inner
one, where the leaving block is owed the values its peer had sent, or the last.
Nothing is timed or compared but exact results.
"""
import numpy as np
import pytest

import dnspir_b200 as dp
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
LIMIT_NS = 2_000_000


@pytest.mark.parametrize("step", [0, 1, 5, 7])
def test_preprocessing_times_out_and_recovers(step):
    l = 8  # 8 chains of 8 steps
    data = np.random.default_rng(step).integers(0, orc.T, size=(8 * l, 2048), dtype=np.uint16)
    db = dp.PIRDatabase(11, l)
    db.set_wait_limit(LIMIT_NS, withhold_step=step)
    with pytest.raises(dp.DnspirError) as e:
        db.set_db(data)
    assert e.value.code == 5
    with pytest.raises(dp.DnspirError) as e:
        db.get_a()
    assert e.value.code == 7  # not preprocessed
    db.set_wait_limit()
    db.set_db(data)
    ref = orc.Database(11, l)
    ref.set_db(data)
    assert np.array_equal(db.get_a().astype(np.int64), ref.get_a())
    db.close()


@pytest.mark.parametrize("engine", [dp.ENGINE_CUDA_CORES, dp.ENGINE_TENSOR])
def test_answers_time_out_and_recover(engine):
    l1, l2 = 1024, 16  # secondary chains of 16 steps
    data = np.random.default_rng(5).integers(0, orc.T, size=(1, 8 * l1, 2048), dtype=np.uint16)
    fleet = dp.Fleet.general(11, l1, l2, 2, 1)
    fleet.set_engine(engine)
    fleet.set_wait_limit(LIMIT_NS)
    fleet.withhold_chain_step(9)
    with pytest.raises(dp.DnspirError) as e:
        fleet.set_shards(0, data)
    assert e.value.code == 5
    q, seed = orc.prepare_query(orc.Rng(bytes([21]) + bytes(31)), 4000, 1, l1, l2)
    with pytest.raises(dp.DnspirError) as e:
        fleet.process_query(q)
    assert e.value.code == 7
    fleet.withhold_chain_step(-1)
    fleet.set_shards(0, data)
    for step in (0, 3, 15):
        fleet.withhold_chain_step(step)
        with pytest.raises(dp.DnspirError) as e:
            fleet.process_query(q)
        assert e.value.code == 5
    fleet.withhold_chain_step(-1)
    ref = orc.Database(11, l1)
    ref.set_db(data[0])
    r = fleet.process_query(q)
    assert r == orc.process_query([ref, ref], q, l2)
    assert np.array_equal(orc.process_reply(r, seed), data[0][4000].astype(np.int64))
    fleet.close()


@pytest.mark.parametrize("engine", [dp.ENGINE_CUDA_CORES, dp.ENGINE_TENSOR])
def test_shortest_limit_leaves_the_device_usable(engine):
    # nothing is withheld: whether a wait of a busy device outlasts the limit or
    # not, the call answers rightly or says that it timed out
    l1, l2 = 1024, 16
    data = np.random.default_rng(6).integers(0, orc.T, size=(1, 8 * l1, 2048), dtype=np.uint16)
    fleet = dp.Fleet.general(11, l1, l2, 2, 1)
    fleet.set_engine(engine)
    fleet.set_shards(0, data)
    fleet.set_batch(4)
    queries = [dp.prepare_query(bytes([k]) + bytes(31), 900 * k, k % 2, l1, l2)[0] for k in range(8)]
    want = fleet.process_queries(queries)
    for ns in (1, 1, 100_000, 0):
        fleet.set_wait_limit(ns)
        try:
            assert fleet.process_queries(queries) == want
        except dp.DnspirError as e:
            assert e.code == 5 and ns
    assert fleet.process_queries(queries) == want
    fleet.close()
