"""Shards answer with the constants of the a-parts that they were preprocessed
under, not with those last built on the device: a database that is being served
keeps its answers when other a-parts (expand, bfv.rs:46-49) are installed and
another shard is prepared under them.  Replies are bytes, compared exactly.
"""
import numpy as np
import pytest

import dnspir_b200 as dp
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [dp.ENGINE_CUDA_CORES, dp.ENGINE_TENSOR])
def test_served_answers_outlive_a_change_of_a_parts(engine):
    l1, l2 = 1024, 16
    data = np.random.default_rng(41).integers(0, orc.T, size=(1, 8 * l1, dp.N), dtype=np.uint16)
    small = np.random.default_rng(42).integers(0, orc.T, size=(8 * 8, dp.N), dtype=np.uint16)
    fleet = dp.Fleet.general(11, l1, l2, 2, 1)
    fleet.set_engine(engine)
    fleet.set_shards(0, data)
    other = dp.PIRDatabase(11, 8)
    queries = [dp.prepare_query(bytes([k]) + bytes(31), 500 * k + 3, k % 2, l1, l2) for k in range(3)]
    want = [fleet.process_query(q) for q, _ in queries]
    for k, ((_, seed), r) in enumerate(zip(queries, want)):
        assert np.array_equal(dp.process_reply(r, seed), data[0][500 * k + 3])
    sv = dp.Server()
    db = sv.add_db(fleet, 4)
    sv.start(graphs=False)
    try:
        dp.set_a_parts(11, np.random.default_rng(43).integers(0, orc.Q, size=(6, dp.N), dtype=np.uint64))
        other.set_db(small)
        for (q, _), r in zip(queries, want):
            assert sv.wait(sv.submit(db, q)) == r
    finally:
        dp.set_a_parts(11, None)
        sv.stop()
        sv.close()
    with pytest.raises(dp.DnspirError) as e:
        fleet.process_query(queries[0][0])
    assert e.value.code == 7  # the a-parts were installed anew since
    fleet.set_shards(0, data)
    assert fleet.process_query(queries[0][0]) == want[0]
    fleet.close()
    other.close()
