"""A served group whose kernel's bounded wait gives up fails alone.

Two groups of one database are in flight at once.  The scan of the second one
(two queries) is made to run out of its limit (withhold hooks, 0.5 ms) while
the first one (48 queries, a secondary phase of about ten milliseconds) is
still on the device: its queries fail with DNSPIR_ERR_TIMEOUT (5), every query
of the first group gets the reply it gets alone, and the next groups are
answered.  Replies are bytes, compared exactly.
"""
import numpy as np
import pytest

import dnspir_b200 as dp
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [False, True])
def test_only_the_group_that_timed_out_fails(graphs):
    l1, l2, shards, first, second = 1024, 2048, 2, 48, 2
    data = np.random.default_rng(31).integers(0, orc.T, size=(shards, 8 * l1, dp.N), dtype=np.uint16)
    fleet = dp.Fleet.general(11, l1, l2, shards)
    fleet.set_engine(dp.ENGINE_TENSOR)
    fleet.set_shards(0, data)
    picks = [((157 * k) % (8 * l1), k % shards) for k in range(first + second)]
    made = [dp.prepare_query(bytes([k]) + bytes(31), i, j, l1, l2) for k, (i, j) in enumerate(picks)]
    fleet.set_batch(first + second)
    alone = fleet.process_queries([q for q, _ in made])
    for (i, j), (_, seed), r in zip(picks, made, alone):
        assert np.array_equal(dp.process_reply(r, seed), data[j][i])
    fleet.set_wait_limit(500_000, withhold_chunk=2)
    fleet.withhold_group_size(second)
    sv = dp.Server()
    db = sv.add_db(fleet, 64)
    sv.start(graphs=graphs)
    try:
        for _ in range(3):
            sv.set_batching(db, first, 1000.0)
            a = [sv.submit(db, q) for q, _ in made[:first]]
            sv.set_batching(db, second, 1000.0)
            b = [sv.submit(db, q) for q, _ in made[first:]]
            assert [sv.wait(t) for t in a] == alone[:first]
            for t in b:
                with pytest.raises(dp.DnspirError) as e:
                    sv.wait(t)
                assert e.value.code == 5
            sv.set_batching(db, 1, 0.0)
            assert sv.wait(sv.submit(db, made[0][0])) == alone[0]
    finally:
        sv.stop()
        sv.close()
        fleet.close()
