"""Groups whose secondary phase takes several chunks, under every schedule
(N = 2048, secondary group of order 2048).  Replies are compared exactly with
the same queries answered one at a time, and with the oracle on both sides of
the line between the chunks.
"""
import numpy as np
import pytest

import dnspir_b200 as dp
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _sms():
    torch = pytest.importorskip("torch")
    return torch.cuda.get_device_properties(0).multi_processor_count


def _data(seed, shards, l1):
    return np.random.default_rng(seed).integers(0, orc.T, size=(shards, 8 * l1, dp.N), dtype=np.uint16)


def _refs(data, l1):
    refs = []
    for d in data:
        refs.append(orc.Database(11, l1))
        refs[-1].set_db(d)
    return refs


def _queries(picks, l1, l2):
    rng = orc.Rng(bytes([l1 % 251, l2 % 251]) + bytes(30))
    return [orc.prepare_query(rng, i, j, l1, l2) for i, j in picks]


@pytest.fixture(scope="module")
def many_chunks():
    # the full secondary group (order 2048, two halves): a chunk is SMs / 2
    # queries, fewer than the CUDA-core engine's groups of 128
    l1, l2, count, nb = 32, 2048, 256, 128
    chunk = _sms() // 2
    assert nb / 2 < chunk < nb
    data = _data(51, 2, l1)
    fleet = dp.Fleet.general(11, l1, l2, count, 2)
    fleet.set_shards(0, data)
    picks = [((53 * k + 7) % (8 * l1), (71 * k) % count) for k in range(2 * nb)]
    queries = _queries(picks, l1, l2)
    alone = fleet.process_queries([q for q, _ in queries])
    refs = _refs(data, l1)
    shards = [refs[k % 2] for k in range(count)]
    for k in (0, chunk - 1, chunk, nb - 1, 2 * nb - 1):  # either side of the line between the chunks
        assert alone[k] == orc.process_query(shards, queries[k][0], l2), k
    for (i, j), (_, seed), r in zip(picks, queries, alone):
        assert np.array_equal(orc.process_reply(r, seed), data[j % 2][i].astype(np.int64))
    yield fleet, [q for q, _ in queries], alone, nb
    fleet.close()


@pytest.mark.parametrize("schedule", [0, 1, 2, 4, 6])
def test_schedules_over_several_chunks(many_chunks, schedule):
    # two groups a call, each of two chunks: the second group's primary phase
    # overlaps the first group's secondary phase, waits for all of it or for its
    # second chunk; with 4 the chains of both chunks are pairs of blocks
    fleet, queries, alone, nb = many_chunks
    fleet.set_batch(nb)
    fleet.set_schedule(nb, schedule)
    before = fleet.launch_count()
    try:
        assert fleet.process_queries(queries) == alone
    finally:
        fleet.set_schedule(nb, -1)
        fleet.set_batch(1)
    # a group: decode, query vectors, scan, and five kernels a chunk
    assert fleet.launch_count() - before == 2 * (3 + 2 * 5)
