"""Preprocessing calls of many shards at N = 2048, whose chains run in other
forms than those of a few.  Replies are compared exactly with those of the same
shards prepared one a call, and with the oracle.
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


@pytest.mark.parametrize("l1,l2,engine,per_sm", [
    (1024, 128, dp.ENGINE_TENSOR, 1), (1024, 128, dp.ENGINE_CUDA_CORES, 1), (2048, 64, dp.ENGINE_TENSOR, 1),
    (32, 512, dp.ENGINE_CUDA_CORES, 3)])
def test_many_shards_prepared_at_once(l1, l2, engine, per_sm):
    # chains of one call: 8 a shard and half.  Beyond two SMs for each they run one
    # per SM (1), beyond one per SM as up to three blocks an SM (3)
    sms, chains = _sms(), 8 * (2 if l1 == 2048 else 1)
    shards = sms // 2 // chains + 1 if per_sm == 1 else sms // chains + 2
    assert sms < 2 * shards * chains and (shards * chains <= sms) == (per_sm == 1)
    data = _data(l1 + engine, shards, l1)
    picks = [((911 * k + 3) % (8 * l1), k) for k in range(shards)]
    queries = _queries(picks, l1, l2)
    got = []
    for step in (shards, 1):  # all in one call, then a shard a call (pairs of blocks)
        fleet = dp.Fleet.general(11, l1, l2, shards)
        fleet.set_engine(engine)
        for first in range(0, shards, step):
            fleet.set_shards(first, data[first:first + step])
        got.append(fleet.process_queries([q for q, _ in queries]))
        fleet.close()
    assert got[0] == got[1]
    for (i, j), (_, seed), r in zip(picks, queries, got[0]):
        assert np.array_equal(orc.process_reply(r, seed), data[j][i].astype(np.int64))
    if l1 == 32:
        refs = _refs(data, l1)
        for k in (0, shards - 1):
            assert got[0][k] == orc.process_query(refs, queries[k][0], l2)
