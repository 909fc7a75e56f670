"""The tensor scan's tiles of 48 queries and the default tiles of overlapping
groups, at N = 2048.  Scan outputs equal the CUDA-core engine's word for word,
replies those of single queries.
"""
import numpy as np
import pytest

import dnspir_b200 as dp
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _data(seed, shards, l1):
    return np.random.default_rng(seed).integers(0, orc.T, size=(shards, 8 * l1, dp.N), dtype=np.uint16)


def _queries(picks, l1, l2):
    return [dp.prepare_query(bytes([k % 251, k // 251]) + bytes(30), i, j, l1, l2) for k, (i, j) in enumerate(picks)]


def _qnat(torch, nq, seed):
    g = np.random.default_rng(seed)
    q = np.empty((nq, 6, 2, dp.N), dtype=np.uint32)
    for p, m in enumerate((dp.Q1, dp.Q2)):
        q[:, :, p, :] = g.integers(0, m, size=(nq, 6, dp.N), dtype=np.uint32)
    return torch.from_numpy(q.view(np.int32)).cuda()


@pytest.fixture(scope="module")
def small_pair():
    l1, l2, shards = dp.get_database_shape(32768)
    data = _data(61, 2, l1)
    fleets = []
    for engine in (dp.ENGINE_CUDA_CORES, dp.ENGINE_TENSOR):
        f = dp.Fleet.general(11, l1, l2, shards, 2)
        f.set_engine(engine)
        f.set_shards(0, data)
        fleets.append(f)
    yield fleets, data, l1, l2, shards
    for f in fleets:
        f.close()


@pytest.mark.parametrize("nq", [33, 37, 48, 49, 95])
def test_tiles_of_48_queries_equal_cuda_core_scan(small_pair, nq):
    # every kernel form with 192 operand rows, for full and ragged tiles and for
    # two tiles of queries
    torch = pytest.importorskip("torch")
    (cuda, tensor), _, _, _, shards = small_pair
    q = _qnat(torch, nq, nq)

    def scan(f):
        o = torch.zeros((nq, shards, 2, dp.N, 8), dtype=torch.int32, device="cuda")
        f.scan(q, o)
        return o.cpu().numpy()

    want = scan(cuda)
    tensor.set_batch(nq)
    try:
        for i, shape in enumerate(dp.tscan_shapes()):
            if shape[0] == 192:
                tensor.set_tile(nq, i)
                assert np.array_equal(scan(tensor), want), shape
    finally:
        tensor.set_tile(nq, -1)
        tensor.set_batch(1)


@pytest.mark.parametrize("batch", [12, 30, 37, 48, 60, 90, 120])
def test_overlapping_groups_on_default_tiles(small_pair, batch):
    # calls of three groups take the tiles of groups that overlap the last one's
    # secondary phase, calls of one group those of a group alone
    (_, tensor), data, l1, l2, shards = small_pair
    picks = [((331 * k + batch) % (8 * l1), k % shards) for k in range(3 * batch - 1)]
    queries = _queries(picks, l1, l2)
    tensor.set_batch(batch)
    try:
        many = tensor.process_queries([q for q, _ in queries])
        one = tensor.process_queries([q for q, _ in queries[:batch]])
    finally:
        tensor.set_batch(1)
    assert one == many[:batch]
    assert tensor.process_queries([q for q, _ in queries[::7]]) == many[::7]
    for (i, j), (_, seed), r in zip(picks, queries, many):
        assert np.array_equal(dp.process_reply(r, seed), data[j % 2][i])
