"""Device memory of preparing shards at N = 2048: what a bulk load takes while it
runs it gives back, a load goes through in smaller pieces where memory is
short, and serving starts with the scratch returned.  Replies are compared
exactly with those of a load that had all the memory it wanted.
"""
import numpy as np
import pytest

import dnspir_b200 as dp
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
GIB = 1 << 30


def _load(torch, shards, l2):
    l1 = 1024
    g = torch.Generator(device="cuda").manual_seed(71)
    data = torch.randint(0, orc.T, (shards, 8 * l1, dp.N), dtype=torch.int16, device="cuda", generator=g)
    data = data.view(torch.uint16)
    torch.cuda.synchronize()
    queries = [dp.prepare_query(bytes([k]) + bytes(31), 700 * k + 1, k, l1, l2) for k in range(shards)]
    return data, queries


def _free(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("engine", [dp.ENGINE_CUDA_CORES, dp.ENGINE_TENSOR])
def test_bulk_load_gives_its_scratch_back_and_fits_where_memory_is_short(engine):
    torch = pytest.importorskip("torch")
    shards, l2 = 10, 128
    data, queries = _load(torch, shards, l2)
    fleet = dp.Fleet.general(11, 1024, l2, shards)
    fleet.set_engine(engine)
    before = _free(torch)
    fleet.set_shards(0, data)
    # one piece of 10 shards takes 2.5 GiB of rows, more than a fleet keeps (the
    # last rows and a-parts of 10 shards, a few MiB, stay)
    assert before - _free(torch) < GIB + (64 << 20)
    want = [fleet.process_query(q) for q, _ in queries]
    for k, ((_, seed), r) in enumerate(zip(queries, want)):
        assert np.array_equal(dp.process_reply(r, seed), data[k][700 * k + 1].cpu().numpy())
    fleet.close()
    fleet = dp.Fleet.general(11, 1024, l2, shards)
    fleet.set_engine(engine)
    hold = torch.empty(_free(torch) - (3 * GIB) // 2, dtype=torch.uint8, device="cuda")
    assert _free(torch) < 2 * GIB
    fleet.set_shards(0, data)
    del hold
    torch.cuda.empty_cache()
    assert [fleet.process_query(q) for q, _ in queries] == want
    fleet.close()


def test_answers_take_the_scratch_where_memory_is_short():
    # groups of 256 over 4 shards need about 0.6 GiB of workspace; the update's 1
    # GiB of rows is what there is
    torch = pytest.importorskip("torch")
    shards, l2 = 4, 32
    data, queries = _load(torch, shards, l2)
    fleet = dp.Fleet.general(11, 1024, l2, shards)
    fleet.set_engine(dp.ENGINE_TENSOR)
    fleet.set_shards(0, data)
    want = [fleet.process_query(q) for q, _ in queries]
    hold = torch.empty(_free(torch) - GIB // 4, dtype=torch.uint8, device="cuda")
    assert _free(torch) < GIB // 3
    fleet.set_batch(256)
    assert fleet.process_queries([q for q, _ in queries] * 64) == want * 64
    del hold
    torch.cuda.empty_cache()
    fleet.close()


def test_updates_and_new_layouts_take_the_kept_scratch_where_memory_is_short():
    # an update from host memory needs staging (32 MiB a shard) besides the rows,
    # a-parts with a zero slot need slabs half as large again (1 -> 1.5 GiB)
    torch = pytest.importorskip("torch")
    shards, l2 = 4, 32
    data, queries = _load(torch, shards, l2)
    host = data.cpu().numpy()
    fleet = dp.Fleet.general(11, 1024, l2, shards)
    fleet.set_shards(0, data)
    want = [fleet.process_query(q) for q, _ in queries]
    hold = torch.empty(_free(torch) - (16 << 20), dtype=torch.uint8, device="cuda")
    fleet.set_shards(1, host[1:2])
    assert [fleet.process_query(q) for q, _ in queries] == want
    del hold
    torch.cuda.empty_cache()
    fleet.set_shards(0, data)
    hold = torch.empty(_free(torch) - GIB // 4, dtype=torch.uint8, device="cuda")
    parts = dp.get_a_parts(11).copy()
    parts[2] = 0
    try:
        dp.set_a_parts(11, parts)
        fleet.set_shards(0, data)
    finally:
        dp.set_a_parts(11, None)
        del hold
        torch.cuda.empty_cache()
    assert fleet.slab_bytes == shards * dp.required_memory_general(11, 1024) * 32
    fleet.set_shards(0, data)
    assert [fleet.process_query(q) for q, _ in queries] == want
    fleet.close()


def test_serving_starts_with_the_scratch_returned():
    torch = pytest.importorskip("torch")
    shards, l2 = 4, 32
    data, queries = _load(torch, shards, l2)
    fleet = dp.Fleet.general(11, 1024, l2, shards)
    fleet.set_engine(dp.ENGINE_TENSOR)
    fleet.set_shards(0, data)
    want = fleet.process_query(queries[1][0])
    before = _free(torch)
    sv = dp.Server()
    db = sv.add_db(fleet, 1)
    sv.start(graphs=False)
    try:
        # 1 GiB of rows back, less the workspace of groups of one (under 64 MiB)
        assert _free(torch) - before > GIB - (64 << 20)
        assert sv.wait(sv.submit(db, queries[1][0])) == want
    finally:
        sv.stop()
        sv.close()
    fleet.set_shards(0, data)  # an update takes its scratch again
    assert fleet.process_query(queries[1][0]) == want
    fleet.close()
