"""a-parts whose query polynomial is zero at some slots of the transform, at
N = 2048: there the entries of a row do not follow from the chain's states, so
the primary shards store three arrays a row (K = 6144 in the tensor scan of a
full shard) and the secondary chains keep their entries at those slots.  Both
primary orders and engines and every form of the secondary chains answer the
oracle's bytes; nothing is compared with a tolerance.
"""
import numpy as np
import pytest

import dnspir_b200 as dp
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
PRIMES = (dp.Q1, dp.Q2)


def _at(poly, slot, pi):
    """Value at zeta^-(2 slot + 1), the transform's slot (weighted_ntt, base_pir.rs:453-466)."""
    p = PRIMES[pi]
    x = pow(int(orc.zeta(11, pi)), p - 2, p)
    x = pow(x, 2 * slot + 1, p)
    v = 0
    for c in reversed([int(c) for c in poly]):
        v = (v * x + c) % p
    return v


def _zero_at(poly, slot, pi):
    """poly less the constant that makes it zero at the slot mod PRIMES[pi], unchanged mod the other prime."""
    p, other = PRIMES[pi], PRIMES[1 - pi]
    out = poly.copy()
    lift = _at(poly, slot, pi) * other * pow(other, -1, p) % (p * other)
    out[0] = (int(out[0]) - lift) % (p * other)
    assert _at(out, slot, pi) == 0
    return out


@pytest.fixture
def zero_slots():
    def install(which):
        parts = dp.get_a_parts(11).copy()
        parts[which] = _zero_at(parts[which], 77, 0)
        parts[which] = _zero_at(parts[which], 1500, 1)
        dp.set_a_parts(11, parts)
        orc.set_aparts(11, parts)
    yield install
    dp.set_a_parts(11, None)
    orc.set_aparts(11, None)


def _data(seed, l1):
    return np.random.default_rng(seed).integers(0, orc.T, size=(1, 8 * l1, dp.N), dtype=np.uint16)


@pytest.mark.parametrize("l1,which", [(1024, 2), (2048, 2), (2048, 3)])
def test_three_arrays_match_oracle(zero_slots, l1, which):
    zero_slots(which)
    l2, data = 16, _data(81 + which, l1)
    ref = orc.Database(11, l1)
    ref.set_db(data[0])
    rng = orc.Rng(bytes([l1 % 251, which]) + bytes(30))
    queries = [orc.prepare_query(rng, (8 * l1 - 1) * k // 9, k % 2, l1, l2)[0] for k in range(10)]
    want = [orc.process_query([ref, ref], q, l2) for q in queries]
    for engine in (dp.ENGINE_CUDA_CORES, dp.ENGINE_TENSOR):
        fleet = dp.Fleet.general(11, l1, l2, 2, 1)
        assert fleet.slab_bytes == dp.required_memory_general(11, l1) * 32
        fleet.set_engine(engine)
        fleet.set_shards(0, data)
        for batch in (1, 16):
            fleet.set_batch(batch)
            assert fleet.process_queries(queries) == want
        if engine == dp.ENGINE_TENSOR:
            for i, shape in enumerate(dp.tscan_shapes()):
                fleet.set_tile(10, i)
                assert fleet.process_queries(queries) == want, shape
        fleet.close()
    db = dp.PIRDatabase(11, l1)
    db.set_db(data[0])
    assert np.array_equal(db.get_a().astype(np.int64), ref.get_a())
    gen = np.random.default_rng(l1)
    qb = gen.integers(0, orc.Q, size=(8, dp.N), dtype=np.int64)
    qc = gen.integers(0, orc.Q, size=(8, dp.N), dtype=np.int64) if l1 == dp.N else None
    gk = gen.integers(0, orc.Q, size=(8, 2, dp.N), dtype=np.int64)
    assert np.array_equal(db.perform_pir_split(qb, qc, gk).astype(np.int64), ref.perform_pir_split(qb, qc, gk))
    db.close()


@pytest.mark.parametrize("l2,which,batch", [(16, 4, 60), (2048, 4, 26), (2048, 5, 26)])
def test_secondary_chains_match_oracle(zero_slots, l2, which, batch):
    # one query (a chain on two SMs), 20 or 26 of order 16 or 2048 (one SM), more
    # (three parts a block), and pairs of blocks at any number (schedule 4)
    zero_slots(which)
    l1 = 1024
    data = _data(91, l1)
    fleet = dp.Fleet.general(11, l1, l2, 2, 1)
    fleet.set_engine(dp.ENGINE_TENSOR)
    fleet.set_shards(0, data)
    ref = orc.Database(11, l1)
    ref.set_db(data[0])
    rng = orc.Rng(bytes([l2 % 251, which]) + bytes(30))
    queries = [orc.prepare_query(rng, 130 * k, k % 2, l1, l2)[0] for k in range(batch)]
    single = fleet.process_queries(queries)
    for k in (0, batch - 1):
        assert single[k] == orc.process_query([ref, ref], queries[k], l2)
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    chains = 3 * (2 if l2 == dp.N else 1)  # of one query
    one_sm = sms // chains
    assert sms < 2 * chains * min(one_sm, batch - 1) and chains * batch > sms
    for nb in (min(one_sm, batch - 1), batch):
        fleet.set_batch(nb)
        assert fleet.process_queries(queries[:nb]) == single[:nb]
        fleet.set_schedule(nb, 4)
        assert fleet.process_queries(queries[:nb]) == single[:nb]
    fleet.close()
