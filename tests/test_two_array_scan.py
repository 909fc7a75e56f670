"""The scan over two stored arrays a row instead of the reference's three
(main_pir_loop, crates/pir/src/base_pir.rs:1085-1247).

On the CPU: the chain that makes the key digits (preprocess / partial_gal,
base_pir.rs:496-594, 782-863) ties the three arrays, and a sum over the chain
states and the high digits with adjusted query vectors equals the sum over
entries and both digits, with the oracle's own arrays.  On the GPU: a-parts
with a zero among the query polynomial's slots, where the entries do not follow
from the states, fall back to three arrays; the same shards and fleets change
layout with the a-parts installed.  Everything is exact: the tolerance is zero.
"""
import numpy as np
import pytest

import dnspir_b200 as dp
from oracle import oracle as orc

PRIMES = ((1 << 26) - (1 << 12) + 1, (1 << 25) - (1 << 12) + 1)


def _slots(poly, log2n, pi):
    """Natural-order transform: slot s is the value at zeta^-(2s+1)."""
    n, p = 1 << log2n, PRIMES[pi]
    z = pow(int(orc.zeta(log2n, pi)), p - 2, p)
    pw = [pow(z, k, p) for k in range(2 * n)]
    idx = (np.arange(n)[None, :] * (2 * np.arange(n)[:, None] + 1)) % (2 * n)
    m = np.array(pw, dtype=np.int64)[idx]
    return (m * (np.asarray(poly, dtype=np.int64) % p)[None, :] % p).sum(axis=1) % p


@pytest.mark.parametrize("log2n,l,seeds", [(3, 8, 0), (3, 4, 1), (4, 2, 0), (6, 64, 0), (6, 64, 1), (6, 32, 0), (6, 8, 1)])
def test_two_arrays_carry_the_scan(log2n, l, seeds):
    n = 1 << log2n
    rng = np.random.default_rng(l + seeds)
    d = orc.Database(log2n, l, seeds)
    d.set_db(rng.integers(0, orc.T, size=(8 * l, n), dtype=np.uint16))
    ap = orc.aparts(log2n)
    idx5 = np.array([((5 * (2 * j + 1)) % (2 * n) - 1) // 2 for j in range(n)])  # slot of 5 (2j+1)
    inv5 = np.argsort(idx5)
    for pi, p in enumerate(PRIMES):
        ga0, ga1 = (_slots(ap[i], log2n, pi)[:, None] for i in (0, 1))
        gk0, gk1 = (rng.integers(0, p, (n, 1)) for _ in range(2))
        c26 = (1 << 26) % p
        kappa = (ga1 - c26 * ga0) % p
        for h in range(2 if l == n else 1):
            qa = _slots(ap[2 + 2 * seeds + h], log2n, pi)[:, None]
            q = rng.integers(0, p, (n, 1))
            E, G0, G1 = (d.array(w, h, pi).astype(np.int64) % p for w in range(3))
            L = E.shape[0]
            # the states: a_(i+1) = G0 gk_a0 + G1 gk_a1 + E qry_a, and G0 = sigma_5(a) - 2^26 G1
            X = (G0 * ga0 % p + G1 * ga1 % p + E * qa % p) % p
            t = np.concatenate([np.zeros((1, n, 8), np.int64), X[:-1, idx5]])
            assert np.array_equal(G0, (t - c26 * G1) % p)
            inv = np.array([[pow(int(v), p - 2, p)] for v in qa[:, 0]])
            assert np.all(qa * inv % p == 1)
            r = q * inv % p
            C = (gk0 - ga0 * r) % p
            VX, VG = (r + C[inv5]) % p, (gk1 - c26 * gk0 - kappa * r % p) % p
            three, two = np.zeros((n, 8), np.int64), np.zeros((n, 8), np.int64)
            for i in range(L):
                k = pow(5, L - 1 - i, 2 * n)
                j = np.array([((k * (2 * u + 1)) % (2 * n) - 1) // 2 for u in range(n)])
                three += (E[i] * q % p + G0[i] * gk0 % p + G1[i] * gk1 % p)[j] % p
                two += (X[i] * VX % p + G1[i] * VG % p)[j] % p
            two -= X[L - 1] * C[inv5] % p
            assert np.array_equal(three % p, two % p)


def _parity(fleet, db, refs, ref, l2, log2n, seed):
    n = 1 << log2n
    rng = orc.Rng(bytes([seed]) * 32)
    sk = orc.gen_sk(rng, log2n)
    args = orc.enc_double_pir(rng, log2n, refs[0].l, l2, sk, 5, 1)
    assert np.array_equal(fleet.perform_double_pir(*args).astype(np.int64), orc.perform_double_pir(refs, l2, *args))
    gen = np.random.default_rng(seed)
    qb = gen.integers(0, orc.Q, size=(8, n), dtype=np.int64)
    qc = gen.integers(0, orc.Q, size=(8, n), dtype=np.int64) if refs[0].conj else None
    gk = gen.integers(0, orc.Q, size=(8, 2, n), dtype=np.int64)
    assert np.array_equal(db.perform_pir_split(qb, qc, gk).astype(np.int64), ref.perform_pir_split(qb, qc, gk))


@pytest.mark.gpu
@pytest.mark.parametrize("engine", [dp.ENGINE_CUDA_CORES, dp.ENGINE_TENSOR])
@pytest.mark.parametrize("l1,zero", [(256, 2), (256, 3), (128, 2)])
def test_a_parts_with_zero_slots_fall_back_to_three_arrays(engine, l1, zero):
    log2n, n, l2 = 8, 256, 16
    data = np.random.default_rng(3).integers(0, orc.T, size=(2, 8 * l1, n), dtype=np.uint16)
    fleet = dp.Fleet.general(log2n, l1, l2, 2)
    fleet.set_engine(engine)
    db = dp.PIRDatabase(log2n, l1)
    two = fleet.slab_bytes
    parts = dp.get_a_parts(log2n).copy()
    parts[zero] = 0  # FirstSet query (2) or its conjugate (3): every slot is zero
    try:
        for step, ap in enumerate((None, parts, None)):
            dp.set_a_parts(log2n, ap)
            orc.set_aparts(log2n, ap)
            fleet.set_shards(0, data)
            db.set_db(data[0])
            assert fleet.slab_bytes == (two if ap is None else two // 2 * 3)
            refs = []
            for s in range(2):
                refs.append(orc.Database(log2n, l1))
                refs[s].set_db(data[s])
            assert np.array_equal(db.get_a().astype(np.int64), refs[0].get_a())
            _parity(fleet, db, refs, refs[0], l2, log2n, 7 + step)
    finally:
        dp.set_a_parts(log2n, None)
        orc.set_aparts(log2n, None)
    fleet.close()
    db.close()


@pytest.mark.gpu
@pytest.mark.parametrize("log2n,l,seeds", [(3, 8, 0), (3, 1, 1), (5, 16, 0), (7, 128, 1), (9, 256, 0), (10, 1024, 0), (11, 8, 1),
                                           (11, 1024, 0)])
def test_split_matches_oracle_over_shapes(log2n, l, seeds):
    n = 1 << log2n
    gen = np.random.default_rng(log2n * 31 + l)
    data = gen.integers(0, orc.T, size=(8 * l, n), dtype=np.uint16)
    db, ref = dp.PIRDatabase(log2n, l, seeds), orc.Database(log2n, l, seeds)
    db.set_db(data)
    ref.set_db(data)
    assert np.array_equal(db.get_a().astype(np.int64), ref.get_a())
    qb = gen.integers(0, orc.Q, size=(8, n), dtype=np.int64)
    qc = gen.integers(0, orc.Q, size=(8, n), dtype=np.int64) if l == n else None
    gk = gen.integers(0, orc.Q, size=(8, 2, n), dtype=np.int64)
    assert np.array_equal(db.perform_pir_split(qb, qc, gk).astype(np.int64), ref.perform_pir_split(qb, qc, gk))
    db.close()


def _wire_fleet(l2, shards=2):
    l1 = 1024
    data = np.random.default_rng(l2).integers(0, orc.T, size=(1, 8 * l1, 2048), dtype=np.uint16)
    fleet = dp.Fleet.general(11, l1, l2, shards, 1)
    fleet.set_engine(dp.ENGINE_TENSOR)
    fleet.set_shards(0, data)
    return fleet, data


@pytest.mark.gpu
@pytest.mark.parametrize("l2,groups", [(2048, (24, 25, 75)), (1024, (49, 50)), (16, (50,))])
def test_chain_forms_give_the_same_replies(l2, groups):
    # one part per block up to one block per SM, three parts per block beyond
    # it, a second chunk beyond one wave
    fleet, _ = _wire_fleet(l2)
    rng = orc.Rng(bytes([l2 % 251]) * 32)
    queries = [orc.prepare_query(rng, (97 * k) % 8192, k % 2, 1024, l2)[0] for k in range(max(groups))]
    single = fleet.process_queries(queries)
    for nb in groups:
        fleet.set_batch(nb)
        assert fleet.process_queries(queries[:nb]) == single[:nb]
    fleet.close()


@pytest.mark.gpu
def test_secondary_a_parts_with_zero_slots():
    # the chains whose b part carries the entries serve a-parts without inverses
    l2 = 16
    parts = dp.get_a_parts(11).copy()
    parts[4] = 0  # SecondSet query
    try:
        dp.set_a_parts(11, parts)
        orc.set_aparts(11, parts)
        fleet, data = _wire_fleet(l2)
        ref = orc.Database(11, 1024)
        ref.set_db(data[0])
        rng = orc.Rng(bytes(range(32)))
        queries = [orc.prepare_query(rng, 31 * k, k % 2, 1024, l2)[0] for k in range(60)]
        want = [orc.process_query([ref, ref], q, l2) for q in queries[:3]]
        for batch in (1, 60):
            fleet.set_batch(batch)
            got = fleet.process_queries(queries)
            assert got[:3] == want
            assert batch == 1 or got == first
            first = got
        fleet.close()
    finally:
        dp.set_a_parts(11, None)
        orc.set_aparts(11, None)


@pytest.mark.gpu
@pytest.mark.parametrize("l2", [8, 16, 32, 64, 128, 256, 512, 1024])
def test_secondary_orders_match_oracle(l2):
    # every length of the encoder's subgroup transforms, with zero columns
    # above the shards' (one shard, or as many as the order takes up to three)
    shards = min(3, l2 // 8)
    fleet, data = _wire_fleet(l2, shards)
    ref = orc.Database(11, 1024)
    ref.set_db(data[0])
    rng = orc.Rng(bytes([7, l2 % 256]) * 16)
    queries = [orc.prepare_query(rng, 1000 + k, k % shards, 1024, l2)[0] for k in range(2)]
    fleet.set_batch(2)
    assert fleet.process_queries(queries) == [orc.process_query([ref] * shards, q, l2) for q in queries]
    fleet.close()
