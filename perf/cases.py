"""Workloads of the answer path, each through the calls that a server's program makes.

A case is a dict of plain values; `kind` says which call it is:

  answer   Fleet.process_queries: `queries` requests (host bytes in and out, or device
           tensors with device=True) against a resident database of `entries` entries,
           answered in groups of `batch`.  Requests are drawn as clients send them: a
           uniform index pair, a key and Galois keys of the client's own.
  refresh  new payloads for the `shards` shards of a small database: pack_payloads,
           Fleet.set_shards (encoding and key-switch chain) and the first answer from them.
  shard    one shard: PIRDatabase.set_db, get_a and one perform_pir_split.
  split    PIRDatabase.perform_pir_split against a resident shard, eight queries a call.
  ring     Fleet.perform_double_pir on ring elements, at the small dimensions too.
  serve    Server: requests of session clients to two databases, submitted at once and
           waited for.

Payloads are 2560 uniform bytes an entry.  `distinct` shards are stored and the logical
shard k is served by k mod distinct, so a pass still streams every logical shard (the
stored ones exceed the L2 many times over wherever a database has that many shards).
Outputs are bytes and whole numbers, so `exact` has nothing to give: they are equal or wrong.
"""
import math
import random

import numpy as np
import torch

import dnspir_b200 as dp

MAX_ENTRIES = 1 << 22


def listed():
    return [
        # the library's smallest answer: the ring dimension of the smoke run, one
        # query; launches and host work are all there is
        dict(name="ring_256", kind="ring", log2_n=8, l1=256, l2=64, shards=4, distinct=2, engine="cuda"),
        # a resolver asking a small zone: one request, the answer is waited for
        dict(name="one_2p15", kind="answer", entries=1 << 15, distinct=4, engine="tensor", batch=1, queries=1,
             device=False),
        # the same on the engine a fleet starts with, at a size that is not a power
        # of two (25 half-size shards)
        dict(name="one_200000_cuda", kind="answer", entries=200000, distinct=8, engine="cuda", batch=1, queries=1,
             device=False),
        # the largest database: the latency of one request
        dict(name="one_2p22", kind="answer", entries=1 << 22, distinct=8, engine="tensor", batch=1, queries=1,
             device=False),
        # the largest database, requests one after the other (the next one's scan
        # runs beside the last one's second level)
        dict(name="stream_2p22", kind="answer", entries=1 << 22, distinct=8, engine="tensor", batch=1, queries=6,
             device=True),
        # a loaded server on the largest database: two groups of 64 with the tile and
        # schedule that its tuner keeps for them
        dict(name="batch64_2p22", kind="answer", entries=1 << 22, distinct=8, engine="tensor", batch=64, queries=128,
             device=False, rows=256, mtiles=2, stages=3, kernel=1, schedule=1),
        # a mid-size database under full load, the largest group, untuned
        dict(name="batch256_2p20", kind="answer", entries=1 << 20, distinct=8, engine="tensor", batch=256, queries=256,
             device=True),
        # a mid-size database of an odd number of shards, ragged groups, untuned
        dict(name="batch37_400000", kind="answer", entries=400000, distinct=7, engine="tensor", batch=37, queries=100,
             device=False),
        # groups on the CUDA-core engine
        dict(name="batch16_2p20_cuda", kind="answer", entries=1 << 20, distinct=8, engine="cuda", batch=16, queries=16,
             device=False),
        # a zone's update: every shard of a 2^15-entry database encoded again, then
        # the first answer
        dict(name="refresh_2p15", kind="refresh", entries=1 << 15, engine="tensor"),
        # one full-size shard through the single-shard calls
        dict(name="shard_2048", kind="shard", log2_n=11, l=2048, seeds=0),
        # a front end serving session clients of two databases
        dict(name="serve_2p15_2p17", kind="serve", entries_a=1 << 15, entries_b=1 << 17, batch=32, requests_a=48,
             requests_b=16, sessions=16),
    ]


# ---- drawn cases

def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _shape(entries):
    return dp.get_database_shape(entries)


def _cost(case):
    """A rough cost of a pass, in the units of shard scans, to keep drawn cases below the listed ones."""
    l1, l2, shards = _shape(case["entries"])
    groups = -(-case["queries"] // case["batch"])
    b = min(case["batch"], case["queries"])
    per = max(1.0, b / 48) if case["engine"] == "tensor" else max(1.0, b / 1.5)
    return groups * shards * (l1 / 2048) * per + case["queries"] * l2 / 512 + groups * l2 / 20


def draw(rng):
    kind = rng.choice(["answer"] * 5 + ["refresh", "shard", "split", "ring", "serve"])
    if kind == "answer":
        limit = 0.55 * max(_cost(c) for c in listed() if c["kind"] == "answer")
        while True:
            engine = rng.choice(["tensor", "tensor", "cuda"])
            queries = _log_int(rng, 1, 256)
            batch = _log_int(rng, 1, queries)
            if engine == "cuda":
                batch = 1 << (batch.bit_length() - 1)
            case = dict(kind=kind, entries=_log_int(rng, 1 << 13, MAX_ENTRIES), engine=engine, batch=batch,
                        queries=queries, device=rng.random() < 0.4)
            case["distinct"] = min(_shape(case["entries"])[2], rng.randint(3, 9))
            if _cost(case) <= limit:
                return case
    if kind == "refresh":
        return dict(kind=kind, entries=_log_int(rng, 1 << 12, 1 << 16), engine=rng.choice(["tensor", "cuda"]))
    if kind in ("shard", "split"):
        log2_n = rng.randint(6, 11)
        l = 1 << rng.choice([log2_n, log2_n - 1, rng.randint(3, log2_n - 1)])
        return dict(kind=kind, log2_n=log2_n, l=l, seeds=rng.randint(0, 1))
    if kind == "ring":
        log2_n = rng.randint(6, 11)
        n = 1 << log2_n
        shards = _log_int(rng, 1, min(40, n // 8))
        lo = max(3, (shards * 8 - 1).bit_length())
        l2 = n if lo >= log2_n else 1 << rng.choice([lo, min(lo + 1, log2_n)])
        l1 = rng.choice([n, n // 2])
        engine = rng.choice(["tensor", "cuda"]) if log2_n >= 8 else "cuda"
        return dict(kind=kind, log2_n=log2_n, l1=l1, l2=l2, shards=shards, distinct=min(shards, rng.randint(1, 4)),
                    engine=engine)
    a = _log_int(rng, 1 << 13, 1 << 17)
    return dict(kind="serve", entries_a=a, entries_b=_log_int(rng, 1 << 13, 1 << 17), batch=rng.choice([8, 16, 32]),
                requests_a=rng.randint(8, 48), requests_b=rng.randint(1, 24), sessions=rng.randint(1, 16))


# ---- states

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _payload(entries, gen):
    return torch.randint(0, 256, (entries, 2560), dtype=torch.uint8, device="cuda", generator=gen)


def _pack(payload):
    out = torch.empty((payload.shape[0], dp.N), dtype=torch.uint16, device="cuda")
    torch.cuda.synchronize()  # the library packs on a stream of its own
    dp.pack_payloads(payload, out)
    return out


def _fill(fleet, distinct, gen):
    per = fleet.entries_per_shard
    for first in range(0, distinct, 8):
        cnt = min(8, distinct - first)
        fleet.set_shards(first, _pack(_payload(cnt * per, gen)).view(cnt, per, dp.N))


def _fleet(entries, distinct, engine, gen):
    fleet = dp.Fleet(entries, distinct)
    if engine == "tensor":
        fleet.set_engine(dp.ENGINE_TENSOR)
    _fill(fleet, fleet.num_distinct, gen)
    return fleet


def _requests(fleet, count, rng):
    return [dp.prepare_query(rng.randbytes(32), rng.randrange(fleet.entries_per_shard),
                             rng.randrange(fleet.num_shards), fleet.primary_order, fleet.secondary_order)[0]
            for _ in range(count)]


def _ring(rng, shape):
    return rng.integers(0, dp.Q, size=shape, dtype=np.uint64)


def _coeffs(shape, gen):
    return torch.randint(0, 1024, shape, dtype=torch.int16, device="cuda", generator=gen).view(torch.uint16)


def prepare(case, seed):
    gen, rng, ring = _gen(seed), random.Random(seed), np.random.default_rng(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "answer":
        fleet = _fleet(case["entries"], case["distinct"], case["engine"], gen)
        fleet.set_batch(case["batch"])
        if "rows" in case:
            tile = (case["rows"], case["mtiles"], case["stages"], case["kernel"])
            fleet.set_tile(case["batch"], dp.tscan_shapes().index(tile))
            fleet.set_schedule(case["batch"], case["schedule"])
        q = _requests(fleet, case["queries"], rng)
        s["fleet"] = fleet
        if case["device"]:
            s["queries"] = torch.from_numpy(np.frombuffer(b"".join(q), np.uint8).reshape(len(q), -1).copy()).cuda()
            s["replies"] = torch.empty((len(q), dp.reply_bytes()), dtype=torch.uint8, device="cuda")
        else:
            s["queries"] = q
    elif kind == "refresh":
        fleet = dp.Fleet(case["entries"])
        if case["engine"] == "tensor":
            fleet.set_engine(dp.ENGINE_TENSOR)
        s["fleet"] = fleet
        s["payload"] = _payload(fleet.num_shards * fleet.entries_per_shard, gen)
        s["coeffs"] = torch.empty((s["payload"].shape[0], dp.N), dtype=torch.uint16, device="cuda")
        s["query"] = _requests(fleet, 1, rng)[0]
    elif kind in ("shard", "split"):
        n, l = 1 << case["log2_n"], case["l"]
        s["db"] = dp.PIRDatabase(case["log2_n"], l, case["seeds"])
        s["entries"] = _coeffs((8 * l, n), gen)
        s["q"] = (_ring(ring, (8, n)), _ring(ring, (8, n)) if l == n else None, _ring(ring, (8, 2, n)))
        torch.cuda.synchronize()
        if kind == "split":
            s["db"].set_db(s["entries"])
    elif kind == "ring":
        n = 1 << case["log2_n"]
        fleet = dp.Fleet.general(case["log2_n"], case["l1"], case["l2"], case["shards"], case["distinct"])
        if case["engine"] == "tensor":
            fleet.set_engine(dp.ENGINE_TENSOR)
        coeffs = _coeffs((case["distinct"], 8 * case["l1"], n), gen)
        torch.cuda.synchronize()
        fleet.set_shards(0, coeffs)
        s["fleet"] = fleet
        s["q"] = (_ring(ring, (n,)), _ring(ring, (n,)) if case["l1"] == n else None, _ring(ring, (n,)),
                  _ring(ring, (n,)) if case["l2"] == n else None, _ring(ring, (2, n)))
    else:
        server = dp.Server(max_sessions=case["sessions"])
        work = []
        for key in ("a", "b"):
            fleet = _fleet(case["entries_" + key], None, "tensor", gen)
            db = server.add_db(fleet, case["batch"])
            count = case["requests_" + key]
            server.set_batching(db, min(count, case["batch"]), 1.0)
            work.append((db, _requests(fleet, count, rng)))
        server.start()
        # a session holds one client's keys; its later requests go without them
        cut = dp.GALOIS_KEY_BYTES
        sessions = [server.open_session(q[:cut]) for q in work[0][1][:case["sessions"]]]
        s["server"] = server
        s["requests"] = [(db, q[cut:] if i < len(sessions) and db == work[0][0] else q,
                          sessions[i] if i < len(sessions) and db == work[0][0] else -1)
                         for db, qs in work for i, q in enumerate(qs)]
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "answer":
        if s["case"]["device"]:
            s["fleet"].process_queries_device(s["queries"], s["replies"])
            return s["replies"]
        return np.frombuffer(b"".join(s["fleet"].process_queries(s["queries"])), np.uint8)
    if kind == "refresh":
        fleet = s["fleet"]
        dp.pack_payloads(s["payload"], s["coeffs"])
        fleet.set_shards(0, s["coeffs"].view(fleet.num_shards, fleet.entries_per_shard, dp.N))
        return np.frombuffer(fleet.process_query(s["query"]), np.uint8)
    if kind == "shard":
        s["db"].set_db(s["entries"])
        return s["db"].get_a().view(np.int64), s["db"].perform_pir_split(*s["q"]).view(np.int64)
    if kind == "split":
        return s["db"].perform_pir_split(*s["q"]).view(np.int64)
    if kind == "ring":
        return s["fleet"].perform_double_pir(*s["q"]).view(np.int64)
    server = s["server"]
    tickets = [server.submit(db, q, session) for db, q, session in s["requests"]]
    return np.frombuffer(b"".join(server.wait(t) for t in tickets), np.uint8)


# ---- the work of a pass

# words of a preprocessed shard that an answer reads, per row, factor, slot and lane:
# the entry and two key digits, which one linear relation along the rows ties together
WORDS = 2


def _loop(l, n):
    return min(l, n // 2) * (2 if l == n else 1)


def _scan(n, l1, shards, groups, queries):
    """(bytes, operations) of the first level: every shard once a group, a multiply-add per word and query."""
    words = 2 * WORDS * _loop(l1, n) * n * 8 * shards
    return 4 * words * groups, 2 * words * queries


def _chain(n, l, chains):
    """Operations of a key-switch chain: four length-n transforms and six products per slot and row, in both factors."""
    return chains * _loop(l, n) * (4 * (n // 2) * int(math.log2(n)) + 2 * 6 * n) * 2


def _encode(n, l, lanes):
    """Operations of set_db's transforms: columns, rows and three lifts per entry column."""
    one = n // 2 * int(math.log2(n)) * 2
    return lanes * (l + n + 3 * _loop(l, n)) * one


def _answer_work(n, l1, l2, shards, groups, queries, io):
    b, f = _scan(n, l1, shards, groups, queries)
    return {"bytes": b + io, "flops": f + queries * (_chain(n, l2, 3) + _encode(n, l2, 3))}


def work(case):
    kind = case["kind"]
    if kind == "answer":
        l1, l2, shards = _shape(case["entries"])
        io = case["queries"] * (dp.query_bytes(l1, l2) + dp.reply_bytes())
        return _answer_work(dp.N, l1, l2, shards, -(-case["queries"] // case["batch"]), case["queries"], io)
    if kind == "refresh":
        l1, l2, shards = _shape(case["entries"])
        w = _answer_work(dp.N, l1, l2, shards, 1, 1, dp.query_bytes(l1, l2) + dp.reply_bytes())
        slab = _scan(dp.N, l1, shards, 1, 1)[0]
        return {"bytes": w["bytes"] + slab + shards * 8 * l1 * (2560 + 4 * dp.N),
                "flops": w["flops"] + _chain(dp.N, l1, 8 * shards) + _encode(dp.N, l1, 8 * shards)}
    if kind in ("shard", "split"):
        n, l = 1 << case["log2_n"], case["l"]
        b, f = _scan(n, l, 1, 1, 1)
        io = 8 * n * 8 * (4 + (l == n))
        if kind == "shard":
            return {"bytes": 2 * b + io + 8 * n * 8 + 8 * l * n * 2, "flops": f + _chain(n, l, 8) + _encode(n, l, 8)}
        return {"bytes": b + io, "flops": f}
    if kind == "ring":
        n = 1 << case["log2_n"]
        return _answer_work(n, case["l1"], case["l2"], case["shards"], 1, 1, 8 * n * 12)
    total = {"bytes": 0, "flops": 0}
    for key in ("a", "b"):
        l1, l2, shards = _shape(case["entries_" + key])
        q = case["requests_" + key]
        w = _answer_work(dp.N, l1, l2, shards, -(-q // case["batch"]), q, q * (dp.query_bytes(l1, l2) + dp.reply_bytes()))
        total = {k: total[k] + w[k] for k in total}
    return total


def exact(case, seed):
    """Outputs are bytes and whole numbers: there is no rounding to measure."""
    return None
