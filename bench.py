#!/usr/bin/env python
"""bench.py -- PIR responses/s, p50/p99 response ms and DB-scan HBM GB/s at
2^22 entries (the reference's `bench --db-entries 4194304`,
crates/pir/src/pir_wrapper.rs:493-615) on B200s.

Workload (one GPU): 2^22 entries of 2560 B, laid out by get_database_shape
(256 full shards of 512 MiB as stored, secondary group of order 2048).  As many distinct
shards as fit in HBM are preprocessed on the GPU from seeded uniform payloads
and logical shard k is served by distinct shard k mod D, as the reference's
--preprocessed-db-count does (pir_wrapper.rs:578).  A step is one query
answered, one query per launch sequence (the plain path): decode, scan of all
256 shards (137 GB), epilogue, secondary database build + key-switch chain,
reply.  Every answer is decrypted by the client and compared with the stored
entry.  The scan runs on the tensor engine (8-bit limb products on tcgen05)
unless --engine cuda selects the CUDA-core engine; both give the same replies.

After the plain run, on the same fleet:
  * the reference bench's own 16 (primary, secondary) index pairs
    (pir_wrapper.rs:562, secondary index j mod S), answered and decrypted;
  * groups of B queries per pass over the slabs (--batched, default 16, 64,
    128 and 256; tile shape and schedule per B from the autotuner):
    responses/s, p50/p99 per-query latency and the scan's effective GB/s
    (B x slab bytes / scan time) in the "batched" object.
Then, with the 2^22 fleet released (unless --quick):
  * "config1": 2^15 entries (4 half shards on 2 distinct), the reference
    bench's 16 index pairs one query per launch sequence, through host
    buffers and as one group; the CPU leg compares the replies with the
    oracle's bytes (cpu_baseline.config1);
  * "config3" / "config4": 2^20 entries (64 full shards, all resident) on the
    CUDA-core and on the tensor engine, groups of 16, 64 and 256;
  * "served": the served mix for a few seconds at 5000 queries/s (below).

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]
                  [--engine tensor|cuda] [--batched 16,64,128,256] [--quick]
  python bench.py --serve [--serve-rate 5000] [--serve-seconds 10]

--serve measures the served mix alone: four resident databases (2^15,
2^18, 2^20 and 2^22 entries; the last on as many distinct shards as fit),
open-loop Poisson arrivals at the given total rate split by --serve-mix,
answered by the serving loop (continuous batching, CUDA graphs, half of the
clients on device-resident sessions).  One JSON line: responses/s delivered
and p50/p99 submit-to-reply latency per database.

--gpus N > 1 runs under torchrun: every rank holds a replica of the database
and answers its own queries (queries are the units; no data-path collective),
value = all ranks' responses / max-over-ranks device time.
--impl reference times the CPU restatement of the reference's answer path
(oracle/; the reference itself is Rust and cannot be built here) on the host
cores, rank 0 only: every step is one whole query (all shards scanned, then
the secondary phase), timed for real.
"""
import argparse
import datetime
import hashlib
import json
import os
import re
import statistics
import subprocess
import sys
import tempfile
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import numpy as np

ENTRIES_DEFAULT = 1 << 22
PAYLOAD = 2560
REF_RESPONSE_S_8T = 4.3  # ARTIFACT-APPENDIX.md:122 (2^22 x 2560 B, 8 threads, Xeon Gold 5318S)
METRIC = "pir_responses_per_sec_2p22"
# the tensor scan kernel of a tile shape (its fourth field)
TILE_KERNELS = ("tscan_kernel (one tile per CTA)", "tscanp_kernel (persistent)",
                "tscan2_kernel (CTA pair, relayed bulk copies)", "tscan2_kernel (CTA pair, tensor-map copies)")
UNIT = "responses/s"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=16)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--entries", type=int, default=ENTRIES_DEFAULT)
    ap.add_argument("--distinct", type=int, default=0, help="distinct shards in HBM (0 = as many as fit)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--engine", default="tensor", choices=["tensor", "cuda"])
    ap.add_argument("--batched", default="16,64,128,256", help="comma-separated group sizes measured after the plain run")
    ap.add_argument("--quick", action="store_true", help="skip the 2^20 and served-mix legs")
    ap.add_argument("--tile", default="", help="B:shape[:schedule],... force a tensor tile shape (and pipeline "
                    "schedule) for group size B (no tuning)")
    ap.add_argument("--cpu-distinct", type=int, default=4, help="distinct shard slabs in host RAM for the CPU arm")
    ap.add_argument("--batched-groups", type=int, default=3, help="timed groups per batched size")
    ap.add_argument("--reserve-gib", type=float, default=0.0, help="HBM left free for workspaces (0: from the group sizes)")
    ap.add_argument("--serve", action="store_true", help="served mix over four databases instead")
    ap.add_argument("--serve-rate", default="5000", help="offered queries/s (comma-separated for several runs)")
    ap.add_argument("--serve-seconds", type=float, default=10.0)
    ap.add_argument("--serve-mix", default="0.7,0.2,0.08,0.02", help="shares of 2^15, 2^18, 2^20, 2^22")
    ap.add_argument("--serve-clients", type=int, default=64, help="distinct clients per database")
    return ap.parse_args()


class RankGroup:
    """The ranks of a torchrun launch: replicas, one GPU each, whose only
    collectives are a barrier around the timed region and the max of the
    per-rank times (no data-path collective)."""

    def __init__(self, pg, device):
        self.pg = pg
        self.device = device

    @classmethod
    def init(cls, backend, world, timeout_s=600):
        if world <= 1:
            return cls(None, "cpu")
        import torch.distributed as tdist
        from datetime import timedelta
        tdist.init_process_group(backend, timeout=timedelta(seconds=timeout_s))
        return cls(tdist, "cuda" if backend == "nccl" else "cpu")

    def barrier(self):
        if self.pg:
            self.pg.barrier()

    def max(self, x):
        if not self.pg:
            return x
        import torch
        t = torch.tensor([x], dtype=torch.float64, device=self.device)
        self.pg.all_reduce(t, op=self.pg.ReduceOp.MAX)
        return float(t.item())


def whole_job_rate(units_per_rank, world, max_seconds):
    """Units all ranks processed / the slowest rank's time."""
    return units_per_rank * world / max_seconds


def dist_env():
    return int(os.environ.get("RANK", "0")), int(os.environ.get("LOCAL_RANK", "0")), int(os.environ.get("WORLD_SIZE", "1"))


def measured_peak_hbm():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def _gemm_rate(torch, fn, n, seconds):
    """Median rate (POPS, 2 ops per MAC) of the second half of 20-call
    batches of an n^3 GEMM called back to back for about `seconds`."""
    fn()
    torch.cuda.synchronize()
    rates, t_end = [], time.time() + seconds
    while time.time() < t_end:
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(20):
            fn()
        e1.record()
        e1.synchronize()
        rates.append(20 * 2.0 * n ** 3 / (e0.elapsed_time(e1) * 1e-3) / 1e15)
    return statistics.median(rates[len(rates) // 2:]), len(rates)


def int8_tensor_peak(torch, dev, n=8192, seconds=1.5):
    """Sustained 8-bit tensor throughput of library GEMMs on this GPU, the
    denominator of the batched scan's tensor fraction: cuBLASLt through
    torch._int_mm (n^3, s8 x s8 -> s32) and through torch._scaled_mm (n^3,
    e4m3 x e4m3 -> bf16, the same nominal tensor rate), each called back to
    back for about `seconds` (long enough to settle under the power cap, as
    the batched scan does).  `pops` is the faster of the two; None if neither
    GEMM is available."""
    out = {"gemm_n": n, "seconds": seconds}
    try:
        a = torch.randint(-128, 128, (n, n), dtype=torch.int8, device=dev)
        b = torch.randint(-128, 128, (n, n), dtype=torch.int8, device=dev).t()  # column-major operand
        out["int8_pops"], _ = _gemm_rate(torch, lambda: torch._int_mm(a, b), n, seconds)
        del a, b
    except Exception as e:  # noqa: BLE001 -- reported, not fatal
        out["int8_error"] = str(e).splitlines()[0][:200]
    try:
        a = torch.randn(n, n, device=dev).to(torch.float8_e4m3fn)
        b = torch.randn(n, n, device=dev).to(torch.float8_e4m3fn).t()
        one = torch.ones((), device=dev)
        out["fp8_pops"], _ = _gemm_rate(
            torch, lambda: torch._scaled_mm(a, b, scale_a=one, scale_b=one, out_dtype=torch.bfloat16), n, seconds)
        del a, b
    except Exception as e:  # noqa: BLE001
        out["fp8_error"] = str(e).splitlines()[0][:200]
    torch.cuda.empty_cache()
    rates = [out[k] for k in ("int8_pops", "fp8_pops") if k in out]
    out["pops"] = max(rates) if rates else None
    return out


def stored_shard_bytes(dp, l1, device=0):
    """Bytes of one preprocessed shard as a fleet stores it (one pass of the scan reads them once)."""
    probe = dp.Fleet.general(dp.LOG2_N, l1, 8, 1, device=device)
    n = probe.slab_bytes
    probe.close()
    return n


def profiled_traffic(name, algo_bytes):
    """dram bytes per launch from a committed ncu summary (profiles/<name>):
    its measured ratio of dram bytes to algorithmic bytes (the captured launch
    reads each slab block once, so traffic grows with the slabs) times this
    launch's algorithmic bytes; None without a summary."""
    p = os.path.join(ROOT, "profiles", name)
    try:
        for line in open(p):
            m = re.match(r"\s*traffic_ratio:\s*([0-9.eE+]+)", line)
            if m:
                return float(m.group(1)) * algo_bytes
    except OSError:
        pass
    return None


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms.  It is
    started before the warm-up (its own start-up, which queries the driver,
    stays out of the timed region) and stopped after; stop() keeps the samples
    whose timestamps fall inside the timed region (host clock), or the one
    nearest to it when the region is shorter than a sampling period."""

    FIELDS = ("timestamp,index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu):
        self.gpu = gpu
        self.proc = None
        self.out = tempfile.NamedTemporaryFile(prefix="clocks", suffix=".csv", delete=False)

    def start(self, settle_s=3.0):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), "--query-gpu=" + self.FIELDS,
                                          "--format=csv,noheader,nounits", "-lms", "200"], stdout=self.out,
                                         stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None
            return
        t_end = time.time() + settle_s  # until the first sample is written
        while time.time() < t_end and os.path.getsize(self.out.name) == 0:
            time.sleep(0.05)

    def stop(self, window=None):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
        self.out.close()
        rows = []
        try:
            for line in open(self.out.name):
                parts = [x.strip() for x in line.split(",")]
                if len(parts) >= 10:
                    try:
                        parts[0] = datetime.datetime.strptime(parts[0], "%Y/%m/%d %H:%M:%S.%f").timestamp()
                    except ValueError:
                        continue
                    rows.append(parts)
        finally:
            os.unlink(self.out.name)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        where = "timed region"
        if window is not None:
            inside = [r for r in rows if window[0] - 0.1 <= r[0] <= window[1] + 0.1]
            if not inside:
                mid = 0.5 * (window[0] + window[1])
                inside = [min(rows, key=lambda r: abs(r[0] - mid))]
                where = "nearest sample to the timed region"
            rows = inside
        sm = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        smax = [float(r[3]) for r in rows if r[3].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if r[6 + i].lower().startswith("active")})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "reasons": reasons, "samples": len(rows), "sampled": where}


def pack_host(payload):
    """pack_bytes_into_coeffs (dns/bucket.rs:289-303) of one 2560-byte entry."""
    b = np.frombuffer(payload, dtype=np.uint8).reshape(-1, 5).astype(np.uint64)
    v = b[:, 0] | (b[:, 1] << 8) | (b[:, 2] << 16) | (b[:, 3] << 24) | (b[:, 4] << 32)
    out = np.stack([(v >> s) & 1023 for s in (0, 10, 20, 30)], axis=1).reshape(-1)
    return out.astype(np.uint16)


def shard_payload(torch, d, entries_per_shard, device, seed0=1000):
    g = torch.Generator(device=device)
    g.manual_seed(seed0 + d)
    return torch.randint(0, 256, (entries_per_shard, PAYLOAD), dtype=torch.uint8, device=device, generator=g)


def group_sizes(cap):
    """The group sizes the server forms: 1, 2, 3, 4, 6, 8, 12, ... (powers of
    two and 1.5 times powers of two) up to cap, and cap."""
    out, p = {cap}, 1
    while p < cap:
        out.add(p)
        if p >= 2 and p + p // 2 < cap:
            out.add(p + p // 2)
        p *= 2
    return sorted(out)


def serve_mix(args, local_rank, rates, seconds):
    """The served mix (continuous batching over four resident databases) at
    each offered rate for `seconds`: (per-rate results, preprocessing s).
    Raises RuntimeError when a sampled reply fails decryption."""
    import torch
    import dnspir_b200 as dp
    dev = torch.device("cuda", local_rank)
    sizes = [1 << 15, 1 << 18, 1 << 20, 1 << 22]
    shares = [float(x) for x in args.serve_mix.split(",")]
    batch_cap = {1 << 15: 256, 1 << 18: 256, 1 << 20: 128, 1 << 22: 64}
    # batching window (min pending queries, max wait ms): cheap databases wait
    # briefly for fuller groups instead of launching near-empty ones
    batch_window = {1 << 15: (32, 4.0), 1 << 18: (16, 8.0), 1 << 20: (8, 16.0), 1 << 22: (1, 0.0)}
    fleets, shapes, distinct = [], [], []
    t0 = time.time()
    for e in sizes:
        l1, l2, shards = dp.get_database_shape(e)
        slab = stored_shard_bytes(dp, l1, local_rank)
        free, _ = torch.cuda.mem_get_info()
        d = shards if e < (1 << 22) else max(1, min(shards, int((free - (40 << 30)) // slab)))
        f = dp.Fleet(e, d, device=local_rank)
        f.set_engine(dp.ENGINE_TENSOR)
        for first in range(0, d, 8):
            cnt = min(8, d - first)
            co = torch.empty((cnt, 8 * l1, dp.N), dtype=torch.uint16, device=dev)
            for i in range(cnt):
                dp.pack_payloads(shard_payload(torch, first + i, 8 * l1, dev, seed0=7000 + 100 * sizes.index(e)),
                                 co[i], device=local_rank)
            f.set_shards(first, co)
            del co
        fleets.append(f)
        shapes.append((l1, l2, shards))
        distinct.append(d)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    prep_s = time.time() - t0
    # client pools: full queries, and for half of the clients a session (keys sent once)
    gk = dp.GALOIS_KEY_BYTES
    pools = []
    for di, (l1, l2, shards) in enumerate(shapes):
        rng = np.random.default_rng(100 + di)
        pool = []
        for c in range(args.serve_clients):
            i, j = int(rng.integers(0, 8 * l1)), int(rng.integers(0, shards))
            q, sk = dp.prepare_query(hashlib.sha256(f"serve-{di}-{c}".encode()).digest(), i, j, l1, l2)
            pool.append((q, sk, i, j))
        pools.append(pool)
    results = []
    for rate in rates:
        sv = dp.Server(max_sessions=2 * args.serve_clients * len(sizes), device=local_rank)
        ids = [sv.add_db(f, batch_cap[e]) for f, e in zip(fleets, sizes)]
        for i, e in zip(ids, sizes):
            sv.set_batching(i, *batch_window[e])
        sv.start(graphs=True)
        sessions = [[sv.open_session(q[:gk]) if c % 2 else -1 for c, (q, _, _, _) in enumerate(pool)]
                    for pool in pools]
        # warm-up, outside the timed window: per database two bursts of every
        # group size the server forms (1, 2, 3, 4, 6, 8, 12, ... up to the
        # admitted maximum), so that every kernel the mix uses is loaded and
        # each size's graphs are captured on both buffer slots
        for di in range(len(sizes)):
            cap = batch_cap[sizes[di]]
            for n in group_sizes(cap):
                for _ in range(2):
                    wt = [sv.submit(ids[di], pools[di][c % len(pools[di])][0]) for c in range(n)]
                    for t in wt:
                        sv.wait(t, timeout_ms=600000)
        base = [sv.stats(i) for i in ids]
        arrivals = np.random.default_rng(7)
        n_total = int(rate * seconds)
        gaps = arrivals.exponential(1.0 / rate, size=n_total)
        which = arrivals.choice(len(sizes), size=n_total, p=np.array(shares) / sum(shares))
        clients = arrivals.integers(0, args.serve_clients, size=n_total)
        tickets = []
        t_start = time.perf_counter()
        t_next = t_start
        for k in range(n_total):
            t_next += gaps[k]
            while True:
                dt = t_next - time.perf_counter()
                if dt <= 0:
                    break
                if dt > 2e-4:
                    time.sleep(dt - 1e-4)
            di, c = int(which[k]), int(clients[k])
            q = pools[di][c][0]
            s = sessions[di][c]
            tickets.append((di, c, sv.submit(ids[di], q[gk:] if s >= 0 else q, session=s)))
        t_submitted = time.perf_counter()
        ok, bad = 0, 0
        checked = set()
        for di, c, t in tickets:
            r = sv.wait(t, timeout_ms=600000)
            if (di, c) not in checked and len(checked) < 32:
                checked.add((di, c))
                q, sk, i, j = pools[di][c]
                want = pack_host(shard_payload(torch, j % distinct[di], 8 * shapes[di][0], dev,
                                               seed0=7000 + 100 * di)[i].cpu().numpy().tobytes())
                if np.array_equal(dp.process_reply(r, sk), want):
                    ok += 1
                else:
                    bad += 1
        t_end = time.perf_counter()
        per_db = {}
        for di, e in enumerate(sizes):
            st = sv.stats(ids[di])
            lat = st["latencies_ms"][len(base[di]["latencies_ms"]):]  # drop the warm-up groups
            per_db[f"2^{e.bit_length() - 1}"] = {
                "offered_per_sec": rate * shares[di] / sum(shares), "completed": int(len(lat)),
                "p50_ms": float(np.percentile(lat, 50)) if len(lat) else None,
                "p99_ms": float(np.percentile(lat, 99)) if len(lat) else None,
                "admitted_batch": st["admitted_batch"], "groups": st["groups"] - base[di]["groups"],
                "graph_groups": st["graph_groups"] - base[di]["graph_groups"], "distinct_shards": distinct[di],
                "shards": shapes[di][2]}
        sv.stop()
        sv.close()
        if bad:
            for f in fleets:
                f.close()
            raise RuntimeError(f"served mix: {bad} of {ok + bad} sampled replies failed decryption")
        results.append({"offered_per_sec": rate, "responses_per_sec": n_total / (t_end - t_start),
                        "submit_seconds": t_submitted - t_start, "drain_seconds": t_end - t_submitted,
                        "per_db": per_db, "checked": {"decrypted_ok": ok, "of": ok + bad}})
    for f in fleets:
        f.close()
    return results, prep_s


def run_serve(args, rank, local_rank):
    """--serve: the served mix alone, one JSON line."""
    import torch
    if rank != 0:
        return 0
    torch.cuda.set_device(local_rank)
    shares = [float(x) for x in args.serve_mix.split(",")]
    try:
        results, prep_s = serve_mix(args, local_rank, [float(r) for r in args.serve_rate.split(",")],
                                    args.serve_seconds)
    except RuntimeError as e:
        print(json.dumps({"error": str(e)}), flush=True)
        return 1
    line = {"metric": "served_mix_responses_per_sec", "value": results[0]["responses_per_sec"],
            "unit": "responses/s", "n_gpus": 1, "higher_is_better": True, "dtype": "u32", "data": "synthetic",
            "config": {"workload": "served mix: Poisson arrivals over four resident databases (2^15, 2^18, 2^20, "
                                   "2^22 entries x 2560 B), continuous batching, CUDA graphs, half of the clients "
                                   "on device-resident sessions", "mix": shares, "clients_per_db": args.serve_clients,
                                   "seconds": args.serve_seconds, "engine": "tensor"},
            "runs": results, "preprocess_s": prep_s,
            "latency_note": "submit-to-reply wall time on the host, queueing included"}
    print(json.dumps(line), flush=True)
    return 0


def workload_config(entries, l1, l2, shards, world):
    """The workload of the headline line, identical in both arms."""
    return {
        "workload": f"plain two-level PIR answer, one query per step, {entries} entries x 2560 B ({shards} shards of "
                    f"group order {l1}, secondary group order {l2})",
        "entries": entries, "shards": shards, "primary_order": l1, "secondary_order": l2,
        "query_bytes": 2 * 2048 * 50 // 8 + (2 if l1 == 2048 else 1) * 2048 * 34 // 8 +
                       (2 if l2 == 2048 else 1) * 2048 * 34 // 8,
        "reply_bytes": 22272,
        "l2": "inputs larger than L2 (each step streams every shard slab: 137 GB at 2^22)",
        "parallelism": f"replica x{world}" if world > 1 else "single process"}


def cpu_query_steps(l1, l2, shards, distinct, warmup, steps):
    """One whole query per step on the host cores (oracle/scan_baseline.cpp):
    the AVX-512 main_pir_loop restatement over every logical shard (distinct
    slabs in RAM, shard k -> k mod distinct) on all threads, then the
    oracle's secondary phase.  Returns per-step (scan s, secondary s) and the
    scan's thread count."""
    from oracle import oracle as orc
    threads = os.cpu_count() or 1
    orc.set_num_threads(threads)
    qb = orc.QueryBench(11, l1, l2, shards, min(distinct, shards))
    try:
        for _ in range(warmup):
            qb.step(threads)
        out, used = [], threads
        for _ in range(steps):
            a, b, used = qb.step(threads)
            out.append((a, b))
    finally:
        qb.close()
    return out, used


def cpu_sample_text(l1, l2, shards, distinct, steps, used, scan_s, sec_s):
    from oracle import oracle as orc
    return (f"{steps} whole queries timed for real: main_pir_loop restatement (AVX-512 op sequence, "
            f"{'AVX-512 present' if orc.cpu_has_avx512() else 'NO AVX-512: scalar loop'}) over all {shards} shards "
            f"({min(distinct, shards)} distinct slabs in host RAM, shard k -> k mod {min(distinct, shards)}) on {used} "
            f"threads, {scan_s:.2f} s per query, then the secondary phase (set_db + scan at order {l2}) on "
            + ("the AVX-512 restatement (8 lanes per register as simd_zn.rs; each half's chain on 4 threads split "
               "as partial_gal's join / par_iter)" if orc.cpu_has_avx512() else "the scalar oracle")
            + f", {sec_s:.2f} s per query")


def run_reference(args, rank):
    """CPU restatement of the reference's answer path, timed on the host cores.
    Uses the oracle only (the product library is not loaded)."""
    if rank != 0:
        return 0
    from oracle import oracle as orc
    world = args.gpus
    l1, l2, shards = orc.get_database_shape(args.entries)
    steps, used = cpu_query_steps(l1, l2, shards, args.cpu_distinct, args.warmup, args.steps)
    per_step = [a + b for a, b in steps]
    total = sum(per_step)
    value = args.steps / total
    scan_s = statistics.mean(a for a, _ in steps)
    sec_s = statistics.mean(b for _, b in steps)
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * total / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": value * REF_RESPONSE_S_8T, "dtype": "u32",
        "data": "synthetic",
        "config": workload_config(args.entries, l1, l2, shards, world),
        "p50_ms": 1e3 * statistics.median(per_step), "p99_ms": 1e3 * float(np.percentile(per_step, 99)),
        "primary_ms": 1e3 * scan_s, "secondary_ms": 1e3 * sec_s,
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": used, "kind": "port",
                         "avx512": bool(orc.cpu_has_avx512()),
                         "sample": cpu_sample_text(l1, l2, shards, args.cpu_distinct, args.steps, used, scan_s, sec_s)},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "note": "C++ restatement of the reference's answer path (the reference is Rust and cannot be built here); "
                "the reference's published 2^22 response time is 4.3 s on 8 threads of a Xeon Gold 5318S "
                "(ARTIFACT-APPENDIX.md:122)",
    }
    print(json.dumps(line), flush=True)
    return 0


def cpu_baseline_line(args, l1, l2, shards):
    from oracle import oracle as orc
    steps, used = cpu_query_steps(l1, l2, shards, args.cpu_distinct, 1, 2)
    per_step = [a + b for a, b in steps]
    scan_s = statistics.mean(a for a, _ in steps)
    sec_s = statistics.mean(b for _, b in steps)
    return {"value": len(per_step) / sum(per_step), "unit": UNIT, "cores": used, "kind": "port",
            "avx512": bool(orc.cpu_has_avx512()),
            "sample": cpu_sample_text(l1, l2, shards, args.cpu_distinct, len(per_step), used, scan_s, sec_s)}


# the (primary, secondary) index pairs of the reference's bench (pir_wrapper.rs:562)
REFERENCE_INDICES = [(0, 0), (1, 0), (0, 1), (1, 1), (2, 2), (1, 2), (2, 0), (2, 1), (2, 2), (2742, 128), (923, 255),
                     (1389, 129), (200, 200), (4000, 255), (3000, 0), (3000, 1)]


def fixed_index_leg(dp, torch, fleet, l1, l2, shards, distinct, per_shard_entries, dev, rank):
    """The reference bench's 16 index pairs, one query per call through the
    host path, each reply decrypted and compared with the stored entry."""
    ok, times = 0, []
    for k, (i, j) in enumerate(REFERENCE_INDICES):
        q, sk = dp.prepare_query(hashlib.sha256(f"fixed-{rank}-{k}".encode()).digest(), i, j % shards, l1, l2)
        t0 = time.perf_counter()
        r = fleet.process_query(q)
        times.append(1e3 * (time.perf_counter() - t0))
        want = pack_host(shard_payload(torch, (j % shards) % distinct, per_shard_entries, dev)[i].cpu().numpy().tobytes())
        ok += int(np.array_equal(dp.process_reply(r, sk), want))
    return {"pairs": "pir_wrapper.rs:562, secondary index j mod S", "of": len(REFERENCE_INDICES), "decrypted_ok": ok,
            "p50_ms": statistics.median(times), "max_ms": max(times),
            "note": "host buffers, one query per call (copies and host staging included)"}


def batched_leg(dp, torch, dev, entries, engine, sizes, groups, check_every=8):
    """BASELINE configs 3 and 4: a database of `entries` entries with every
    shard resident, groups of B queries per pass on one engine; responses/s,
    per-query p50/p99, scan and secondary time per group, decryption of a
    sample of every group size."""
    l1, l2, shards = dp.get_database_shape(entries)
    per = 8 * l1
    slab_bytes = stored_shard_bytes(dp, l1)
    t0 = time.time()
    fleet = dp.Fleet(entries, shards)
    if engine == "tensor":
        fleet.set_engine(dp.ENGINE_TENSOR)
    for first in range(0, shards, 8):
        cnt = min(8, shards - first)
        co = torch.empty((cnt, per, dp.N), dtype=torch.uint16, device=dev)
        for i in range(cnt):
            dp.pack_payloads(shard_payload(torch, first + i, per, dev, seed0=3000), co[i], device=dev.index or 0)
        fleet.set_shards(first, co)
        del co
    torch.cuda.synchronize()
    prep_s = time.time() - t0
    stream = torch.cuda.current_stream()
    fleet.set_stream(stream.cuda_stream)
    rng = np.random.default_rng(20)
    pool_n = 2 * max(sizes)
    pidx = [(int(rng.integers(0, per)), int(rng.integers(0, shards))) for _ in range(pool_n)]
    pq, pseeds = [], []
    for k, (i, j) in enumerate(pidx):
        q, sk = dp.prepare_query(hashlib.sha256(f"c34-{engine}-{k}".encode()).digest(), i, j, l1, l2)
        pq.append(q)
        pseeds.append(sk)
    qlen = len(pq[0])
    pdev = torch.tensor(np.frombuffer(b"".join(pq), dtype=np.uint8).reshape(pool_n, qlen), device=dev)
    out = {"entries": entries, "shards": shards, "primary_order": l1, "secondary_order": l2,
           "resident": f"all {shards} shards ({shards * slab_bytes / 2**30:.0f} GiB)", "engine": engine,
           "preprocess_s": prep_s, "groups": {}}
    for B in sizes:
        if engine == "tensor":
            ch, tms, shapes = fleet.tune(B, pipeline=True)
            tile = {"rows_per_cta": shapes[ch][0], "mtiles_per_cta": shapes[ch][1], "stages": shapes[ch][2],
                    "persistent": bool(shapes[ch][3]), "kernel": TILE_KERNELS[shapes[ch][3]],
                    "schedule": fleet.get_schedule(B)}
        else:
            pb, _ = fleet.tune_cuda_cores(B)
            tile = {"queries_per_block": pb}
        fleet.set_batch(B)
        nq = B * groups
        sel = torch.arange(nq, device=dev) % pool_n
        qin = pdev[sel].contiguous()
        rout = torch.zeros((nq, dp.reply_bytes()), dtype=torch.uint8, device=dev)
        fleet.process_queries_device(qin[:2 * B], rout[:2 * B])  # warm-up: both buffer slots
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        fleet.process_queries_device(qin, rout)
        e1.record(stream)
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1)
        bt = fleet.batch_timings(nq)
        host = rout.cpu().numpy()
        check = list(range(0, nq, max(1, nq // check_every)))
        good = 0
        for k in check:
            i, j = pidx[k % pool_n]
            want = pack_host(shard_payload(torch, j, per, dev, seed0=3000)[i].cpu().numpy().tobytes())
            good += int(np.array_equal(dp.process_reply(host[k].tobytes(), pseeds[k % pool_n]), want))
        scan = statistics.mean(float(bt[3, g * B]) for g in range(groups))
        out["groups"][str(B)] = {
            "responses_per_sec": nq / (ms * 1e-3), "p50_ms": float(np.median(bt[0])),
            "p99_ms": float(np.percentile(bt[0], 99)), "scan_ms_per_group": scan,
            "secondary_ms_per_group": statistics.mean(float(bt[2, g * B]) for g in range(groups)),
            "scan_hbm_gbs": shards * slab_bytes / (scan * 1e-3) / 1e9,
            "scan_tensor_pops": (16 * 2 * B * shards * (slab_bytes // 4) / (scan * 1e-3) / 1e15
                                 if engine == "tensor" else None),
            "tile": tile, "checked": {"decrypted_ok": good, "of": len(check)}}
        del qin, rout
        if good != len(check):
            fleet.close()
            raise RuntimeError(f"{entries} entries, {engine}, B={B}: {len(check) - good} answers failed")
    fleet.set_batch(1)
    fleet.close()
    del pdev
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return out


def config1_leg(dp, torch, dev, rank):
    """BASELINE config 1, the reference's own CPU-runnable bench (`bench
    --db-entries 32768 --preprocessed-db-count 2`, pir_wrapper.rs:493-615):
    4 half shards on 2 distinct, the 16 index pairs of pir_wrapper.rs:562
    (secondary index j mod 4) answered one query per launch sequence (device
    events) and through host buffers, then as one group of 16.  Every reply
    decrypts; the replies and the shards' coefficients are kept for the CPU
    leg, which compares them with the oracle's bytes."""
    entries = 1 << 15
    l1, l2, shards = dp.get_database_shape(entries)
    per = 8 * l1
    fleet = dp.Fleet(entries, 2)
    fleet.set_engine(dp.ENGINE_TENSOR)
    co = torch.empty((2, per, dp.N), dtype=torch.uint16, device=dev)
    for i in range(2):
        dp.pack_payloads(shard_payload(torch, i, per, dev, seed0=5000), co[i], device=dev.index or 0)
    fleet.set_shards(0, co)
    pairs = [(i, j % shards) for i, j in REFERENCE_INDICES]
    qs = [dp.prepare_query(hashlib.sha256(f"c1-{rank}-{k}".encode()).digest(), i, j, l1, l2)
          for k, (i, j) in enumerate(pairs)]
    qlen = len(qs[0][0])
    qdev = torch.tensor(np.frombuffer(b"".join(q for q, _ in qs), dtype=np.uint8).reshape(len(qs), qlen), device=dev)
    rdev = torch.zeros((len(qs), dp.reply_bytes()), dtype=torch.uint8, device=dev)
    stream = torch.cuda.current_stream()
    fleet.set_stream(stream.cuda_stream)
    for _ in range(3):  # warm-up
        fleet.process_queries_device(qdev[:2], rdev[:2])
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    fleet.process_queries_device(qdev, rdev)  # one query per launch sequence, back to back
    e1.record(stream)
    torch.cuda.synchronize()
    plain_ms = e0.elapsed_time(e1)
    lat = fleet.batch_timings(len(qs))[0]
    fleet.set_batch(16)
    rb = torch.zeros_like(rdev)
    fleet.process_queries_device(qdev, rb)
    torch.cuda.synchronize()
    e0.record(stream)
    fleet.process_queries_device(qdev, rb)
    e1.record(stream)
    torch.cuda.synchronize()
    group_ms = e0.elapsed_time(e1)
    fleet.set_batch(1)
    fleet.set_stream(None)
    t0 = time.perf_counter()
    host = fleet.process_queries([q for q, _ in qs])
    e2e_s = time.perf_counter() - t0
    dev_replies = [r.tobytes() for r in rdev.cpu().numpy()]
    grp_replies = [r.tobytes() for r in rb.cpu().numpy()]
    coeffs = co.cpu().numpy()
    ok = sum(int(np.array_equal(dp.process_reply(r, sk), coeffs[j % 2][i]) and r == h and r == g)
             for (i, j), (q, sk), r, h, g in zip(pairs, qs, dev_replies, host, grp_replies))
    fleet.close()
    del co, qdev, rdev, rb
    out = {"entries": entries, "shards": shards, "distinct": 2, "primary_order": l1, "secondary_order": l2,
           "query_bytes": qlen, "indices": "pir_wrapper.rs:562, secondary index j mod 4",
           "responses_per_sec": len(qs) / (plain_ms * 1e-3), "p50_ms": float(np.median(lat)),
           "e2e_responses_per_sec": len(qs) / e2e_s, "group16_responses_per_sec": len(qs) / (group_ms * 1e-3),
           "checked": {"decrypted_ok": ok, "of": len(qs), "note": "device, host and group replies equal, and decrypt"}}
    return out, {"coeffs": coeffs, "queries": [q for q, _ in qs], "replies": dev_replies, "shards": shards}


def config1_cpu(check):
    """The oracle (C++ restatement of process_query) on config 1's shards and
    queries: its replies against the GPU's, byte for byte, and its time."""
    from oracle import oracle as orc
    threads = os.cpu_count() or 1
    orc.set_num_threads(threads)
    refs = []
    for i in range(2):
        d = orc.Database(11, check["coeffs"].shape[1] // 8)
        d.set_db(check["coeffs"][i])
        refs.append(d)
    fleet_refs = [refs[k % 2] for k in range(check["shards"])]
    t0 = time.perf_counter()
    want = [orc.process_query(fleet_refs, q) for q in check["queries"]]
    dt = time.perf_counter() - t0
    same = sum(int(a == b) for a, b in zip(want, check["replies"]))
    return {"value": len(want) / dt, "unit": UNIT, "cores": threads, "kind": "port",
            "sample": "the oracle's process_query (scalar C++ restatement) on the 16 queries of config 1",
            "gpu_replies_equal_oracle": {"equal": same, "of": len(want)}}


def extra_legs(args, dp, torch, dev, local_rank):
    """BASELINE configs 1 (2^15), 3, 4 (2^20, both engines) and 5 (served
    mix), run after the 2^22 fleet is released."""
    legs = {}
    try:
        legs["config1"], legs["_config1_check"] = config1_leg(dp, torch, dev, 0)
        if legs["config1"]["checked"]["decrypted_ok"] != legs["config1"]["checked"]["of"]:
            raise RuntimeError("config 1: a reply failed its check")
        legs["config3"] = batched_leg(dp, torch, dev, 1 << 20, "cuda", [16, 64, 256], 2)
        legs["config3"]["note"] = ("CUDA-core modular-MAC scan (u32 x u32 -> u64), one launch per group; the reference "
                                   "rule gives full shards at 2^20 (pir_wrapper.rs:188, 223-227)")
        legs["config4"] = batched_leg(dp, torch, dev, 1 << 20, "tensor", [16, 64, 256], 3)
        legs["config4"]["note"] = ("INT8 limb products on tcgen05 (u8 x u8 -> s32, 16 limb products per residue "
                                   "product, K = 4096, so no partial sum overflows), recombined and reduced mod each "
                                   "prime; scan_tensor_pops counts int8 limb operations (2 per MAC)")
        results, prep_s = serve_mix(args, local_rank, [5000.0], 3.0)
        legs["served"] = {"offered_per_sec": 5000.0, "seconds": 3.0, "preprocess_s": prep_s,
                          "mix": [float(x) for x in args.serve_mix.split(",")], **results[0],
                          "latency_note": "submit-to-reply wall time on the host, queueing included"}
    except RuntimeError as e:
        return {"error": str(e)}
    return legs


def main():
    args = parse()
    rank, local_rank, world = dist_env()
    if args.impl == "reference":
        return run_reference(args, rank)
    if args.serve:
        return run_serve(args, rank, local_rank)

    import torch
    import dnspir_b200 as dp

    torch.cuda.set_device(local_rank)
    ranks = RankGroup.init("nccl", world)
    barrier, max_over_ranks = ranks.barrier, ranks.max
    pg = ranks.pg

    dev = torch.device("cuda", local_rank)
    l1, l2, shards = dp.get_database_shape(args.entries)
    per_shard_entries = 8 * l1
    slab_bytes = stored_shard_bytes(dp, l1, local_rank)
    free, _ = torch.cuda.mem_get_info()
    sizes = [int(x) for x in args.batched.split(",") if x.strip()]
    # workspaces: two buffer slots, each with the scan output of the largest
    # group, the secondary phase's chunk (at most 8 GiB) and headroom
    per_query_ws = shards * 2 * dp.N * 8 * 4 + l2 * 3 * dp.N * 2
    reserve = args.reserve_gib * (1 << 30) if args.reserve_gib > 0 else \
        2 * max(sizes + [1]) * per_query_ws + (10 << 30)
    fit = int((free - int(reserve)) // slab_bytes)
    distinct = args.distinct if args.distinct > 0 else max(1, min(shards, fit))

    # ---- build and preprocess the fleet on the GPU
    t0 = time.time()
    fleet = dp.Fleet(args.entries, distinct, device=local_rank)
    if args.engine == "tensor":
        fleet.set_engine(dp.ENGINE_TENSOR)
    batch = 8
    for first in range(0, distinct, batch):
        cnt = min(batch, distinct - first)
        coeffs = torch.empty((cnt, per_shard_entries, dp.N), dtype=torch.uint16, device=dev)
        for i in range(cnt):
            dp.pack_payloads(shard_payload(torch, first + i, per_shard_entries, dev), coeffs[i], device=local_rank)
        fleet.set_shards(first, coeffs)
        del coeffs
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    prep_s = time.time() - t0

    # ---- queries (client side, host): uniform indices from seed 1
    rng = np.random.default_rng(1 + rank)
    total_q = args.warmup + args.steps
    idx = [(int(rng.integers(0, per_shard_entries)), int(rng.integers(0, shards))) for _ in range(total_q)]
    queries, seeds = [], []
    for k, (i, j) in enumerate(idx):
        rs = hashlib.sha256(f"query-{rank}-{k}".encode()).digest()
        q, sk = dp.prepare_query(rs, i, j, l1, l2)
        queries.append(q)
        seeds.append(sk)
    qlen = len(queries[0])
    qdev = torch.tensor(np.frombuffer(b"".join(queries), dtype=np.uint8).reshape(total_q, qlen), device=dev)
    rdev = torch.zeros((total_q, dp.reply_bytes()), dtype=torch.uint8, device=dev)
    stream = torch.cuda.current_stream()
    fleet.set_stream(stream.cuda_stream)

    # ---- unloaded latency: one query per call, nothing else in flight
    for w in range(args.warmup):
        fleet.process_queries_device(qdev[w:w + 1], rdev[w:w + 1])
    unloaded = []
    clocks = ClockSampler(local_rank)
    clocks.start()
    for w in range(args.warmup):
        fleet.process_queries_device(qdev[w:w + 1], rdev[w:w + 1])
        unloaded.append(fleet.batch_timings(1)[0, 0])
    torch.cuda.synchronize()

    # ---- device-resident path (value): K queries in HBM answered back to back
    # (the primary phase of query k+1 overlaps the secondary phase of query k)
    barrier()
    torch.cuda.synchronize()
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    w0 = args.warmup
    launches0 = fleet.launch_count()
    t_timed0 = time.time()
    ev0.record(stream)
    fleet.process_queries_device(qdev[w0:w0 + args.steps], rdev[w0:w0 + args.steps])
    ev1.record(stream)
    launches = fleet.launch_count() - launches0
    torch.cuda.synchronize()
    t_timed1 = time.time()
    barrier()
    torch.cuda.synchronize()
    clk = clocks.stop((t_timed0, t_timed1))
    total_ms = max_over_ranks(ev0.elapsed_time(ev1))
    tim = fleet.batch_timings(args.steps)
    step_ms = list(tim[0])
    phase = [(tim[1, k], tim[2, k], tim[3, k]) for k in range(tim.shape[1])]

    # ---- end to end through the C ABI with host buffers (H2D and D2H inside)
    fleet.set_stream(None)
    barrier()
    t_e2e = time.perf_counter()
    host_replies = fleet.process_queries(queries[w0:w0 + args.steps])
    e2e_s = max_over_ranks(time.perf_counter() - t_e2e)

    # ---- checks: every answer decrypts to its entry; host and device replies agree
    dev_replies = rdev[args.warmup:].cpu().numpy()
    ok = 0
    for k in range(args.steps):
        i, j = idx[args.warmup + k]
        d = j % distinct
        payload = shard_payload(torch, d, per_shard_entries, dev)[i].cpu().numpy().tobytes()
        want = pack_host(payload)
        got = dp.process_reply(host_replies[k], seeds[args.warmup + k])
        same = host_replies[k] == dev_replies[k].tobytes()
        ok += int(np.array_equal(got, want) and same)
    if ok != args.steps:
        print(json.dumps({"error": f"{args.steps - ok} of {args.steps} answers failed the decryption check"}),
              flush=True)
        return 1

    # ---- the reference bench's own index list (pir_wrapper.rs:562), secondary
    # index j mod S, answered one query at a time through the host path
    fixed = fixed_index_leg(dp, torch, fleet, l1, l2, shards, distinct, per_shard_entries, dev, rank)
    if fixed["decrypted_ok"] != fixed["of"]:
        print(json.dumps({"error": f"fixed index list: {fixed['of'] - fixed['decrypted_ok']} answers failed"}),
              flush=True)
        return 1

    # ---- batched: groups of B queries per pass over the slabs, same fleet
    batched = {}
    if args.engine == "cuda":
        sizes = [b for b in sizes if b <= 256 and b & (b - 1) == 0]
    if sizes:
        fleet.set_stream(stream.cuda_stream)
        pool_n = 2 * max(sizes)
        pidx = [(int(rng.integers(0, per_shard_entries)), int(rng.integers(0, shards))) for _ in range(pool_n)]
        pq, pseeds = [], []
        for k, (i, j) in enumerate(pidx):
            q, sk = dp.prepare_query(hashlib.sha256(f"client-{rank}-{k}".encode()).digest(), i, j, l1, l2)
            pq.append(q)
            pseeds.append(sk)
        pdev = torch.tensor(np.frombuffer(b"".join(pq), dtype=np.uint8).reshape(pool_n, qlen), device=dev)
        # --tile B:shape[:schedule]
        forced = {int(f[0]): [int(x) for x in f[1:]] for f in (x.split(":") for x in args.tile.split(",") if x.strip())}
        for B in sizes:
            shape = None
            if args.engine == "tensor" and B in forced:
                fleet.set_tile(B, forced[B][0])
                if len(forced[B]) > 1:
                    fleet.set_schedule(B, forced[B][1])
                sh = dp.tscan_shapes()[forced[B][0]]
                shape = {"rows_per_cta": sh[0], "mtiles_per_cta": sh[1], "stages": sh[2], "persistent": bool(sh[3]),
                         "kernel": TILE_KERNELS[sh[3]],
                         "schedule": {"order": ("overlap", "serial", "last chunk")[fleet.get_schedule(B) & 3],
                                      "cluster_chains": bool(fleet.get_schedule(B) & 4)},
                         "tuner": "forced (--tile)"}
            elif args.engine == "tensor":
                ch, tms, shapes = fleet.tune(B, pipeline=True)
                shape = {"rows_per_cta": shapes[ch][0], "mtiles_per_cta": shapes[ch][1], "stages": shapes[ch][2],
                         "persistent": bool(shapes[ch][3]), "kernel": TILE_KERNELS[shapes[ch][3]],
                         "schedule": {"order": ("overlap", "serial", "last chunk")[fleet.get_schedule(B) & 3],
                                      "cluster_chains": bool(fleet.get_schedule(B) & 4)},
                         "tuned_ms_per_group": round(float(tms[ch]), 3), "tuner": "whole-group pipeline"}
            else:
                pb, tms = fleet.tune_cuda_cores(B)
                shape = {"queries_per_block": pb, "tuned_scan_ms": round(float(tms[[1, 2, 4, 8, 16].index(pb)]), 3),
                         "tuner": "scan alone"}
            fleet.set_batch(B)
            nq = B * max(2, args.batched_groups)
            sel = torch.arange(nq, device=dev) % pool_n
            qin = pdev[sel].contiguous()
            rout = torch.zeros((nq, dp.reply_bytes()), dtype=torch.uint8, device=dev)
            fleet.process_queries_device(qin[:2 * B], rout[:2 * B])  # warm-up: both buffer slots
            barrier()
            torch.cuda.synchronize()
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            fleet.process_queries_device(qin, rout)
            e1.record(stream)
            torch.cuda.synchronize()
            bms = max_over_ranks(e0.elapsed_time(e1))
            bt = fleet.batch_timings(nq)
            good = 0
            host = rout.cpu().numpy()
            check = list(range(0, nq, max(1, nq // 8)))
            for k in check:
                i, j = pidx[k % pool_n]
                want = pack_host(shard_payload(torch, j % distinct, per_shard_entries, dev)[i].cpu().numpy().tobytes())
                good += int(np.array_equal(dp.process_reply(host[k].tobytes(), pseeds[k % pool_n]), want))
            if good != len(check):
                print(json.dumps({"error": f"batched B={B}: {len(check) - good} of {len(check)} answers failed"}),
                      flush=True)
                return 1
            gscan = [float(bt[3, g * B]) for g in range(args.batched_groups)]
            batched[str(B)] = {
                "scan_tensor_pops": (16 * 2 * B * shards * (slab_bytes // 4) / (statistics.mean(gscan) * 1e-3) / 1e15
                                     if args.engine == "tensor" else None),
                "responses_per_sec": whole_job_rate(nq, world, bms * 1e-3), "groups": args.batched_groups,
                "p50_ms": float(np.median(bt[0])), "p99_ms": float(np.percentile(bt[0], 99)),
                "scan_ms_per_group": statistics.mean(gscan),
                "effective_scan_gbs": B * (shards * slab_bytes) / (statistics.mean(gscan) * 1e-3) / 1e9,
                "secondary_ms_per_group": statistics.mean(float(bt[2, g * B]) for g in range(args.batched_groups)),
                "tile": shape, "checked": {"decrypted_ok": good, "of": len(check)}}
        fleet.set_batch(1)
        fleet.set_stream(None)
        del pdev, qin, rout

    # ---- report
    scan_ms = [p[2] for p in phase]
    scan_avg = statistics.mean(scan_ms)
    algo_bytes = shards * slab_bytes + 2 * 4 * dp.N * 4  # slabs + the per-factor query vectors
    achieved = algo_bytes / (scan_avg * 1e-3) / 1e9
    peak, peak_kind = measured_peak_hbm()
    kname = "tscan_kernel" if args.engine == "tensor" else "scan_batch_kernel"
    traffic = profiled_traffic("tscan_2p22.md" if args.engine == "tensor" else "scan_batch_2p22.md", algo_bytes)
    value = whole_job_rate(args.steps, world, total_ms * 1e-3)
    fleet.close()
    del qdev, rdev
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    int8_peak = None
    if args.engine == "tensor" and batched:
        int8_peak = int8_tensor_peak(torch, dev)
        for v in batched.values():
            v["scan_tensor_frac"] = (v["scan_tensor_pops"] / int8_peak["pops"]) if int8_peak["pops"] else None
    legs = {}
    if not args.quick and world == 1:
        legs = extra_legs(args, dp, torch, dev, local_rank)
        if "error" in legs:
            print(json.dumps({"error": legs["error"]}), flush=True)
            return 1
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": value * REF_RESPONSE_S_8T,
        "vs_baseline_ref": "reference response time 4.3 s at 2^22, 8 threads, Xeon Gold 5318S (ARTIFACT-APPENDIX.md:122)",
        "dtype": "u32", "data": "synthetic",
        "config": workload_config(args.entries, l1, l2, shards, world),
        "distinct_resident": distinct,
        "resident_note": f"{distinct} distinct full shards resident in HBM, logical shard k served by k mod {distinct} "
                         "(the reference's --preprocessed-db-count, pir_wrapper.rs:578); consecutive queries overlap "
                         "the secondary phase of one with the primary phase of the next",
        "p50_ms": statistics.median(step_ms), "p99_ms": float(np.percentile(step_ms, 99)),
        "latency_note": "p50/p99: per-query device latency (copy-in to reply) with queries back to back",
        "unloaded_p50_ms": statistics.median(unloaded) if unloaded else None,
        "primary_ms": statistics.mean(p[0] for p in phase), "secondary_ms": statistics.mean(p[1] for p in phase),
        "scan_ms": scan_avg, "scan_hbm_gbs": achieved, "preprocess_s": prep_s,
        "engine": args.engine,
        "batched": batched,
        "batched_vs_plain": {b: v["responses_per_sec"] / value for b, v in batched.items()},
        "int8_tensor_peak": int8_peak,
        "int8_tensor_peak_note": "scan_tensor_frac of each group size = scan_tensor_pops / the faster of two "
                                 "library 8-bit GEMMs (cuBLASLt int8 and fp8), sustained, measured in the same run",
        "roofline": {"kernel": kname, "bound": "hbm", "achieved": achieved, "peak": peak,
                     "peak_kind": peak_kind, "unit": "GB/s", "frac": achieved / peak,
                     "traffic": traffic, "algorithmic_bytes": algo_bytes},
        "e2e": {"value": whole_job_rate(args.steps, world, e2e_s), "unit": UNIT, "h2d_bytes_per_step": qlen,
                "d2h_bytes_per_step": dp.reply_bytes()},
        "gpu_launches": launches,
        "gpu_launches_note": "kernels the library launched in the timed region, counted at each launch "
                             "(dnspir_fleet_launch_count)",
        "fixed_indices": fixed,
        "clocks": clk,
        "checked": {"decrypted_ok": ok, "of": args.steps},
    }
    check1 = legs.pop("_config1_check", None)
    if int8_peak and int8_peak["pops"] and "config4" in legs:
        for v in legs["config4"]["groups"].values():
            v["scan_tensor_frac"] = v["scan_tensor_pops"] / int8_peak["pops"]
    line.update(legs)
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        line["cpu_baseline"] = cpu_baseline_line(args, l1, l2, shards)
        if check1 is not None:
            c1 = config1_cpu(check1)
            line["cpu_baseline"]["config1"] = c1
            if c1["gpu_replies_equal_oracle"]["equal"] != c1["gpu_replies_equal_oracle"]["of"]:
                print(json.dumps({"error": "config 1: GPU replies differ from the oracle's"}), flush=True)
                return 1
    if rank == 0:
        print(json.dumps(line), flush=True)
    if pg:
        pg.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
