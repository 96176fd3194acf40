"""Benchmark: Fibonacci STARK proofs/s on B200 (log_n = 24, blowup 4, 80 queries).

One step = one whole proof of the Fibonacci AIR at 2^24 rows (2^26-point
circle LDE): trace, LDE, trace / quotient / FRI commitments, transcript,
queries and decommitment, on the device.

  value    proofs/s with the proof state resident in HBM (device path:
           vx_prover_prove_async, four proofs in flight on four streams),
           all ranks.
  e2e      the same metric through the C ABI with host buffers
           (vx_prove_fib_batch: launch, run, copy the proof bytes to the host).
  p50/p99  per-proof latency through vx_prove_fib, one proof at a time, ms.
  roofline the dominant kernel, the trace commitment (Blake2s, integer ALU
           pipe), against a register-only Blake2s probe on the same GPU and
           against the ALU-pipe ceiling; lde_roofline: the LDE (interpolate
           + zero-pad + evaluate) against the measured HBM copy bandwidth.
  served   the metric's mixed log_n 16-24 stream: the serving engine and the
           plain one-at-a-time path, swept over arrival rates, compared by
           the rate each sustains at common p99 bounds.

The line holds the figures of every leg; ``--full`` prints their whole objects
(sweeps, work, sources) in their place.

N > 1 (torchrun): independent replicas, one per GPU, no collective on the
data path ("replicas only"); barrier + max-over-ranks timing.
``--impl reference`` times the CPU oracle (a C restatement of the reference's
path, OpenMP over all host cores) on the same workload.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "Fib STARK proofs/s + p50/p99 prove ms, mixed log_n 16-24; LDE HBM GB/s"
SEED = 0x5EED_2024
IN_FLIGHT = 4  # proofs in flight per GPU, as in vx_prove_fib_batch


def _peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index: int):
        self.dev = device_index
        self.proc = None
        self.path = None

    def start(self):
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.dev), f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if not self.proc:
            return None
        time.sleep(0.25)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        rows = []
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                rows.append(parts)
            except Exception:
                pass
        os.unlink(self.path)
        if not rows:
            return None
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if r[5 + i].lower().startswith("active")})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(rows)}


def cpu_baseline(log_n: int):
    """One proof of the same workload with the CPU oracle on all host cores."""
    from oracle import oracle as O
    from vortexstark_b200.workload import fib_inputs

    O.lib()
    cores = O.get_threads()
    a, b = fib_inputs(SEED ^ 0xC0FFEE, 1)[0]
    t0 = time.perf_counter()
    O.prove(a, b, 20)
    t20 = time.perf_counter() - t0
    est = t20 * (1 << (log_n - 20)) * (log_n + 2) / 22.0
    if est <= 40.0:
        t0 = time.perf_counter()
        O.prove(a, b, log_n)
        dt = time.perf_counter() - t0
        sample = f"one full log_n={log_n} proof (2^{log_n + 2}-point LDE, 80 queries)"
        return {"value": 1.0 / dt, "unit": "proofs/s", "cores": cores, "kind": "port", "sample": sample,
                "seconds": dt}
    k = log_n - 2
    t0 = time.perf_counter()
    O.prove(a, b, k)
    dt = time.perf_counter() - t0
    scale = (1 << (log_n - k)) * (log_n + 2) / (k + 2)
    return {"value": 1.0 / (dt * scale), "unit": "proofs/s", "cores": cores, "kind": "port",
            "sample": f"one log_n={k} proof ({dt:.2f} s) scaled by the N log N work ratio {scale:.2f} to log_n={log_n}",
            "seconds": dt}


PLAIN_RATE_MULTS = (0.5, 0.6, 0.7, 0.8, 0.85, 0.9, 0.95)
ENGINE_RATE_MULTS = (0.5, 0.6, 0.7, 0.8, 0.9, 1.0, 1.1, 1.2, 1.3, 1.4, 1.5)
SERVED_REPEATS = 2


def sustainable_rate(points, bound_ms):
    """Highest arrival rate whose p99 stays within bound_ms: walk the sweep
    (rate, p99) up from the lowest rate to the first point above the bound
    and interpolate linearly between it and the last point within it.  None
    if the lowest rate already exceeds the bound; the highest swept rate (a
    lower bound) if no point does."""
    best, prev = None, None
    for rate, p99 in sorted(points):
        if p99 <= bound_ms:
            best, prev = rate, (rate, p99)
            continue
        if prev is not None:
            r0, p0 = prev
            best = r0 + (bound_ms - p0) * (rate - r0) / (p99 - p0)
        break
    return best


def _pooled(runs, rate, sizes):
    """One sweep point from repeated runs at the same offered rate: latency
    percentiles over all their requests, throughput over their makespans."""
    from vortexstark_b200.serving import _summary

    lat, szs = [], []
    for r in runs:
        lat += r["lat_ms"]
        szs += sizes
    out = _summary(lat, sum(r["makespan_s"] for r in runs), sum(r["n"] for r in runs), szs)
    out.pop("lat_ms")
    out["rate"] = rate
    return out


def _plain_service(reqs):
    """Median one-at-a-time service time per size through the plain path
    (a cached slot and a pinned host buffer per size), and the caches."""
    import statistics as st

    from vortexstark_b200 import prover
    from vortexstark_b200.serving import plain_caches

    sizes = sorted({r[0] for r in reqs})
    caches = plain_caches(sizes)
    svc = {}
    for ln in sizes:
        prover.prove_cached_bytes(1, 2, caches[ln])
        t = []
        for i in range(5):
            t0 = time.perf_counter()
            prover.prove_cached_bytes(3 + i, 5, caches[ln])
            t.append(time.perf_counter() - t0)
        svc[ln] = st.median(t)
    return svc, caches


def plain_sweep(reqs, cap, seed, caches, mults=PLAIN_RATE_MULTS):
    from vortexstark_b200.serving import poisson_arrivals, run_sequential

    n, sizes, out = len(reqs), [r[0] for r in reqs], []
    for m in mults:
        runs = [run_sequential(reqs, poisson_arrivals(n, m * cap, seed + 1 + 7 * k), caches=caches)
                for k in range(SERVED_REPEATS)]
        out.append(_pooled(runs, m * cap, sizes))
    return out


def engine_sweep(reqs, cap, seed, policy=None, mults=ENGINE_RATE_MULTS, queue=None):
    """The serving engine over the same stream at each offered rate; returns
    the sweep and the engine's slot statistics.  `policy` and `queue` are
    keyword arguments of ProofServer.set_policy / set_queue_order."""
    from vortexstark_b200.serving import ProofServer, poisson_arrivals, run_stream

    n, sizes = len(reqs), [r[0] for r in reqs]
    with ProofServer(budget_bytes=64 << 30, max_inflight=24) as srv:
        if policy:
            srv.set_policy(**policy)
        if queue:
            srv.set_queue_order(**queue)
        counts = {16: 12, 18: 8, 20: 6, 22: 3, 24: 2}
        for ln in sorted(set(sizes)):
            srv.prewarm(ln, counts.get(ln, 2))
        run_stream(srv, reqs[:64], [0.0] * 64)  # warm-up
        sweep = []
        for m in mults:
            runs = [run_stream(srv, reqs, poisson_arrivals(n, m * cap, seed + 2 + 7 * k))[0]
                    for k in range(SERVED_REPEATS)]
            sweep.append(_pooled(runs, m * cap, sizes))
        stats = srv.stats()
    return sweep, stats


def equal_p99_rates(plain, engine, cap):
    """For the plain path's own p99 at 0.8x, 0.9x and 0.95x its capacity as bounds:
    the highest rate each path sustains within the bound, and their ratio."""
    plain_pts = [(r["rate"], r["p99_ms"]) for r in plain]
    eng_pts = [(r["rate"], r["p99_ms"]) for r in engine]
    out = {}
    for m in (0.8, 0.9, 0.95):
        bound = min(plain, key=lambda r: abs(r["rate"] - m * cap))["p99_ms"]
        pr, er = sustainable_rate(plain_pts, bound), sustainable_rate(eng_pts, bound)
        out[f"plain_p99_at_{m}x_capacity"] = {"p99_bound_ms": bound, "plain_rate_per_s": pr,
                                              "engine_rate_per_s": er, "ratio": (er / pr) if (er and pr) else None}
    return out


def served_benchmark(seed: int, n_requests: int = 512, policy=None):
    """Mixed-size served stream (log_n in {16,...,24}, weights {.4,.25,.2,.1,.05},
    Poisson arrivals): the continuous-batching engine against the plain
    one-proof-at-a-time path.

    Both paths are swept over arrival rates (multiples of the plain path's
    capacity; plain up to 0.95x), each point pooling SERVED_REPEATS runs of
    n_requests with different arrival seeds.  For common p99 bounds (the plain
    path's own p99 at 0.8x and at 0.9x its capacity) the highest rate each
    path sustains within the bound is interpolated from its sweep, and the
    ratio of those rates is the speed-up at equal p99 (also at the plain
    path's p99 at 0.95x its capacity)."""
    import statistics as st

    from vortexstark_b200.workload import served_stream

    reqs = served_stream(seed, n_requests)
    svc, caches = _plain_service(reqs)
    cap = 1.0 / st.fmean(svc[r[0]] for r in reqs)
    plain = plain_sweep(reqs, cap, seed, caches)
    for c in caches.values():
        c.close()
    sweep, stats = engine_sweep(reqs, cap, seed, policy)
    at_bound = equal_p99_rates(plain, sweep, cap)
    return {
        "requests": n_requests, "repeats_per_rate": SERVED_REPEATS,
        "log_n_weights": {"16": 0.4, "18": 0.25, "20": 0.2, "22": 0.1, "24": 0.05},
        "plain_service_ms": {str(k): 1e3 * v for k, v in svc.items()},
        "plain_capacity_per_s": cap,
        "plain_sweep": plain,
        "served_sweep": sweep,
        "sustainable_rate_at_equal_p99": at_bound,
        "speedup_at_equal_p99": {k: v["ratio"] for k, v in at_bound.items()},
        "method": "highest arrival rate with pooled p99 <= bound, interpolated between sweep points; "
                  "ratio = engine rate / plain rate at the same bound",
        "engine": {"max_inflight": 24, "policy": policy or "default", "slots": stats["slots"],
                   "device_bytes": stats["bytes_used"]},
    }


# DRAM bytes of one LDE (iNTT 2^24 + evaluate 2^26) at log_n = 24 from an ncu
# capture of the current kernels (dram__bytes_read.sum + dram__bytes_write.sum
# of the LDE's pass launches); None until measured.
LDE_TRAFFIC_LOG24 = 1141.07e6 + 671.70e6
LDE_TRAFFIC_SOURCE = ("ncu dram__bytes_read.sum + dram__bytes_write.sum of the LDE's six pass launches (plans "
                      "11 + 7 + 6 each way), one proof slot at log_n = 24, one-pass metrics: "
                      "profiles/ntt_vec_lde_log24.md. The bottom evaluate pass reads its twiddles, as large as "
                      "the data")

# DRAM bytes of the trace commitment at log_n = 24 (2^26 leaves: leaf subtrees,
# nodes, reduce) from an ncu capture of one proof slot.
TRACE_COMMIT_TRAFFIC_LOG24 = (269.68e6 + 176.98e6) + (142.14e6 + 18.34e6) + (8.41e6 + 0.0) + (2.17e6 + 0.0)
TRACE_COMMIT_TRAFFIC_SOURCE = ("ncu dram__bytes_read.sum + dram__bytes_write.sum of the trace commitment's four launches "
                               "(leaf_subtree_kernel<LeafM31>, node_subtree_kernel twice, tree_reduce_kernel<LeafM31>), one "
                               "proof slot at log_n = 24, one-pass metrics: profiles/merkle_trace_commit_log24.md. "
                               "Reads: the 2^26 leaf words once, then the stored level of 2^22 hashes")

LIFT_LOGS = [16] * 8 + [18] * 16 + [20] * 10  # 34 columns, blowup 4: LDEs of 2^18 / 2^20 / 2^22


def lifted_workload(seed: int, logs=None):
    from vortexstark_b200.workload import m31_array

    logs = LIFT_LOGS if logs is None else logs
    return [m31_array(seed + 7919 * c, 1 << L) for c, L in enumerate(logs)]


def batched_commit_benchmark(seed: int, steps: int, warmup: int, peak_gbs: float, probe_rate: float,
                             cpu: bool = True, contexts: int = 4):
    """Batched lifted commitment of uneven-size columns (34 M31 columns,
    8 x 2^16, 16 x 2^18, 10 x 2^20, blowup 4, one lifted tree with S = 22,
    a random QM31 combination folded by FRI, 80 queries), replayed as one
    CUDA graph.  Device-resident throughput (`contexts` commitments in flight,
    and one at a time), end-to-end throughput with the columns
    uploaded from pinned host memory and the words read back every step,
    per-stage times and the two rooflines."""
    import torch

    from vortexstark_b200.lifted import LiftedCommitter

    cols = lifted_workload(seed)
    pinned = [torch.from_numpy(c.view("int32")).pin_memory() for c in cols]
    ptrs = [t.data_ptr() for t in pinned]
    com = LiftedCommitter(LIFT_LOGS, 2, 80)
    st = torch.cuda.Stream()
    s = st.cuda_stream
    for _ in range(warmup):
        com.upload_async(ptrs, s)
        com.commit_async(s, graph=True)
    st.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.nvtx.range_push("timed_commits")  # lets a profiler select exactly these launches
    e0.record(st)
    for _ in range(steps):
        com.commit_async(s, graph=True)
    e1.record(st)
    st.synchronize()
    torch.cuda.nvtx.range_pop()
    dev_ms = e0.elapsed_time(e1) / steps
    # end to end: H2D of every column, the commitment, D2H of the words
    h2d = sum(4 * len(c) for c in cols)
    lat = []
    for _ in range(steps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(st)
        com.upload_async(ptrs, s)
        com.commit_async(s, graph=True)
        com.fetch_async(s)
        b.record(st)
        b.synchronize()
        lat.append(a.elapsed_time(b))
    com.result_bytes()
    e2e_ms = statistics.median(lat)
    # several commitments in flight: more contexts, each on its own stream,
    # taken in turn.  End to end, one commitment's column upload (copy
    # engine) overlaps the others' device work; every commitment still
    # uploads all its columns and reads its words back inside the timed region
    extra = [LiftedCommitter(LIFT_LOGS, 2, 80) for _ in range(contexts - 1)]
    ctx = [(com, st)] + [(c, torch.cuda.Stream()) for c in extra]

    def in_flight(upload: bool) -> float:
        for c, t in ctx:
            c.upload_async(ptrs, t.cuda_stream)
            c.commit_async(t.cuda_stream, graph=True)
            c.fetch_async(t.cuda_stream)
        torch.cuda.synchronize()
        q0, q1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        q0.record(st)
        for _, t in ctx[1:]:
            t.wait_event(q0)
        for i in range(contexts * steps):
            c, t = ctx[i % contexts]
            if upload:
                c.upload_async(ptrs, t.cuda_stream)
            c.commit_async(t.cuda_stream, graph=True)
            if upload:
                c.fetch_async(t.cuda_stream)
        for _, t in ctx[1:]:
            j = torch.cuda.Event()
            j.record(t)
            st.wait_event(j)
        q1.record(st)
        q1.synchronize()
        return q0.elapsed_time(q1) / (contexts * steps)

    pipe_ms = in_flight(True)
    pipe_equal = all(c.result_bytes() == com.result_bytes() for c, _ in ctx[1:])
    # device-resident (no uploads): one's latency-bound FRI tail overlaps the
    # others' hashing
    dev2_ms = in_flight(False)
    for c in extra:
        c.close()
    # per-stage device times
    names = ["lde", "lifted_tree", "combination_tree", "circle_fold", "line_folds", "queries", "openings"]
    reps = 3
    ev = [[torch.cuda.Event(enable_timing=True) for _ in range(len(names) + 1)] for _ in range(reps)]
    for r in range(reps):
        for k in range(len(names)):
            ev[r][k].record(st)
            com.stage_async(k, s)
        ev[r][-1].record(st)
    st.synchronize()
    stages = {n: statistics.median([ev[r][k].elapsed_time(ev[r][k + 1]) for r in range(reps)])
              for k, n in enumerate(names)}
    # LDE bytes: per column 8n (iNTT) + 4n (coefficients read) + 4N (LDE written)
    lde_bytes = sum(12 * (1 << L) + 4 * (1 << (L + 2)) for L in LIFT_LOGS)
    lde_gbs = lde_bytes / (stages["lde"] / 1e3) / 1e9
    S = max(LIFT_LOGS) + 2
    n_leaves = 1 << S
    tree_comp = n_leaves * 3 + (n_leaves - 1)  # 34-word leaves: 3 compressions each
    tree_rate = tree_comp / (stages["lifted_tree"] / 1e3)
    out = {
        "workload": "lifted commitment: 34 M31 columns (8 x 2^16, 16 x 2^18, 10 x 2^20), blowup 4, "
                    "one lifted Blake2s tree (2^22 leaves of 34 words), QM31 combination + FRI to 8 values, "
                    "80 queries; one CUDA graph per commitment",
        "value": 1e3 / dev2_ms, "unit": "commitments/s", "ms_per_commit": dev2_ms,
        "in_flight": f"{contexts} commitments: {contexts} contexts on {contexts} streams taken in turn, graph "
                     "replays, CUDA events around the loop",
        "value_one_in_flight": 1e3 / dev_ms, "ms_per_commit_one_in_flight": dev_ms,
        "e2e": {"value": 1e3 / pipe_ms, "unit": "commitments/s", "ms_per_commit": pipe_ms,
                "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": com.size,
                "how": f"{contexts} contexts on {contexts} streams, CUDA events around the loop: each commitment "
                       "uploads its 34 columns from pinned memory, commits and reads its words back",
                "latency_ms": e2e_ms, "latency_how": "one commitment alone: upload, commit, read back (CUDA events)",
                "contexts_bytes_equal": pipe_equal},
        "launches_per_commit": com.launches(), "device_bytes": com.device_bytes(),
        "stages_ms": stages,
        "roofline": {"bound": "hbm", "kernel": "stwo LDE of all 34 columns", "achieved": lde_gbs,
                     "peak": peak_gbs, "unit": "GB/s", "frac": lde_gbs / peak_gbs, "algorithmic_bytes": lde_bytes},
        "roofline_alu": {"bound": "int-alu (Blake2s)", "kernel": "lifted tree (2^22 leaves, 3 compressions each)",
                         "achieved": tree_rate, "peak": probe_rate, "unit": "compressions/s",
                         "frac": tree_rate / probe_rate},
    }
    com.close()
    if cpu:
        from oracle import oracle as O

        O.lib()
        t0 = time.perf_counter()
        O.commit_lifted(cols, 2, 80)
        dt = time.perf_counter() - t0
        out["cpu_baseline"] = {"value": 1.0 / dt, "unit": "commitments/s", "cores": O.get_threads(), "kind": "port",
                               "sample": "one full commitment of the same 34 columns"}
    return out


def _ntt_words_equal_reference(O, cache, k: int) -> dict:
    """Evaluate, then interpolate, the same 2^k input with this library's
    launchers and with the reference's own (circle_ntt.cu:248-312) on the
    same tables; every output word compared on the device."""
    import torch

    from vortexstark_b200 import _lib, ntt
    from vortexstark_b200.ntt import _host_u32
    from vortexstark_b200.workload import m31_array

    n = 1 << k
    R = O.ref_lib()
    for name in ("cuda_circle_ntt_evaluate", "cuda_circle_ntt_interpolate"):
        getattr(R, name).argtypes = _lib._SIGS[name]
    x = torch.from_numpy(m31_array(SEED + 3 * k, n).view("int32")).cuda()
    mine, theirs = x.clone(), x.clone()
    offs, sizes = _host_u32(cache.layer_offsets), _host_u32(cache.layer_sizes)
    ntt.evaluate(mine, cache)
    R.cuda_circle_ntt_evaluate(theirs.data_ptr(), cache.d_twiddles.data_ptr(), cache.d_circle_twids.data_ptr(),
                               offs, sizes, k - 1, n)
    torch.cuda.synchronize()
    ev_eq = bool(torch.equal(mine, theirs))
    ntt.interpolate(mine, cache)
    R.cuda_circle_ntt_interpolate(theirs.data_ptr(), cache.d_itwiddles.data_ptr(), cache.d_circle_itwids.data_ptr(),
                                  offs, sizes, k - 1, n)
    torch.cuda.synchronize()
    out = {"evaluate": ev_eq, "interpolate": bool(torch.equal(mine, theirs)),
           "round_trip": bool(torch.equal(mine, x)), "words": n}
    del x, mine, theirs
    return out


def lde_only(log_n: int, steps: int, warmup: int) -> dict:
    """The LDE of one Fibonacci proof slot: trace, then interpolate and
    evaluate (the timed part) per step, inside an NVTX range 'lde' after
    the warm-up steps.  One slot keeps the device footprint small."""
    import torch

    from vortexstark_b200 import _lib, prover

    L = _lib.lib()
    cache = prover.ProverCache(log_n)
    ms = []
    for r in range(warmup + steps):
        if r == warmup:
            torch.cuda.nvtx.range_push("lde")
        _lib.check(L.vx_prover_stage_async(cache._p, 0, 3, 5, None))
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        _lib.check(L.vx_prover_stage_async(cache._p, 1, 3, 5, None))
        _lib.check(L.vx_prover_stage_async(cache._p, 2, 3, 5, None))
        e1.record()
        e1.synchronize()
        if r >= warmup:
            ms.append(e0.elapsed_time(e1))
    torch.cuda.nvtx.range_pop()
    torch.cuda.synchronize()
    cache.close()
    n, N = 1 << log_n, 1 << (log_n + 2)
    t = statistics.median(ms)
    peak, _ = _peaks()
    return {"log_n": log_n, "steps": steps, "ms": t, "gbs": (8 * n + 4 * n + 4 * N) / (t / 1e3) / 1e9,
            "frac": (8 * n + 4 * n + 4 * N) / (t / 1e3) / 1e9 / peak}


def trace_commit_only(log_n: int, steps: int, warmup: int) -> dict:
    """The trace commitment of one Fibonacci proof slot (the Blake2s tree of
    the 2^(log_n+2)-point LDE: leaf-subtree, node and reduce kernels), --steps
    times inside an NVTX range 'trace_commit' after the warm-up steps; the
    trace and its LDE are computed once before.  One slot keeps the device
    footprint small (2.3 GB at log_n = 24)."""
    import torch

    from vortexstark_b200 import _lib, prover

    L = _lib.lib()
    cache = prover.ProverCache(log_n)
    for k in range(3):
        _lib.check(L.vx_prover_stage_async(cache._p, k, 3, 5, None))
    ms = []
    for r in range(warmup + steps):
        if r == warmup:
            torch.cuda.nvtx.range_push("trace_commit")
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        _lib.check(L.vx_prover_stage_async(cache._p, 3, 3, 5, None))
        e1.record()
        e1.synchronize()
        if r >= warmup:
            ms.append(e0.elapsed_time(e1))
    torch.cuda.nvtx.range_pop()
    torch.cuda.synchronize()
    cache.close()
    N = 1 << (log_n + 2)
    t = statistics.median(ms)
    return {"log_n": log_n, "steps": steps, "ms": t, "compressions": 2 * N - 1,
            "g_compressions_per_s": (2 * N - 1) / (t / 1e3) / 1e9, "leaf_bytes": 4 * N}


def ntt_microbench(peak_gbs: float, sizes=(20, 24, 28), reps: int = 5):
    """Standalone circle NTT / iNTT on 2^k uniform M31 values over
    half_coset(k), through the reference-compatible launchers
    (cuda_circle_ntt_evaluate / _interpolate, which synchronise like the
    reference's), timed with CUDA events on the legacy stream around `reps`
    calls; the reference's own kernels compiled for sm_100a are timed the same
    way when they are built.  Algorithmic bytes: 8 per element (one read, one
    write)."""
    import ctypes as C

    import torch

    from vortexstark_b200 import _lib, ntt
    from vortexstark_b200.circle import Coset
    from vortexstark_b200.workload import m31_array

    out = {}
    ds = torch.cuda.default_stream()
    for k in sizes:
        n = 1 << k
        cache = ntt.TwiddleCache(Coset.half_coset(k))
        d = torch.from_numpy(m31_array(SEED + k, n).view("int32")).cuda()
        ntt.evaluate(d, cache)
        ntt.interpolate(d, cache)
        res = {}
        for name, fn in (("evaluate", ntt.evaluate), ("interpolate", ntt.interpolate)):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(ds)
            for _ in range(reps):
                fn(d, cache)
            e1.record(ds)
            e1.synchronize()
            ms = e0.elapsed_time(e1) / reps
            res[name] = {"ms": ms, "gbs": 8 * n / (ms / 1e3) / 1e9, "frac": 8 * n / (ms / 1e3) / 1e9 / peak_gbs}
        try:
            from oracle import oracle as O

            if O.ref_available():
                re_, ri = O.ref_ntt_time(k, reps)
                res["reference_kernels_ms"] = {"evaluate": re_, "interpolate": ri}
                res["words_equal_reference_kernels"] = _ntt_words_equal_reference(O, cache, k)
        except Exception as exc:  # the reference kernels are optional here
            res["reference_kernels_ms"] = f"unavailable: {exc}"
        out[f"2^{k}"] = res
        del d, cache
        torch.cuda.empty_cache()
    # batched (ntt.rs:191-281 as the reference's default `forge-ntt-batch` build calls it: the _forge
    # symbols with a host array of column pointers): the batched commitment's largest size group,
    # 10 columns of 2^22
    k, ncol = 22, 10
    n = 1 << k
    cache = ntt.TwiddleCache(Coset.half_coset(k))
    cols = [torch.from_numpy(m31_array(SEED + 50 + c, n).view("int32")).cuda() for c in range(ncol)]
    ptrs = (C.c_void_p * ncol)(*[c.data_ptr() for c in cols])
    host_u32 = lambda v: (C.c_uint32 * max(len(v), 1))(*v)
    libs = {"vortex": _lib.lib()}
    try:
        from oracle import oracle as O

        if O.ref_available():
            R = O.ref_lib()
            for name in ("cuda_circle_ntt_evaluate_batch_forge", "cuda_circle_ntt_interpolate_batch_forge"):
                getattr(R, name).argtypes = _lib._SIGS[name]
            libs["reference_kernels"] = R
    except Exception:
        pass
    res, outs = {}, {}
    for name, Lx in libs.items():
        def ev(Lx=Lx):
            Lx.cuda_circle_ntt_evaluate_batch_forge(ptrs, cache.d_twiddles.data_ptr(),
                                              cache.d_circle_twids.data_ptr(), host_u32(cache.layer_offsets),
                                              host_u32(cache.layer_sizes), k - 1, n, ncol)

        def it(Lx=Lx):
            Lx.cuda_circle_ntt_interpolate_batch_forge(ptrs, cache.d_itwiddles.data_ptr(),
                                                 cache.d_circle_itwids.data_ptr(), host_u32(cache.layer_offsets),
                                                 host_u32(cache.layer_sizes), k - 1, n, ncol)
        ev()
        outs[name] = hash(b"".join(bytes(c.cpu().numpy().tobytes()) for c in cols))
        it()
        for op, fn in (("evaluate", ev), ("interpolate", it)):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(ds)
            for _ in range(reps):
                fn()
            e1.record(ds)
            e1.synchronize()
            ms = e0.elapsed_time(e1) / reps
            res[f"{op}_{name}"] = {"ms": ms, "gbs": 8 * n * ncol / (ms / 1e3) / 1e9,
                                   "frac": 8 * n * ncol / (ms / 1e3) / 1e9 / peak_gbs}
    res["values_equal"] = len(set(outs.values())) == 1
    out[f"batch_{ncol}x2^{k}"] = res
    del cols, ptrs, cache
    torch.cuda.empty_cache()
    return out


def stage_roofline_table(stages_ms: dict, log_n: int, peak_gbs: float, probe_rate: float) -> dict:
    """Each proof stage against its bound, with the fixed algorithmic work:
    HBM stages in bytes (NTT of m = 8m, zero-pad + evaluate = 4n + 4N, trace
    written = 4n), hashing stages in Blake2s compressions (a tree of M leaves
    of at most 16 words = 2M - 1) against the register-only probe; the folds
    and the quotient fused into the hashing stages are listed as their bytes
    beside the compressions."""
    n, N = 1 << log_n, 1 << (log_n + 2)
    layers = [N >> k for k in range(1, log_n + 2 - 3 + 1)]  # FRI layer sizes N/2 .. 8
    line_bytes = sum(24 * m for m in layers[:-1])           # line fold M -> M/2 for M = N/2 .. 16
    work = {
        "trace": ("hbm", 4 * n, "bytes"),
        "interpolate": ("hbm", 8 * n, "bytes"),
        "lde_evaluate": ("hbm", 4 * n + 4 * N, "bytes"),
        "trace_commit": ("int-alu", 2 * N - 1, "compressions"),
        "quotient_commit": ("int-alu", 2 * N - 1, "compressions", 20 * N),
        "circle_fold_commit": ("int-alu", 2 * (N // 2) - 1, "compressions", 24 * N),
        "line_folds_commit": ("int-alu", sum(2 * m - 1 for m in layers[1:]), "compressions", line_bytes),
    }
    out = {}
    for name, w in work.items():
        ms = stages_ms.get(name)
        if not ms:
            continue
        rate = w[1] / (ms / 1e3)
        row = {"bound": w[0], "work": w[1], "unit": w[2], "ms": ms}
        if w[0] == "hbm":
            row.update(achieved_gbs=rate / 1e9, frac=rate / 1e9 / peak_gbs)
        else:
            row.update(achieved_per_s=rate, frac=rate / probe_rate, int_ops_per_s=1120 * rate)
            if len(w) > 3:
                row["fused_bytes"] = w[3]
        out[name] = row
    return out


def _time_ms(fn, stream, reps):
    import torch

    fn()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(reps):
        fn()
    e1.record(stream)
    e1.synchronize()
    return e0.elapsed_time(e1) / reps


def kernel_microbench(peak_gbs: float, probe_rate: float, log_n: int = 26, reps: int = 5, cpu: bool = True):
    """The standalone kernels of the log_n=24 proof's configuration at 2^26:
    a Blake2s Merkle commitment over 2^26 M31 leaves, a FRI fold of a
    2^26-point QM31 codeword down to 2 values (circle fold, then line folds;
    once as bare folds, once with every layer committed and its challenge
    drawn from the transcript, beside the CPU oracle),
    the QM31 / M31 bit-reversals and the half-coset-to-canonic permutation.  Each runs through this library's
    reference-compatible launchers (the reference's own call sequence:
    merkle.rs commit_root_only = tiled 1024-leaf roots + hash_nodes +
    reduce_to_root; fri.rs fold_*_with_twiddles) and, when they are built,
    through the reference's own kernels (same symbols, same calls); the
    Merkle commitment also through this library's fused tree
    (vx_merkle_root_cols).  CUDA events on the legacy stream around `reps`
    calls.  HBM figures use algorithmic bytes (each array read and written
    once); the Merkle figures count compressions (2^26 leaves + 2^26 - 1
    nodes)."""
    import ctypes as C

    import numpy as np
    import torch

    from vortexstark_b200 import _lib, fri
    from vortexstark_b200.field import qm31_mul
    from vortexstark_b200.merkle import FusedRoot
    from vortexstark_b200.workload import m31_array

    ds = torch.cuda.default_stream()
    n = 1 << log_n
    libs = {"vortex": _lib.lib()}
    try:
        from oracle import oracle as O

        if O.ref_available():
            R = O.ref_lib()
            for name in ("cuda_merkle_tiled_generic", "cuda_merkle_hash_nodes", "cuda_merkle_reduce_to_root",
                         "cuda_fold_line_soa", "cuda_fold_circle_into_line_soa", "cuda_bit_reverse_qm31",
                         "cuda_bit_reverse_m31", "cuda_permute_hc_to_canonic_brt", "cuda_eval_at_point",
                         "cuda_barycentric_eval", "cuda_compute_coset_points", "cuda_extract_and_squash",
                         "cuda_batch_inverse_m31", "cuda_fibonacci_quotient", "cuda_stwo_ntt_evaluate",
                         "cuda_stwo_ntt_interpolate", "cuda_stwo_ntt_batch_evaluate",
                         "cuda_stwo_ntt_batch_interpolate"):
                getattr(R, name).argtypes = _lib._SIGS[name]
            libs["reference_kernels"] = R
    except Exception:
        pass
    out = {"log_n": log_n, "reps": reps}

    # ---- Merkle commitment over 2^26 M31 leaves ----
    col = torch.from_numpy(m31_array(SEED + 1, n).view("int32")).cuda()
    ptrs = torch.tensor([col.data_ptr()], dtype=torch.int64, device="cuda")
    tiles = n // 1024
    sub_roots = torch.empty(tiles * 8, dtype=torch.int32, device="cuda")
    scratch = [torch.empty(max(tiles >> (j + 1), 1) * 8, dtype=torch.int32, device="cuda") for j in range(20)]
    root = torch.empty(8, dtype=torch.int32, device="cuda")
    comps = 2 * n - 1
    merkle = {}
    roots = {}
    for name, Lx in libs.items():
        def commit(Lx=Lx):
            Lx.cuda_merkle_tiled_generic(ptrs.data_ptr(), sub_roots.data_ptr(), 1, n)
            cur, size, j = sub_roots, tiles, 0
            while size > 1024:
                size //= 2
                Lx.cuda_merkle_hash_nodes(cur.data_ptr(), scratch[j].data_ptr(), size)
                cur, j = scratch[j], j + 1
            Lx.cuda_merkle_reduce_to_root(cur.data_ptr(), root.data_ptr(), size)
        ms = _time_ms(commit, ds, reps)
        roots[name] = bytes(root.cpu().numpy().tobytes())
        merkle[name] = {"ms": ms, "compressions_per_s": comps / (ms / 1e3),
                        "frac_of_probe": comps / (ms / 1e3) / probe_rate}
    fr = FusedRoot(log_n)
    ms = _time_ms(lambda: fr.commit_async([col]), ds, reps)
    roots["fused"] = bytes(fr.root_dev.cpu().numpy().tobytes())
    merkle["vortex_fused_tree"] = {"ms": ms, "compressions_per_s": comps / (ms / 1e3),
                                   "frac_of_probe": comps / (ms / 1e3) / probe_rate}
    merkle["roots_equal"] = len(set(roots.values())) == 1
    out["merkle_commit_m31"] = merkle
    del col, ptrs, sub_roots, scratch, fr
    torch.cuda.empty_cache()

    # ---- FRI fold chain 2^26 -> 2 ----
    rng = np.random.default_rng(SEED + 2)
    src = [torch.from_numpy(rng.integers(0, 0x7FFFFFFF, n, dtype=np.uint32).view(np.int32)).cuda() for _ in range(4)]
    dst = [torch.empty(n // 2, dtype=torch.int32, device="cuda") for _ in range(4)]
    ping = [[torch.empty(n // 4, dtype=torch.int32, device="cuda") for _ in range(4)] for _ in range(2)]
    tws = fri.precompute_fri_twiddles(log_n, 1)  # circle fold at 2^26, line folds 2^25 .. 2^2
    a4 = [int(x) for x in rng.integers(0, 0x7FFFFFFF, 4)]
    alpha = (C.c_uint32 * 4)(*a4)
    alpha_sq = (C.c_uint32 * 4)(*[int(x) for x in qm31_mul(a4, a4)])
    # algorithmic bytes (fixed formulas: circle fold N -> N/2 = 24N, line fold M -> M/2 = 24M; twiddles and
    # the circle fold's accumulator read excluded), and the bytes the launchers actually move
    fold_bytes, moved = 24 * n, 16 * n + 2 * 16 * (n // 2) + 4 * (n // 2)
    m = n // 2
    while m > 2:
        fold_bytes += 24 * m
        moved += 16 * m + 4 * (m // 2) + 16 * (m // 2)
        m //= 2
    fold = {"bytes": fold_bytes, "bytes_moved_incl_twiddles_and_accumulator": moved}
    finals = {}
    for name, Lx in libs.items():
        def chain(Lx=Lx):
            Lx.cuda_fold_circle_into_line_soa(*[d.data_ptr() for d in dst], *[s.data_ptr() for s in src],
                                              tws[0].data_ptr(), alpha, alpha_sq, n // 2)
            cur, m, j = dst, n // 2, 0
            while m > 2:
                nxt = ping[j & 1]
                Lx.cuda_fold_line_soa(*[c.data_ptr() for c in cur], tws[j + 1].data_ptr(),
                                      *[c.data_ptr() for c in nxt], alpha, m // 2)
                cur, m, j = nxt, m // 2, j + 1
            return cur
        for d in dst:
            d.zero_()
        last = chain()  # the circle fold accumulates into dst: time from a fixed start
        finals[name] = b"".join(bytes(c[:2].cpu().numpy().tobytes()) for c in last)
        def timed(Lx=Lx):
            chain(Lx)
        ms = _time_ms(timed, ds, reps)
        fold[name] = {"ms": ms, "gbs": fold_bytes / (ms / 1e3) / 1e9, "frac": fold_bytes / (ms / 1e3) / 1e9 / peak_gbs}
    fold["final_values_equal"] = len(set(finals.values())) == 1
    out["fri_fold_qm31_to_2"] = fold
    del dst, ping, tws
    torch.cuda.empty_cache()

    # ---- FRI chain with a commitment per layer, transcript-drawn challenges (vx_fri_chain) ----
    from vortexstark_b200.fri import FriChain

    state = [int(x) for x in rng.integers(0, 1 << 32, 8, dtype=np.uint64)]
    chain = FriChain(log_n)
    ms = _time_ms(lambda: chain.commit_async(src, state), ds, reps)
    roots, _, last = chain.result()
    comps = sum((1 << l) + (1 << l) - 1 for l in range(1, log_n))  # layer of 2^l values: leaves + nodes
    fc = {"ms": ms, "layers": chain.layers, "launches": chain.launches(), "compressions": comps,
          "compressions_per_s": comps / (ms / 1e3), "frac_of_probe": comps / (ms / 1e3) / probe_rate,
          "fold_bytes": fold_bytes, "fold_gbs": fold_bytes / (ms / 1e3) / 1e9}
    if cpu:
        from oracle import oracle as O

        host = np.stack([s.cpu().numpy().view(np.uint32) for s in src])
        t0 = time.perf_counter()
        oroots, _, olast = O.fri_chain(host, state)
        fc["cpu_baseline"] = {"ms": 1e3 * (time.perf_counter() - t0), "cores": O.get_threads(), "kind": "port",
                              "equal": bool(np.array_equal(np.array(roots, np.uint32), oroots)
                                            and np.array_equal(np.array(last, np.uint32), olast))}
    out["fri_chain_committed"] = fc
    chain.close()
    del src
    torch.cuda.empty_cache()

    # ---- bit-reversals ----
    qa = torch.from_numpy(rng.integers(0, 0x7FFFFFFF, 4 * n, dtype=np.uint32).view(np.int32)).cuda()
    qb = torch.empty_like(qa)
    br = {}
    for name, Lx in libs.items():
        ms = _time_ms(lambda Lx=Lx: Lx.cuda_bit_reverse_qm31(qa.data_ptr(), qb.data_ptr(), n, log_n), ds, reps)
        br[f"qm31_{name}"] = {"ms": ms, "gbs": 32 * n / (ms / 1e3) / 1e9,
                              "frac": 32 * n / (ms / 1e3) / 1e9 / peak_gbs}
        ms = _time_ms(lambda Lx=Lx: Lx.cuda_bit_reverse_m31(qa.data_ptr(), log_n + 2), ds, reps)
        br[f"m31_2^{log_n + 2}_{name}"] = {"ms": ms, "gbs": 32 * n / (ms / 1e3) / 1e9,
                                          "frac": 32 * n / (ms / 1e3) / 1e9 / peak_gbs}
        ms = _time_ms(lambda Lx=Lx: Lx.cuda_permute_hc_to_canonic_brt(qa.data_ptr(), qb.data_ptr(), 4 * n, log_n + 2),
                      ds, reps)
        br[f"permute_m31_2^{log_n + 2}_{name}"] = {"ms": ms, "gbs": 32 * n / (ms / 1e3) / 1e9,
                                                  "frac": 32 * n / (ms / 1e3) / 1e9 / peak_gbs}
    out["bit_reverse"] = br
    del qa, qb
    torch.cuda.empty_cache()

    # ---- stwo NTT (PolyOps::evaluate_polynomials / interpolate, poly_ops.rs): one column of 2^(log_n-2) and a
    # batch of 16 columns of 2^(log_n-6), tables in stwo's layout built on the device; 8 B per element ----
    sn = {}
    for tag, lg, ncol in (("single", log_n - 2, 1), ("batch16", log_n - 6, 16)):
        m = 1 << lg
        tw = torch.empty(m // 2, dtype=torch.int32, device="cuda")
        itw = torch.empty(m // 2, dtype=torch.int32, device="cuda")
        _lib.check(_lib.lib().vx_stwo_twiddles(lg, 0, tw.data_ptr(), None))
        _lib.check(_lib.lib().vx_stwo_twiddles(lg, 1, itw.data_ptr(), None))
        cols = [torch.from_numpy(m31_array(SEED + 8 + c, m).view("int32")).cuda() for c in range(ncol)]
        ptrs = (C.c_void_p * ncol)(*[c.data_ptr() for c in cols])
        outs = {}
        for name, Lx in libs.items():
            if ncol == 1:
                ev = lambda Lx=Lx: Lx.cuda_stwo_ntt_evaluate(cols[0].data_ptr(), tw.data_ptr(), m)
                it = lambda Lx=Lx: Lx.cuda_stwo_ntt_interpolate(cols[0].data_ptr(), itw.data_ptr(), m)
            else:
                ev = lambda Lx=Lx: Lx.cuda_stwo_ntt_batch_evaluate(ptrs, tw.data_ptr(), m, ncol)
                it = lambda Lx=Lx: Lx.cuda_stwo_ntt_batch_interpolate(ptrs, itw.data_ptr(), m, ncol)
            ev()
            outs[name] = hash(b"".join(bytes(c.cpu().numpy().tobytes()) for c in cols))
            it()
            b = 8 * m * ncol
            for op, fn in (("evaluate", ev), ("interpolate", it)):
                ms = _time_ms(fn, ds, reps)
                sn[f"{tag}_2^{lg}_{op}_{name}"] = {"ms": ms, "gbs": b / (ms / 1e3) / 1e9,
                                                   "frac": b / (ms / 1e3) / 1e9 / peak_gbs}
        sn[f"{tag}_values_equal"] = len(set(outs.values())) == 1
        del cols, tw, itw
    out["stwo_ntt"] = sn
    torch.cuda.empty_cache()

    # ---- zero-pad of 2^(log_n-2) coefficients into a 2^log_n-point buffer (prover.rs:308) ----
    zs = torch.from_numpy(m31_array(SEED + 7, n >> 2).view("int32")).cuda()
    zd = torch.empty(n, dtype=torch.int32, device="cuda")
    zp = {}
    for name, Lx in libs.items():
        Lx.cuda_zero_pad.argtypes = _lib._SIGS["cuda_zero_pad"]
        ms = _time_ms(lambda Lx=Lx: Lx.cuda_zero_pad(zs.data_ptr(), zd.data_ptr(), n >> 2, n), ds, reps)
        zb = 4 * (n >> 2) + 4 * n  # read the coefficients, write the buffer
        zp[name] = {"ms": ms, "gbs": zb / (ms / 1e3) / 1e9, "frac": zb / (ms / 1e3) / 1e9 / peak_gbs}
    out["zero_pad"] = zp
    del zs, zd
    torch.cuda.empty_cache()

    # ---- Fibonacci quotient over a 2^log_n-point evaluation (reads 4 B, writes 4 x 4 B per point) ----
    tr = torch.from_numpy(m31_array(SEED + 6, n).view("int32")).cuda()
    qo = [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(4)]
    qa = (C.c_uint32 * 4)(*[int(x) for x in rng.integers(0, 0x7FFFFFFF, 4)])
    qt, qs = {}, {}
    for name, Lx in libs.items():
        ms = _time_ms(lambda Lx=Lx: Lx.cuda_fibonacci_quotient(tr.data_ptr(), *[q.data_ptr() for q in qo], qa, n),
                      ds, reps)
        qs[name] = hash(b"".join(bytes(q.cpu().numpy().tobytes()) for q in qo))
        qt[name] = {"ms": ms, "gbs": 20 * n / (ms / 1e3) / 1e9, "frac": 20 * n / (ms / 1e3) / 1e9 / peak_gbs}
    qt["values_equal"] = len(set(qs.values())) == 1
    out["fibonacci_quotient"] = qt
    del tr, qo
    torch.cuda.empty_cache()

    # ---- stwo PolyOps: eval_at_point over 2^log_n coefficients (4 bytes each), barycentric_eval over
    # 2^(log_n-2) points (an M31 value and a QM31 weight: 20 bytes each), 256 blocks as poly_ops.rs launches ----
    from oracle import oracle as O_

    coeffs = torch.from_numpy(m31_array(SEED + 5, n).view("int32")).cuda()
    factors = torch.from_numpy(rng.integers(0, 0x7FFFFFFF, 4 * log_n, dtype=np.uint32).view(np.int32)).cuda()
    s1 = torch.empty(2 * n, dtype=torch.int32, device="cuda")
    s2 = torch.empty(n, dtype=torch.int32, device="cuda")
    nb = n >> 2
    weights = torch.from_numpy(rng.integers(0, 0x7FFFFFFF, 4 * nb, dtype=np.uint32).view(np.int32)).cuda()
    n_blocks = min((nb + 255) // 256, 256)
    part = torch.empty(4 * n_blocks, dtype=torch.int32, device="cuda")
    res = (C.c_uint32 * 4)()
    so, vals, parts = {}, {}, {}
    for name, Lx in libs.items():
        ms = _time_ms(lambda Lx=Lx: Lx.cuda_eval_at_point(coeffs.data_ptr(), factors.data_ptr(), res, n,
                                                          s1.data_ptr(), s2.data_ptr()), ds, reps)
        vals[name] = tuple(res)
        so[f"eval_at_point_2^{log_n}_{name}"] = {"ms": ms, "gbs": 4 * n / (ms / 1e3) / 1e9,
                                                 "frac": 4 * n / (ms / 1e3) / 1e9 / peak_gbs}
        ms = _time_ms(lambda Lx=Lx: Lx.cuda_barycentric_eval(coeffs.data_ptr(), weights.data_ptr(), nb,
                                                             part.data_ptr(), n_blocks), ds, reps)
        parts[name] = bytes(part.cpu().numpy().tobytes())
        so[f"barycentric_2^{log_n - 2}_{name}"] = {"ms": ms, "gbs": 20 * nb / (ms / 1e3) / 1e9,
                                                   "frac": 20 * nb / (ms / 1e3) / 1e9 / peak_gbs}
    so["values_equal"] = len(set(vals.values())) == 1 and len(set(parts.values())) == 1
    if cpu:
        hc = coeffs.cpu().numpy().view(np.uint32)
        hf = factors.cpu().numpy().view(np.uint32).reshape(log_n, 4)
        t0 = time.perf_counter()
        ov = O_.eval_at_point(hc, hf)
        so["eval_at_point_cpu_baseline"] = {"ms": 1e3 * (time.perf_counter() - t0), "cores": 1, "kind": "port",
                                            "equal": tuple(int(x) for x in ov) == vals["vortex"]}
        hw = weights.cpu().numpy().view(np.uint32).reshape(nb, 4)
        t0 = time.perf_counter()
        op = O_.barycentric_partials(hc[:nb], hw, n_blocks)
        so["barycentric_cpu_baseline"] = {"ms": 1e3 * (time.perf_counter() - t0), "cores": 1, "kind": "port",
                                          "equal": op.tobytes() == parts["vortex"]}
    out["stwo_poly_ops"] = so
    del coeffs, factors, s1, s2, weights, part
    torch.cuda.empty_cache()

    # ---- twiddle tables of half_coset(log_n), forward and inverse, by the reference's call sequence
    # (circle.rs:454-550: coset points, one extract-and-squash per line layer, batch inverses) ----
    from vortexstark_b200.circle import Coset

    co = Coset.half_coset(log_n)
    xs, ys = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    line, iline = (torch.empty(n - 1, dtype=torch.int32, device="cuda") for _ in range(2))
    icirc = torch.empty(n // 2, dtype=torch.int32, device="cuda")
    sq = [torch.empty(n >> (j + 1), dtype=torch.int32, device="cuda") for j in range(log_n - 1)]
    tw, tables = {}, {}
    for name, Lx in libs.items():
        def build(Lx=Lx):
            Lx.cuda_compute_coset_points(co.initial.x, co.initial.y, co.step.x, co.step.y, xs.data_ptr(),
                                         ys.data_ptr(), n)
            cur, m, off = xs, n, 0
            for j in range(log_n - 1):
                Lx.cuda_extract_and_squash(cur.data_ptr(), line.data_ptr() + 4 * off, sq[j].data_ptr(), m // 2)
                off += m // 2
                cur, m = sq[j], m // 2
            Lx.cuda_batch_inverse_m31(line.data_ptr(), iline.data_ptr(), n - 1)
            Lx.cuda_batch_inverse_m31(ys.data_ptr(), icirc.data_ptr(), n // 2)
        ms = _time_ms(build, ds, reps)
        tables[name] = hash(bytes(line.cpu().numpy().tobytes()) + bytes(iline.cpu().numpy().tobytes())
                            + bytes(icirc.cpu().numpy().tobytes()))
        # bytes: coset points 8n written; the line layers 16n (each reads its points, writes its twiddles and
        # the squashed points); the batch inverses 12n (read and write n - 1 + n/2 words)
        tb = 36 * n
        tw[name] = {"ms": ms, "gbs": tb / (ms / 1e3) / 1e9, "frac": tb / (ms / 1e3) / 1e9 / peak_gbs}
    tw["bytes"] = 36 * n
    tw["tables_equal"] = len(set(tables.values())) == 1
    out["twiddle_tables"] = tw
    del xs, ys, line, iline, icirc, sq
    torch.cuda.empty_cache()
    return out


def pow_benchmark(probe_rate: float, bits: int = 26, cpu: bool = True):
    """Proof-of-work search at 26 bits (stwo's order (hi << 32) | low) from a
    seeded channel state: device time of vx_grind_pow and the candidates it
    had to hash, beside the CPU oracle's search of the same nonce."""
    import hashlib
    import struct

    from vortexstark_b200.channel import Channel
    from vortexstark_b200.grind import grind_prefixed

    ch = Channel()
    ch.mix_digest(struct.unpack("<8I", hashlib.blake2s(struct.pack("<Q", SEED)).digest()))
    pre = ch.pow_prefix(bits)
    grind_prefixed(pre, 8)  # warm-up
    times, nonce = [], 0
    for _ in range(3):
        t0 = time.perf_counter()
        nonce = grind_prefixed(pre, bits)
        times.append(time.perf_counter() - t0)
    t = statistics.median(times)
    # candidates at or before the answer in the search order (hi * 2^20 + low + 1):
    # the work any search that returns the smallest nonce must do
    below = (nonce >> 32) * (1 << 20) + (nonce & 0xFFFFFFFF) + 1
    launches = (nonce >> 32) // 64 + 1
    out = {"pow_bits": bits, "nonce": nonce, "valid": ch.verify_pow_nonce(bits, nonce), "ms": 1e3 * t,
           "candidates_to_answer": below, "launches": launches,
           "candidates_per_s": below / t, "frac_of_probe": below / t / probe_rate,
           "probe_compressions_per_s": probe_rate,
           "note": "host-timed around the synchronous call (launches of 64 x 2^20 candidates, result read back "
                   "between launches); each candidate is one Blake2s compression"}
    if cpu:
        from oracle import oracle as O

        O.lib()
        t0 = time.perf_counter()
        cn = O.grind_pow(list(pre), bits)
        out["cpu_baseline"] = {"ms": 1e3 * (time.perf_counter() - t0), "nonce_equal": cn == nonce,
                               "cores": O.get_threads(), "kind": "port"}
    return out


def blake2s_probe_rate(stream) -> float:
    """Register-only Blake2s compressions/s on this GPU (the ALU roofline)."""
    import torch

    from vortexstark_b200 import _lib

    L = _lib.lib()
    s = stream.cuda_stream
    out = torch.empty(148 * 8 * 256, dtype=torch.int32, device="cuda")
    iters = 256
    _lib.check(L.vx_probe_blake2s(148 * 8, 256, iters, out.data_ptr(), s))
    pa, pb = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    pa.record(stream)
    _lib.check(L.vx_probe_blake2s(148 * 8, 256, iters, out.data_ptr(), s))
    pb.record(stream)
    stream.synchronize()
    return 148 * 8 * 256 * iters / (pa.elapsed_time(pb) / 1e3)


def _rounded(x):
    """Floats to six significant digits, in nested dicts and lists."""
    if isinstance(x, float):
        return float(f"{x:.6g}")
    if isinstance(x, dict):
        return {k: _rounded(v) for k, v in x.items()}
    return [_rounded(v) for v in x] if isinstance(x, list) else x


def _timed_leaves(d, path=()):
    """(path, dict) of every timed measurement in a microbench object."""
    for k, v in d.items():
        if isinstance(v, dict):
            if "ms" in v:
                yield path + (k,), v
            yield from _timed_leaves(v, path + (k,))


def _flags(d):
    """Every equality or validity flag of a nested object."""
    for k, v in d.items():
        if isinstance(v, dict):
            yield from _flags(v)
        elif isinstance(v, bool) and ("equal" in k or k == "valid"):
            yield v


def summary_line(full):
    """The bench line: the headline whole, every other leg as its figures.  It
    stays below 2900 characters, short enough for a log that keeps the last
    3000 (with the served sweeps it came to 22 000); --full prints all."""
    top = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
           "vs_baseline", "dtype", "data")
    out = {k: full[k] for k in top}
    out["config"] = {k: full["config"][k] for k in ("workload", "log_n", "blowup_bits", "n_queries", "parallelism",
                                                    "in_flight", "l2")}
    out["config"]["in_flight"] = out["config"]["in_flight"].split(" (")[0]
    out["e2e"] = {**full["e2e"], "api": full["e2e"]["api"].split(" ")[0]}
    out["gpu_launches"] = full["gpu_launches"]
    out["clocks"] = full["clocks"]
    for k in ("value_one_in_flight", "p50_ms", "p99_ms", "lde_hbm_gbs"):
        out[k] = full[k]
    out["roofline"] = {k: full["roofline"][k] for k in ("bound", "achieved", "peak", "unit", "frac",
                                                        "frac_of_nominal", "traffic")}
    out["roofline"]["kernel"] = full["roofline"]["kernel"].split(":")[0]
    out["lde_roofline"] = {k: full["lde_roofline"][k] for k in ("bound", "peak", "frac", "traffic")}
    out["stages_ms"] = {k: float(f"{v:.4g}") for k, v in full["stages_ms"].items()}
    kernels = {}  # [ms, share of its bound]
    for leg in ("ntt_microbench", "kernel_microbench"):
        for path, v in _timed_leaves(full.get(leg, {})):
            if any("reference" in p or "cpu" in p for p in path):
                continue
            name = "/".join(p for p in path if p not in ("vortex", "evaluate", "interpolate"))
            name = name.replace("_vortex", "")
            if leg == "ntt_microbench":
                name = "ntt_" + name + {"evaluate": "_e", "interpolate": "_i"}.get(path[-1], "")
            frac = v.get("frac", v.get("frac_of_probe"))
            kernels[name] = [float(f"{v['ms']:.4g}")] + ([round(frac, 3)] if frac is not None else [])
    if kernels:
        out["kernels"] = kernels
    if "pow_grind" in full:
        out["pow_grind"] = {k: full["pow_grind"][k] for k in ("candidates_per_s", "frac_of_probe")}
    if "batched_commit" in full:
        b = full["batched_commit"]
        out["batched_commit"] = {"value": b["value"], "one_in_flight": b["value_one_in_flight"],
                                 "e2e": b["e2e"]["value"]}
    if "served" in full:
        sv = full["served"]
        out["served"] = {"plain_capacity": sv["plain_capacity_per_s"],
                         "engine_peak": max(r["proofs_per_s"] for r in sv["served_sweep"]),
                         "ratio_at_equal_p99": list(sv["speedup_at_equal_p99"].values())}
    flags = list(_flags(full))
    if flags:
        out["outputs_equal"] = f"{sum(flags)}/{len(flags)}"
    if "cpu_baseline" in full:
        out["cpu_baseline"] = full["cpu_baseline"]
    return _rounded(out)


def max_over_ranks(values, dist, device="cpu"):
    """Each value's maximum over the ranks (a replica job is as slow as its
    slowest GPU); the values themselves when there is one rank."""
    if dist is None:
        return list(values)
    import torch

    t = torch.tensor([float(v) for v in values], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return [float(x) for x in t.cpu()]


def rank_inputs(rank: int, count: int):
    """Public inputs of one rank's proofs: a replica per GPU, each its own seeded stream."""
    from vortexstark_b200.workload import fib_inputs

    return fib_inputs(SEED + rank, count)


def run_reference(args, rank: int):
    """CPU oracle arm: each step one proof of the workload (or a bounded
    sample of it), all host threads."""
    if rank != 0:
        return
    from oracle import oracle as O
    from vortexstark_b200.workload import fib_inputs

    O.lib()
    cores = O.get_threads()
    ins = fib_inputs(SEED, args.steps + args.warmup)
    for a, b in ins[: args.warmup]:
        O.prove(a, b, 16)
    a, b = ins[0]
    t0 = time.perf_counter()
    O.prove(a, b, 20)
    t20 = time.perf_counter() - t0
    per = t20 * 2.0 ** (args.log_n - 20) * (args.log_n + 2) / 22.0
    full = per * args.steps <= 240.0
    k = args.log_n if full else args.log_n - 2
    scale = 1.0 if full else (1 << (args.log_n - k)) * (args.log_n + 2) / (k + 2)
    times = []
    for a, b in ins[args.warmup:]:
        t0 = time.perf_counter()
        O.prove(a, b, k)
        times.append(time.perf_counter() - t0)
    total = sum(times) * scale
    value = args.steps / total
    sample = (f"each step one full log_n={k} proof" if full else
              f"each step one log_n={k} proof scaled by the N log N work ratio {scale:.2f} to log_n={args.log_n}")
    line = {
        "metric": METRIC, "value": value, "unit": "proofs/s", "impl": "reference", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1000.0 * total / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32 (M31)",
        "data": "synthetic (seeded SplitMix64 public inputs)",
        "config": {"workload": f"fibonacci_stark log_n={args.log_n} blowup=4 queries=80 (2^{args.log_n + 2}-point LDE)",
                   "log_n": args.log_n, "blowup_bits": 2, "n_queries": 80, "parallelism": "cpu"},
        "cpu_baseline": {"value": value, "unit": "proofs/s", "cores": cores, "kind": "port", "sample": sample},
        "e2e": {"value": value, "unit": "proofs/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "p50_ms": 1000.0 * statistics.median(times) * scale,
        "p99_ms": 1000.0 * max(times) * scale,
    }
    print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="vortex", choices=["vortex", "reference"])
    ap.add_argument("--log-n", type=int, default=24)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-served", action="store_true", help="skip the mixed-size served stream")
    ap.add_argument("--no-batched", action="store_true", help="skip the batched lifted commitment")
    ap.add_argument("--no-micro", action="store_true", help="skip the NTT / iNTT microbench (2^20, 2^24, 2^28)")
    ap.add_argument("--no-tune", action="store_true", help="keep the built-in NTT plans and leaf-kernel shapes")
    ap.add_argument("--full", action="store_true", help="print every leg's whole object, sweeps and sources included")
    ap.add_argument("--kernels-only", action="store_true",
                    help="run only the standalone kernel microbench (Merkle, FRI folds, bit reversals) and print it")
    ap.add_argument("--kernel-log", type=int, default=26, help="log2 size of the standalone kernel microbench")
    ap.add_argument("--batched-only", action="store_true",
                    help="run only the batched lifted commitment and print its object")
    ap.add_argument("--lde-only", action="store_true",
                    help="run only the LDE (trace, interpolate, evaluate) of one proof slot, --steps times inside "
                         "an NVTX range 'lde', and print its time (the small case for profiling the NTT passes)")
    ap.add_argument("--trace-commit-only", action="store_true",
                    help="run only the trace commitment (Blake2s tree of the LDE) of one proof slot, --steps times "
                         "inside an NVTX range 'trace_commit', and print its time (the small case for profiling the "
                         "tree kernels)")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))

    if args.impl == "reference":
        run_reference(args, rank)
        return

    import torch

    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime

        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120),
                                device_id=torch.device("cuda", local))

    # per-device launch shapes, chosen before any slot or context is carved
    tuned = None
    if not args.no_tune:
        from vortexstark_b200 import tune

        t0 = time.perf_counter()
        tune_log = min(28, max(args.log_n + 2, 0 if args.no_micro else 28))
        tuned = tune.autotune(tune_log)
        tuned = {"max_log": tune_log, "seconds": round(time.perf_counter() - t0, 2),
                 "ntt_plan": {k: v[:2] for k, v in tuned["ntt"].items()},
                 "leaf_k": {k: v[0] for k, v in tuned["leaf_k"].items()},
                 "fold_leaf_k": {k: v[0] for k, v in tuned["fold_leaf_k"].items()}}

    if args.kernels_only:
        peak, _ = _peaks()
        probe = blake2s_probe_rate(torch.cuda.Stream())
        res = kernel_microbench(peak, probe, log_n=args.kernel_log, cpu=not args.no_cpu_baseline)
        if rank == 0:
            print(json.dumps({"kernel_microbench": res}), flush=True)
        return

    if args.trace_commit_only:
        res = trace_commit_only(args.log_n, args.steps, args.warmup)
        if rank == 0:
            print(json.dumps({"trace_commit_only": res}), flush=True)
        return

    if args.lde_only:
        res = lde_only(args.log_n, args.steps, args.warmup)
        if rank == 0:
            print(json.dumps({"lde_only": res}), flush=True)
        return

    if args.batched_only:
        peak, _ = _peaks()
        probe = blake2s_probe_rate(torch.cuda.Stream())
        res = batched_commit_benchmark(SEED, max(args.steps, 5), args.warmup, peak, probe,
                                       cpu=not args.no_cpu_baseline)
        if rank == 0:
            print(json.dumps({"batched_commit": res}), flush=True)
        return

    import ctypes as C

    from vortexstark_b200 import _lib, prover
    from vortexstark_b200.workload import fib_inputs

    L = _lib.lib()
    log_n = args.log_n
    cache = prover.ProverCache(log_n)
    # IN_FLIGHT slots on as many streams keep that many proofs in flight (the
    # batch API's depth); a slot after the first only while it fits in half of
    # the free device memory
    caches = [cache]
    while len(caches) < IN_FLIGHT and 2 * cache.slot_bytes() < torch.cuda.mem_get_info()[0]:
        caches.append(prover.ProverCache(log_n))
    size = cache.size
    ins = rank_inputs(rank, args.steps + args.warmup)
    streams = [torch.cuda.Stream() for _ in caches]
    stream = streams[0]
    s = stream.cuda_stream
    slots = list(zip(caches, streams))
    nslot = len(slots)
    timed = ins[args.warmup:]
    K = len(timed)
    batch_a = (C.c_uint32 * K)(*[x[0] for x in timed])
    batch_b = (C.c_uint32 * K)(*[x[1] for x in timed])
    batch_out = (C.c_uint8 * (K * size))()
    batch_sz = C.c_size_t()

    def barrier():
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize()

    # warm-up (device path and e2e path)
    host = torch.empty(size, dtype=torch.uint8, pin_memory=True)
    out_len = C.c_size_t()
    for j, (a, b) in enumerate(ins[: args.warmup]):
        c, st = slots[j % nslot]
        _lib.check(L.vx_prover_prove_async(c._p, a, b, st.cuda_stream))
        _lib.check(L.vx_prove_fib(a, b, log_n, 2, 80, host.data_ptr(), size, C.byref(out_len)))
    for c, st in slots:  # every slot has proved once before the timed region
        _lib.check(L.vx_prover_prove_async(c._p, ins[0][0], ins[0][1], st.cuda_stream))
    # the batch API's slots are created by its first call with IN_FLIGHT or more proofs
    nw = max(IN_FLIGHT, 2)
    wa = (C.c_uint32 * nw)(*[ins[i % len(ins)][0] for i in range(nw)])
    wb = (C.c_uint32 * nw)(*[ins[i % len(ins)][1] for i in range(nw)])
    warm_out = (C.c_uint8 * (nw * size))()
    _lib.check(L.vx_prove_fib_batch(wa, wb, nw, log_n, 2, 80, warm_out, nw * size, C.byref(batch_sz)))
    del warm_out
    torch.cuda.synchronize()
    launches_per_proof = int(L.vx_prover_launches(cache._p))

    clk = ClockSampler(local)
    clk.start()
    # ---- device-resident throughput: nslot proofs in flight (one slot and stream each) ----
    barrier()
    cur = torch.cuda.current_stream()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.nvtx.range_push("timed_proofs")  # lets a profiler select exactly these launches
    e0.record(cur)
    for st in streams:
        st.wait_stream(cur)
    for j, (a, b) in enumerate(timed):
        c, st = slots[j % nslot]
        _lib.check(L.vx_prover_prove_async(c._p, a, b, st.cuda_stream))
    for st in streams:
        cur.wait_stream(st)
    e1.record(cur)
    e1.synchronize()
    torch.cuda.nvtx.range_pop()
    barrier()
    dev_ms = e0.elapsed_time(e1)
    for c in caches:
        _lib.check(L.vx_prover_check(c._p))
    # the same proofs one at a time on one stream, for comparison
    e2, e3 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e2.record(stream)
    for a, b in timed:
        _lib.check(L.vx_prover_prove_async(cache._p, a, b, s))
    e3.record(stream)
    stream.synchronize()
    dev_ms_one = e2.elapsed_time(e3)
    _lib.check(L.vx_prover_check(cache._p))

    # ---- end to end through the C ABI with host buffers: vx_prove_fib_batch ----
    barrier()
    t0 = time.perf_counter()
    _lib.check(L.vx_prove_fib_batch(batch_a, batch_b, K, log_n, 2, 80, batch_out, K * size, C.byref(batch_sz)))
    t_all = (time.perf_counter() - t0) * 1e3
    barrier()
    # ---- per-proof latency: one vx_prove_fib call per proof ----
    lat = []
    for a, b in timed:
        ea, eb = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ea.record(torch.cuda.current_stream())
        _lib.check(L.vx_prove_fib(a, b, log_n, 2, 80, host.data_ptr(), size, C.byref(out_len)))
        eb.record(torch.cuda.current_stream())
        eb.synchronize()
        lat.append(ea.elapsed_time(eb))
    barrier()
    clocks = clk.stop()

    # ---- stage timing: LDE roofline, Merkle ALU roofline ----
    reps = 5
    a, b = ins[0]
    _lib.check(L.vx_prover_stage_async(cache._p, 0, a, b, s))
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2 * reps)]
    lde_ms = []
    for r in range(reps):
        ev[2 * r].record(stream)
        _lib.check(L.vx_prover_stage_async(cache._p, 1, a, b, s))
        _lib.check(L.vx_prover_stage_async(cache._p, 2, a, b, s))
        ev[2 * r + 1].record(stream)
        _lib.check(L.vx_prover_stage_async(cache._p, 0, a, b, s))  # regenerate the trace (not timed)
    stream.synchronize()
    lde_ms = [ev[2 * r].elapsed_time(ev[2 * r + 1]) for r in range(reps)]
    n, N = 1 << log_n, 1 << (log_n + 2)
    lde_bytes = 8 * n + 4 * n + 4 * N
    lde_t = statistics.median(lde_ms) / 1e3
    peak, peak_kind = _peaks()
    lde_gbs = lde_bytes / lde_t / 1e9

    tc = [torch.cuda.Event(enable_timing=True) for _ in range(2 * reps)]
    for r in range(reps):
        tc[2 * r].record(stream)
        _lib.check(L.vx_prover_stage_async(cache._p, 3, a, b, s))
        tc[2 * r + 1].record(stream)
    stream.synchronize()
    tcommit_t = statistics.median([tc[2 * r].elapsed_time(tc[2 * r + 1]) for r in range(reps)]) / 1e3
    compressions = 2 * N - 1
    probe_rate = blake2s_probe_rate(stream)
    merkle_rate = compressions / tcommit_t
    sm_mhz = float((clocks or {}).get("sm_mhz") or 1965.0)
    alu_nominal = 148 * 64 * sm_mhz * 1e6 / 640

    # per-stage device time of one proof (vx_prover_stage_async, stages in order)
    stage_names = ["trace", "interpolate", "lde_evaluate", "trace_commit", "quotient_commit",
                   "circle_fold_commit", "line_folds_commit", "queries", "decommit"]
    st_ev = [[torch.cuda.Event(enable_timing=True) for _ in range(len(stage_names) + 1)] for _ in range(reps)]
    for r in range(reps):
        for k in range(len(stage_names)):
            st_ev[r][k].record(stream)
            _lib.check(L.vx_prover_stage_async(cache._p, k, a, b, s))
        st_ev[r][-1].record(stream)
    stream.synchronize()
    stages_ms = {name: statistics.median([st_ev[r][k].elapsed_time(st_ev[r][k + 1]) for r in range(reps)])
                 for k, name in enumerate(stage_names)}

    # the job's times are its slowest rank's
    dev_ms, t_all, dev_ms_one = max_over_ranks([dev_ms, t_all, dev_ms_one], dist, "cuda")

    steps = args.steps
    value = world * steps / (dev_ms / 1e3)
    e2e = world * steps / (t_all / 1e3)
    lat.sort()
    p99 = lat[min(len(lat) - 1, int(round(0.99 * (len(lat) - 1))))]

    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": "proofs/s", "n_gpus": world, "steps": steps,
            "warmup": args.warmup, "ms_per_step": dev_ms / steps, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "u32 (M31)", "data": "synthetic (seeded SplitMix64 public inputs)",
            "config": {"workload": f"fibonacci_stark log_n={log_n} blowup=4 queries=80 (2^{log_n + 2}-point LDE)",
                       "stream": f"value, e2e and p50/p99 are single-size log_n={log_n} proofs; the metric's mixed "
                                 "log_n 16-24 stream is under served (engine and plain one-at-a-time path)",
                       "log_n": log_n, "blowup_bits": 2, "n_queries": 80,
                       "parallelism": f"replicas x{world}",
                       "in_flight": f"{nslot} proofs per GPU ({nslot} slots on {nslot} streams, the depth of "
                                    "vx_prove_fib_batch); value_one_in_flight is the same proofs one at a time "
                                    "on one stream",
                       "l2": (f"per-step working set > L2 (LDE {4 << (log_n + 2) >> 20} MiB + FRI layers "
                              f"{16 << (log_n + 2) >> 20} MiB); no flush needed" if log_n >= 22 else
                              "per-step working set below L2 at this size: a reduced case, not the headline")},
            "e2e": {"value": e2e, "unit": "proofs/s", "h2d_bytes_per_step": 8, "d2h_bytes_per_step": size,
                    "api": "vx_prove_fib_batch (ProverPipeline::prove_batch) over the timed inputs, proof bytes "
                           "into a host buffer; host-timed around the synchronous call"},
            "value_one_in_flight": world * steps / (dev_ms_one / 1e3),
            "p50_ms": statistics.median(lat), "p99_ms": p99,
            "latency_api": "vx_prove_fib, one call per proof, CUDA events",
            "lde_hbm_gbs": lde_gbs,
            # the dominant kernel: the Blake2s leaf subtrees (~94% of a proof), bound by the integer ALU pipe
            "roofline": {"bound": "int-alu",
                         "kernel": f"trace commitment: leaf_subtree_kernel<LeafM31> + node/reduce kernels "
                                   f"(2^{log_n + 2} leaves, 2^{log_n + 3} - 1 compressions)",
                         "achieved": merkle_rate / 1e9, "peak": probe_rate / 1e9, "unit": "G compressions/s",
                         "frac": merkle_rate / probe_rate, "time_ms": tcommit_t * 1e3,
                         "peak_source": "measured in this run: a register-only chain of the same Blake2s compression "
                                        "on every SM (vx_probe_blake2s)",
                         "peak_nominal": alu_nominal / 1e9,
                         "frac_of_nominal": merkle_rate / alu_nominal,
                         "nominal_source": f"ALU-pipe ceiling: 148 SMs x 64 lanes x {sm_mhz:.0f} MHz (median SM clock "
                                           "of the timed region) / 640 ALU-pipe ops per compression (10 rounds x 8 G x "
                                           "4 xor + 4 rotate; the additions run on the FMA pipe)",
                         "traffic": TRACE_COMMIT_TRAFFIC_LOG24 if log_n == 24 else None,
                         "traffic_source": TRACE_COMMIT_TRAFFIC_SOURCE,
                         "algorithmic_bytes": 4 * (1 << (log_n + 2)),
                         "algorithmic_note": "the leaves read once (4 B each); the stored tree levels written for the "
                                             "decommitment (32 B per hash at heights 4, 8, ...) are outputs on top"},
            "lde_roofline": {"bound": "hbm",
                             "kernel": f"LDE (interpolate 2^{log_n} + zero-pad + evaluate 2^{log_n + 2})",
                             "achieved": lde_gbs, "peak": peak, "unit": "GB/s", "frac": lde_gbs / peak,
                             "peak_source": peak_kind,
                             "traffic": LDE_TRAFFIC_LOG24 if log_n == 24 else None,
                             "traffic_source": LDE_TRAFFIC_SOURCE,
                             "algorithmic_bytes": lde_bytes, "time_ms": lde_t * 1e3},
            "stages_ms": stages_ms,
            "stage_rooflines": stage_roofline_table(stages_ms, log_n, peak, probe_rate),
            "gpu_launches": launches_per_proof * steps,
            "launches_per_proof": launches_per_proof,
            "clocks": clocks,
            "autotune": tuned,
        }
        if world == 1 and not args.no_micro:
            line["ntt_microbench"] = ntt_microbench(peak)
            line["kernel_microbench"] = kernel_microbench(peak, probe_rate, cpu=not args.no_cpu_baseline)
            line["pow_grind"] = pow_benchmark(probe_rate, cpu=not args.no_cpu_baseline)
        if world == 1 and not args.no_batched:
            line["batched_commit"] = batched_commit_benchmark(SEED, max(steps, 5), args.warmup, peak, probe_rate,
                                                              cpu=not args.no_cpu_baseline)
        if world == 1 and not args.no_served:
            cache.close()
            line["served"] = served_benchmark(SEED)
        if world == 1 and not args.no_cpu_baseline:
            cb = cpu_baseline(log_n)
            cb.pop("seconds", None)
            line["cpu_baseline"] = cb
        print(json.dumps(line) if args.full else json.dumps(summary_line(line), separators=(",", ":")), flush=True)
    cache.close()
    if dist is not None:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
