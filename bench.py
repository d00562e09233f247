#!/usr/bin/env python3
"""bench.py -- K/s of the AP26 10-shift per-K search on B200.

Workload (N=1): 64 consecutive K starting at the seeded KMIN 43241056
(numpy default_rng(26).integers(1e6, 5e7 - 64)), SHIFT=0 -- the plain-GPU
drop-in configuration.  A step is one batch of 8 consecutive K (its
searchable ones) through the batched persistent pipeline
(ap26_search_batch); 8 steps cover the 64-K range.  With N ranks
(torchrun), each rank searches its own 64-K range (KMIN + 64*rank): weak
scaling, no collective on the data path (replicas of an independent
search).

  value    K/s over all ranks from CUDA-event device time of the pipeline
           (inputs are (K, SHIFT) scalars; nothing to stage)
  e2e      K/s wall-clock through the C ABI with host buffers: ap26_search_batch
           (raw reports, result_hash) and ap26_report_batch (SOL lines), with
           their host<->device copies; ReportSolution runs on the device
  roofline the class sieve kernel: the table rows that its dense phase reads
           (20 moduli x 64 bytes for every point and row that 71 does not
           exclude) / measured sieve launch time, against the measured
           shared-memory peak
  cpu_baseline  the reference CPU build (oracle/_ref/ref_harness: the
           reference's own Search_avx2) on every host core, bounded samples
  cpu_avx512    companion: the AVX-512 restatement of the same search
           (oracle/ap26_avx512.c) on every host core, bounded sample

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
"""
import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

KMIN_SEEDED = 43241056          # numpy default_rng(26).integers(1_000_000, 50_000_000 - 64)
RANGE_K = 64
STEP_K = 8
SHIFT = 0
N59_PER_K = 4808136200          # lattice positions per K (10840 n43 x 443555)
# The class sieve's dense rows, per lattice value and shift word: a point is 8
# lattice values of 10 words each, its (b, j) that pass 61 and 67 fill 4 rows of
# 512 bits, 27.6% of their quarters are excluded by 71, and the others are read
# in the tables of 20 moduli.
ROW_BYTES_PER_CELL = 4 * 64 * 20 * 0.724 / 80
# H2D/D2H payload per K-job and per call (sizes of the C ABI structures)
KJOB_BYTES, DEVSTATE_BYTES, APREC_BYTES, COUNT_BYTES, FINAL_BYTES = 128, 128, 24, 8, 56
REF_HARNESS = os.path.join(ROOT, "oracle", "_ref", "ref_harness")


def will_search(k):
    return all(k % p for p in (29, 31, 37, 41, 43, 47, 53, 59))


_T0 = time.time()


def progress(msg):
    """One line per phase on stderr, so a slow phase shows where it is."""
    print(f"[bench {time.time() - _T0:7.1f}s] {msg}", file=sys.stderr, flush=True)


# ---- clocks during the timed region -------------------------------------------
class ClockSampler:
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device):
        self.device = device
        self.samples = []
        self.proc = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.Q}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None
        return self

    def _read(self):
        for ln in self.proc.stdout:
            self.samples.append([x.strip() for x in ln.split(",")])

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(s[1]) for s in self.samples if s[1].replace(".", "").isdigit()]
        mx = [float(s[2]) for s in self.samples if s[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = set()
        for s in self.samples:
            for i, nm in enumerate(names):
                if len(s) > 5 + i and s[5 + i].lower() == "active":
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(mx) if mx else None, "reasons": sorted(reasons),
                "samples": len(self.samples)}


# ---- CPU baseline: the reference's own search on all host cores ------------------
PASS_ITERS = (0, 4, 8)          # Search_avx2's three passes (shift words 0-3, 4-7, 8-9)
N43_PER_PASS = 10840


def ref_sample(ks, ticks):
    """One ref_harness process per host core, all concurrent: process i
    runs the pass starting at shift word PASS_ITERS[i % 3] of K ks[i] and is
    stopped after `ticks` of the pass's 85 (i31, i37) pairs.  Each pass's
    time per lattice value comes from the first tick to the stop (its table
    set-up is timed separately), so a K costs
    sum over passes of (set-up + 10840 x time per value).
    Returns (K/s on these cores, wall seconds, processes)."""
    t0 = time.time()
    procs = [subprocess.Popen([REF_HARNESS, "sample", str(k), str(SHIFT), str(ticks), "avx2",
                               str(PASS_ITERS[i % len(PASS_ITERS)])],
                              stdout=subprocess.PIPE, text=True) for i, k in enumerate(ks)]
    per_value = {it: [] for it in PASS_ITERS}
    setup = {it: [] for it in PASS_ITERS}
    for p in procs:
        out, _ = p.communicate()
        for ln in out.splitlines():
            if ln.startswith("SAMPLE"):
                f = ln.split()
                done, it, setup_s, tick_s = int(f[2]), int(f[6]), float(f[7]), float(f[8])
                if done > 0:
                    per_value[it].append(tick_s / done)
                    setup[it].append(setup_s)
    wall = time.time() - t0
    k_seconds = sum(statistics.mean(setup[it]) + N43_PER_PASS * statistics.mean(per_value[it])
                    for it in PASS_ITERS)
    return len(ks) / k_seconds, wall, len(ks)


def port_sample(ks, seconds=10.0):
    """Fallback when the reference binary is absent: the oracle port timed on
    a bounded slice of each K's lattice (one thread per K)."""
    import ctypes
    import numpy as np
    from concurrent.futures import ThreadPoolExecutor
    L = ctypes.CDLL(os.path.join(ROOT, "oracle", "liboracle.so"))
    L.ao_search.restype = ctypes.c_int64
    f_span = 2_000_000
    def one(k):
        cap = 4096
        a = np.zeros(cap, np.int32); b = np.zeros(cap, np.int64); c = np.zeros(cap, np.uint64)
        nc = ctypes.c_int64()
        L.ao_search(k, SHIFT, ctypes.c_int64(0), ctypes.c_int64(f_span),
                    a.ctypes.data_as(ctypes.c_void_p), b.ctypes.data_as(ctypes.c_void_p),
                    c.ctypes.data_as(ctypes.c_void_p), ctypes.c_int64(cap), ctypes.byref(nc), 1)
    t0 = time.time()
    with ThreadPoolExecutor(len(ks)) as ex:
        list(ex.map(one, ks))
    return len(ks) * f_span / 4808136200, time.time() - t0, len(ks)


def cpu_baseline_value(ks_pool, ticks):
    ncores = os.cpu_count() or 1
    ks = [ks_pool[i % len(ks_pool)] for i in range(ncores)]
    if os.access(REF_HARNESS, os.X_OK) and ncores >= len(PASS_ITERS):
        kps, secs, n = ref_sample(ks, ticks)
        kind = "reference"
        sample = (f"reference Search_avx2 (oracle/_ref/ref_harness), {n} concurrent processes, "
                  f"each the first {ticks} of 85 progress ticks of one of the 3 passes of one K "
                  "(SHIFT=0, K from the workload); per-pass time per lattice value x 10840 + "
                  "set-up, summed over the passes")
    else:
        frac, secs, n = port_sample(ks)
        kps = frac / secs
        kind = "port"
        sample = f"oracle port, {n} threads x 2e6 lattice values of one K each"
    return {"value": kps, "unit": "K/s", "cores": n, "kind": kind, "sample": sample,
            "seconds": round(secs, 2)}


def avx512_companion(k, seconds=8.0):
    """The AVX-512 restatement (oracle/ap26_avx512.c: sieve + chain walk) on
    every host core over a bounded lattice slice of one K of the workload,
    sized from a short calibration run to take about `seconds`; None on a
    CPU without AVX-512 VBMI2."""
    import ctypes
    import numpy as np
    L = ctypes.CDLL(os.path.join(ROOT, "oracle", "liboracle.so"))
    if not L.a5_supported():
        return None
    L.a5_search.restype = ctypes.c_int64
    ncores = os.cpu_count() or 1
    cap = 1 << 16
    bufs = [np.zeros(cap, t) for t in (np.int32, np.int64, np.int64, np.uint64)]
    def run(span):
        t0 = time.time()
        n = L.a5_search(k, SHIFT, ctypes.c_int64(0), ctypes.c_int64(span),
                        *[b.ctypes.data_as(ctypes.c_void_p) for b in bufs],
                        ctypes.c_int64(cap), None, ncores)
        assert n >= 0
        return time.time() - t0
    cal = 200_000 * ncores
    t = run(cal)
    span = int(min(N59_PER_K, max(cal, cal * seconds / max(t, 1e-3))))
    secs = run(span)
    return {"value": span / N59_PER_K / secs, "unit": "K/s", "cores": ncores, "kind": "port",
            "sample": f"AVX-512 restatement (oracle/ap26_avx512.c), {ncores} threads over "
                      f"lattice positions [0, {span}) of K={k} (SHIFT=0)",
            "seconds": round(secs, 2)}


# ---- parity against the reference's own results ---------------------------------
GOLDEN = os.path.join(ROOT, "tests", "golden")


def ref_fixture(K, shift):
    """The reference's raw reports of (K, SHIFT), recorded from its own
    Search_avx2 (tests/golden/ref_raw), or None where none is recorded."""
    path = os.path.join(GOLDEN, "ref_raw", f"shift{shift}", f"{K}.txt")
    if not os.path.exists(path):
        return None
    with open(path) as f:
        return [tuple(map(int, ln.split())) for ln in f if not ln.startswith("#")]


def ref_counts():
    """(K, SHIFT) -> sieve survivors counted in the reference's own search
    (tests/golden/ref_counts.json)."""
    path = os.path.join(GOLDEN, "ref_counts.json")
    if not os.path.exists(path):
        return {}
    with open(path) as f:
        return {(e["K"], e["shift"]): e["survivors"] for e in json.load(f)}


def host_hash(A, reports, start=0):
    """result_hash after the library's host ReportSolution of the reports."""
    r = A.Reporter(start)
    r.report_all(reports)
    return r.hash.value


def item_parity(A, items, got_reports, got_hashes):
    """Items whose every searchable K has a recorded reference fixture: the
    device reports (in order) and result_hash must equal the reference's
    reports and their ReportSolution hash."""
    checked, bad, ks = 0, [], 0
    for (iid, a, b, sh), reps, h in zip(items, got_reports, got_hashes):
        exp = []
        for K in range(a, b + 1):
            if will_search(K):
                f = ref_fixture(K, sh)
                if f is None:
                    exp = None
                    break
                exp += f
        if exp is None:
            continue
        checked += 1
        ks += sum(will_search(K) for K in range(a, b + 1))
        if [tuple(r[:3]) for r in reps] != exp or h != host_hash(A, exp):
            bad.append(iid)
    # no item checked is no parity claim: ok needs at least one checked item
    return {"items_checked_vs_reference": checked, "k_checked": ks, "items": len(items),
            "all_items_checked": checked == len(items), "mismatched": bad,
            "ok": checked > 0 and not bad}


def parity_check(seen, kmin):
    """Timed-run reports of every K that has a recorded reference raw-report
    fixture (tests/golden/ref_raw/shift0/<K>.txt, the reference's own
    Search_avx2 output) must equal it exactly, in order."""
    checked, bad = 0, []
    for K in sorted(seen):
        ref = ref_fixture(K, SHIFT)
        if ref is None:
            continue
        checked += 1
        if seen[K] != ref:
            bad.append(K)
    return {"k_checked_vs_reference": checked, "k_with_reports": len(seen),
            "mismatched": bad, "ok": checked > 0 and not bad}


# ---- reference arm ---------------------------------------------------------------
def run_reference(args, rank, world):
    if rank != 0:
        return
    ks = [k for k in range(KMIN_SEEDED, KMIN_SEEDED + RANGE_K) if will_search(k)]
    ticks = 2
    vals = []
    for i in range(args.warmup + args.steps):
        cb = cpu_baseline_value(ks[(i * 8) % len(ks):] + ks, ticks)
        if i >= args.warmup:
            vals.append(cb)
    kps = sum(v["value"] for v in vals) / len(vals)
    secs = sum(v["seconds"] for v in vals)
    line = {
        "impl": "reference", "metric": "K/s, 10-shift search", "value": kps, "unit": "K/s",
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1000 * secs / len(vals), "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "int64", "data": "synthetic (seeded K range)",
        "config": {"workload": f"64 consecutive K from KMIN={KMIN_SEEDED}, SHIFT=0 "
                               "(bounded CPU samples of the same K)",
                   "kmin": KMIN_SEEDED, "k_count": RANGE_K, "shift": SHIFT},
        "cpu_baseline": {"value": kps, "unit": "K/s", "cores": vals[0]["cores"],
                         "kind": vals[0]["kind"], "sample": vals[0]["sample"]},
        "e2e": {"value": kps, "unit": "K/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


# ---- secondary keys of the default line -------------------------------------------
IMAD_PER_MULMOD = 9    # 32 x 32 products of one 64-bit Montgomery square:
                       # 3 for x*x, 3 for m = lo*n', 3 for the high half of m*N
ALG_BYTES_PER_K = N59_PER_K * 10 * ROW_BYTES_PER_CELL


def _mixed_items(rng, n, max_len, shifts=(0, 640, 1280)):
    import math
    items = []
    for i in range(n):
        length = int(math.exp(rng.uniform(0, math.log(max_len)))) if max_len > 1 else 1
        length = max(1, min(max_len, length))
        k0 = int(rng.integers(1_000_000, 50_000_000 - max_len))
        items.append((i, k0, k0 + length - 1, int(rng.choice(shifts))))
    return items


# ---- the seeded workloads of the secondary bench keys ------------------------------
# Each is a stated prefix of its full-size configuration, sized so that the
# whole default run stays within a few minutes; tests/golden/make_golden.py
# records the reference's own raw reports and survivor counts for every
# (K, SHIFT) they contain.
BATCHED_FULL_ITEMS = 4096      # the full batched configuration: 4096 items ...
BATCHED_MAX_LEN = 64           # ... of log-uniform length 1..64 K
BATCHED_ITEMS = 5              # bench prefix: the first 5 items (20 searchable K)
SERVE_UNITS, SERVE_MAX_K = 32, 8
SIEVE_PAIR_KMIN = 27872096     # default_rng(31).integers(1e6, 5e7 - 1024): 1024 K at SHIFT 640
SIEVE_PAIR_FULL, SIEVE_PAIR_K, SIEVE_PAIR_PINNED, SIEVE_PAIR_SHIFT = 1024, 64, 56, 640


def batched_items(n=BATCHED_ITEMS):
    """The first n of the 4096 seeded mixed work items (seed 44)."""
    import numpy as np
    return _mixed_items(np.random.default_rng(44), BATCHED_FULL_ITEMS, BATCHED_MAX_LEN)[:n]


def serve_units(n=SERVE_UNITS, max_k=SERVE_MAX_K):
    """Seeded serving units (seed 55): log-uniform 1..max_k K, mixed SHIFT."""
    import numpy as np
    return _mixed_items(np.random.default_rng(55), n, max_k)


def sieve_pair_ks(n=SIEVE_PAIR_K):
    """The first n K of the 1024 consecutive K of the sieve roofline pair."""
    return list(range(SIEVE_PAIR_KMIN, SIEVE_PAIR_KMIN + n))


def fixture_pairs():
    """Every (K, SHIFT) of the secondary workloads whose reference results are
    recorded: the 56 searchable K of the sieve pair's first 64, then the batched
    and serving items' searchable K."""
    out = [(k, SIEVE_PAIR_SHIFT) for k in sieve_pair_ks() if will_search(k)][:SIEVE_PAIR_PINNED]
    for _, a, b, sh in batched_items() + serve_units():
        out += [(k, sh) for k in range(a, b + 1) if will_search(k)]
    seen, uniq = set(), []
    for p in out:
        if p not in seen:
            seen.add(p)
            uniq.append(p)
    return uniq


def _spread(xs):
    return (max(xs) - min(xs)) / statistics.mean(xs) if len(xs) > 1 else 0.0


def measure_batched(ctx, A, reps=3, n_items=BATCHED_ITEMS):
    """The batched persistent form against the plain one-K-per-launch-sequence
    form on the same seeded mixed items (the first BATCHED_ITEMS of the 4096):
    each form `reps` times, end to end through the C ABI with host buffers
    (batched: ap26_search_batch + ap26_report_batch for the SOL lines; plain:
    ap26_search_k_sol per K, the reference's per-K loop with ReportSolution on
    the device) and on the device."""
    items = batched_items(n_items)
    nk = sum(will_search(K) for _, a, b, _ in items for K in range(a, b + 1))
    bw, bd, pw, pd = [], [], [], []
    per = res = None
    plain_hash = {}
    for _ in range(reps):
        t0 = time.perf_counter()
        per, res, st = ctx.search_batch(items)
        for reps_i in per:
            if reps_i:
                rc, _, _ = ctx.report_batch(reps_i)
                assert rc == A.OK, rc
        bw.append(time.perf_counter() - t0)
        bd.append(st.device_ms / 1e3)
        t0 = time.perf_counter()
        dev = 0.0
        for iid, a, b, sh in items:
            h = 0
            for K in range(a, b + 1):
                if will_search(K):
                    h, _, s2 = ctx.search_k_sol(K, sh, result_hash=h)
                    dev += s2.device_ms
            plain_hash[iid] = h
        pw.append(time.perf_counter() - t0)
        pd.append(dev / 1e3)
    par = item_parity(A, items, per, [r.result_hash for r in res])
    par["plain_hash_equals_batched"] = all(plain_hash[r.id] == r.result_hash for r in res)
    par["ok"] = par["ok"] and par["plain_hash_equals_batched"]
    b_e2e = [nk / t for t in bw]
    p_e2e = [nk / t for t in pw]
    return {
        "workload": f"the first {len(items)} of {BATCHED_FULL_ITEMS} seeded items (seed 44): "
                    f"log-uniform 1..{BATCHED_MAX_LEN} K, SHIFT in {{0,640,1280}}",
        "items": len(items), "searched_k": nk, "repeats": reps,
        "batched": {"e2e_kps": b_e2e, "device_kps": [nk / t for t in bd],
                    "form": "ap26_search_batch (one CUDA-graph launch per batch) + "
                            "ap26_report_batch"},
        "plain": {"e2e_kps": p_e2e, "device_kps": [nk / t for t in pd],
                  "form": "ap26_search_k_sol per K (search + ReportSolution on the device)"},
        "e2e_ratio": statistics.mean(b_e2e) / statistics.mean(p_e2e),
        "device_ratio": statistics.mean(pd) / statistics.mean(bd),
        "e2e_spread": {"batched": _spread(b_e2e), "plain": _spread(p_e2e)},
        "parity": par,
    }


def measure_serve(ctx, A, capacity_kps, roofline_kps, n_units=SERVE_UNITS, max_k=SERVE_MAX_K):
    """Continuous batching: Poisson arrivals of the seeded units at 0.8x the
    measured batched capacity; units admitted by device memory, two slices
    queued on the device, each unit's hash and checkpoint kept there."""
    import numpy as np
    units = serve_units(n_units, max_k)
    ks_of = {u[0]: sum(will_search(K) for K in range(u[1], u[2] + 1)) for u in units}
    mean_k = statistics.mean(ks_of.values())
    rate = 0.8 * capacity_kps / mean_k                    # units per second
    arrivals = np.cumsum(np.random.default_rng(56).exponential(1.0 / rate, len(units)))
    lat, res_of = {}, {}
    t0 = time.perf_counter()
    nxt, done, total_k = 0, 0, 0
    limit_s = 60.0 + 4.0 * sum(ks_of.values()) / max(capacity_kps, 0.1)
    last = 0.0
    while done < len(units):
        if time.perf_counter() - t0 - last > 10.0:
            last = time.perf_counter() - t0
            progress(f"serving: {nxt} of {len(units)} units submitted, {done} returned")
        if time.perf_counter() - t0 > limit_s:
            raise RuntimeError(f"serving did not finish in {limit_s:.0f} s: {done} of "
                               f"{len(units)} units returned, {nxt} submitted")
        now = time.perf_counter() - t0
        while nxt < len(units) and arrivals[nxt] <= now:
            rc = ctx.serve_submit(*units[nxt])
            assert rc == A.OK, rc
            nxt += 1
        active = ctx.serve_step()
        while True:
            r = ctx.serve_poll()
            if r is None:
                break
            res, aps = r
            lat[res.id] = (time.perf_counter() - t0) - arrivals[res.id]
            res_of[res.id] = (res, aps)
            total_k += res.ks_searched
            done += 1
        now = time.perf_counter() - t0
        until = arrivals[nxt] - now if nxt < len(units) else 1.0
        if active == 0:
            if nxt < len(units):
                time.sleep(max(0.0, until))
        else:
            ctx.serve_wait(max(0.0005, min(until, 1.0)))
    span = time.perf_counter() - t0
    ls = sorted(lat.values())
    # latency at the roofline: the unit's K alone at the sieve's shared-memory roofline
    frac = sorted(ks_of[i] / roofline_kps / lat[i] for i in lat if ks_of[i])
    par = item_parity(A, units, [res_of[u[0]][1] for u in units],
                      [res_of[u[0]][0].result_hash for u in units])
    return {
        "workload": f"{len(units)} seeded units (seed 55): log-uniform 1..{max_k} K, "
                    "SHIFT in {0,640,1280}, Poisson arrivals (seed 56) at 0.8x capacity",
        "max_k": max_k,
        "units": len(units), "searched_k": total_k, "capacity_kps": capacity_kps,
        "arrival_rate_units_per_s": rate,
        "p50_s": float(np.percentile(ls, 50)), "p99_s": float(np.percentile(ls, 99)),
        "max_s": ls[-1], "sustained_kps": total_k / span,
        "sustained_frac_of_roofline": total_k / span / roofline_kps,
        "latency_frac_of_roofline": {"p50": float(np.percentile(frac, 50)),
                                     "p1": float(np.percentile(frac, 1)),
                                     "note": "per unit with a searchable K: its K at the "
                                             "sieve roofline alone / measured completion "
                                             "latency"},
        "parity": par,
    }


def measure_sieve_pair(ctx, A, smem_gbs, n=SIEVE_PAIR_K):
    """Sieve alone: survivor counts of the first SIEVE_PAIR_K of the 1024
    consecutive K at SHIFT 640; counts of the pinned prefix must equal the
    reference's own."""
    import numpy as np
    ks = sieve_pair_ks(n)
    # calls of at most 64 K each, so that no single device wait outlasts
    # the context's wait limit at the full 1024 K
    counts, dev_ms, sieve_ms, cells = [], 0.0, 0.0, 0
    for i in range(0, len(ks), 64):
        c, st = ctx.sieve_count(ks[i:i + 64], SIEVE_PAIR_SHIFT)
        counts.append(c)
        dev_ms += st.device_ms
        sieve_ms += st.sieve_ms
        cells += st.sieve_cells
    counts = np.concatenate(counts)
    achieved = cells * ROW_BYTES_PER_CELL / (sieve_ms / 1e3) / 1e9
    pinned = ref_counts()
    chk = [(k, int(c), pinned[(k, SIEVE_PAIR_SHIFT)]) for k, c in zip(ks, counts)
           if (k, SIEVE_PAIR_SHIFT) in pinned]
    return {
        "workload": f"sieve survivor counts of the first {len(ks)} of {SIEVE_PAIR_FULL} "
                    f"consecutive K from {SIEVE_PAIR_KMIN}, SHIFT={SIEVE_PAIR_SHIFT}",
        "k_count": len(ks), "kps": len(ks) / (dev_ms / 1e3),
        "raw_kps": len(ks) / (dev_ms / 1e3),
        "roofline": {"bound": "smem", "achieved": achieved, "peak": smem_gbs, "unit": "GB/s",
                     "frac": achieved / smem_gbs, "kernel": "class_sieve_kernel"},
        "survivors_total": int(counts.sum()),
        "parity": {"k_checked_vs_reference": len(chk),
                   "mismatched": [k for k, c, r in chk if c != r],
                   "ok": bool(chk) and all(c == r for _, c, r in chk)},
    }


def measure_sprp(ctx, A, int_tops, log2=24):
    """Strong-PRP microbenchmark: 2^log2 odd values in [2^40, 2^63), half
    probable primes and half composites as the device test classifies them;
    verdict parity against the reference's own strong_prp verdicts
    (tests/golden/sprp_vectors.txt)."""
    import numpy as np
    rng = np.random.default_rng(32)
    n = 1 << log2
    want = n // 2
    primes, comps = [], []
    have_p = have_c = 0
    while have_p < want or have_c < want:
        cand = rng.integers(1 << 40, (1 << 63) - 1, 1 << 24, dtype=np.uint64) | np.uint64(1)
        v, _ = ctx.sprp_batch(cand)
        p, c = cand[v == 1], cand[v == 0]
        primes.append(p[:max(0, want - have_p)])
        comps.append(c[:max(0, want - have_c)])
        have_p += len(primes[-1])
        have_c += len(comps[-1])
    vals = np.concatenate(primes + comps)
    rng.shuffle(vals)
    ctx.sprp_batch(vals[:1 << 16])
    v, st = ctx.sprp_batch(vals)
    mm_s = st.late_items / (st.device_ms / 1e3)            # modular squarings per second
    peak = int_tops * 1e12 / IMAD_PER_MULMOD
    vec = []
    with open(os.path.join(GOLDEN, "sprp_vectors.txt")) as f:
        for ln in f:
            if not ln.startswith("#"):
                N, a, ver = map(int, ln.split())
                if a == 2 and N % 2 == 1 and N < (1 << 63):
                    vec.append((N, ver))
    vv, _ = ctx.sprp_batch(np.array([x for x, _ in vec], dtype=np.uint64))
    bad = [N for (N, ver), got in zip(vec, vv) if int(got) != ver]
    return {
        "workload": f"{n} odd values in [2^40, 2^63), half primes by the device test (seed 32)",
        "values": n, "tests_per_s": n / (st.device_ms / 1e3), "mulmod_per_s": mm_s,
        "roofline": {"bound": "int", "achieved": mm_s, "peak": peak, "unit": "mulmod/s",
                     "frac": mm_s / peak, "kernel": "sprp_batch_kernel",
                     "note": f"peak = measured IMAD rate / {IMAD_PER_MULMOD} multiply-adds "
                             "per 64-bit Montgomery product; unit = modular squaring"},
        "primes": int(v.sum()),
        "parity": {"reference_vectors": len(vec), "mismatched": len(bad), "ok": not bad},
    }


# ---- our arm ---------------------------------------------------------------------
# DRAM bytes per sieve cell: dram__bytes_read.sum + dram__bytes_write.sum of the
# one class sieve launch of a K (4.808e10 cells) in an ncu capture, 637.3 MB read
# + 623.3 MB written.  Nearly all of it is the candidate ring: 38.8 M survivors
# x 16 B written, and the L2's fills of the partly written sectors read back; it
# grows with the survivors, so with the cells, and scales to any launch.
SIEVE_DRAM_BYTES_PER_CELL = (637.27e6 + 623.30e6) / (N59_PER_K * 10)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=8)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-plain", action="store_true")
    ap.add_argument("--no-autotune", action="store_true")
    ap.add_argument("--no-secondary", action="store_true",
                    help="skip the batched / serve / sieve_pair / sprp keys")
    # sizes of the secondary keys (defaults: the stated prefixes; the full
    # configurations are 4096 items, units of 1..256 K and 1024 K)
    ap.add_argument("--batched-items", type=int, default=BATCHED_ITEMS)
    ap.add_argument("--serve-units", type=int, default=SERVE_UNITS)
    ap.add_argument("--serve-max-k", type=int, default=SERVE_MAX_K)
    ap.add_argument("--sieve-k", type=int, default=SIEVE_PAIR_K)
    ap.add_argument("--prp-log2", type=int, default=24)
    args = ap.parse_args()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        return run_reference(args, rank, world)

    import torch
    import torch.distributed as dist
    torch.cuda.set_device(local)
    if world > 1:
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=600),
                                device_id=torch.device("cuda", local))
    import ap26_b200 as A
    from ap26_b200 import replicas

    ctx = A.Context(local, profile=1, wait_timeout_s=300.0)
    progress("context created")
    tuned = None
    if not args.no_autotune:
        tuned = ctx.autotune(KMIN_SEEDED + 64 * rank if will_search(KMIN_SEEDED + 64 * rank)
                             else KMIN_SEEDED)
    progress(f"autotuned: {tuned}")
    smem_gbs, int_tops = ctx.probe_peaks()
    roofline_kps = smem_gbs * 1e9 / ALG_BYTES_PER_K
    kmin, _ = replicas.rank_range(KMIN_SEEDED, RANGE_K, rank)
    nsteps_range = RANGE_K // STEP_K

    def step_items(i):
        k0 = kmin + STEP_K * (i % nsteps_range)
        return [(i, k0, k0 + STEP_K - 1, SHIFT)]

    seen = {}
    item_hash = {}

    def run_step(i, sol_lines):
        # the public API a host uses for a workunit: ap26_search_batch (raw
        # reports and the item's result_hash, computed on the device), then
        # ap26_report_batch for the SOL lines (device-side ReportSolution)
        t0 = time.perf_counter()
        its = step_items(i)
        per, res, st = ctx.search_batch(its)
        for reps in per:
            if reps:
                rc, fin, _ = ctx.report_batch(reps)
                assert rc == A.OK, rc
                st.launches += 1          # its report_kernel
                sol_lines += [(ln, r[1], fi) for r, f in zip(reps, fin) for ln, fi in f.sols()]
        wall = time.perf_counter() - t0
        local = {}
        for reps in per:
            for k, K, first, _n in reps:
                local.setdefault(K, []).append((k, K, first))
        seen.update(local)
        item_hash[its[0][1]] = (res[0].result_hash, its[0][1], its[0][2])
        nk = sum(r.ks_searched for r in res)
        naps = sum(r.n_aps for r in res)
        h2d = KJOB_BYTES * nk + DEVSTATE_BYTES + APREC_BYTES * naps
        d2h = DEVSTATE_BYTES + (COUNT_BYTES + 10 * COUNT_BYTES) * nk + \
            (APREC_BYTES + FINAL_BYTES) * naps
        return st, wall, nk, h2d, d2h

    for i in range(args.warmup):
        run_step(i, [])
    seen.clear()
    progress("warm-up steps done")

    def barrier():
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()

    rep = []
    tot = {"dev_ms": 0.0, "sieve_ms": 0.0, "cells": 0, "launches": 0, "ks": 0, "h2d": 0,
           "d2h": 0, "kernels": 0, "cand": 0}
    barrier()
    with ClockSampler(local) as clk:
        ev0 = torch.cuda.Event(enable_timing=True)
        ev1 = torch.cuda.Event(enable_timing=True)
        t0 = time.perf_counter()
        ev0.record()
        for i in range(args.steps):
            st, wall, nk, h2d, d2h = run_step(i, rep)
            tot["dev_ms"] += st.device_ms
            tot["sieve_ms"] += st.sieve_ms
            tot["cells"] += st.sieve_cells
            tot["launches"] += st.sieve_launches
            tot["kernels"] += st.launches
            tot["ks"] += nk
            tot["h2d"] += h2d
            tot["d2h"] += d2h
            tot["cand"] += st.candidates
        ev1.record()
        barrier()
        wall = time.perf_counter() - t0
    ev_ms = ev0.elapsed_time(ev1)
    raw_k = STEP_K * args.steps
    progress(f"timed steps done: {tot['ks']} K in {wall:.1f} s")

    vec = torch.tensor([tot["dev_ms"], wall, ev_ms, tot["sieve_ms"]], dtype=torch.float64,
                       device="cuda")
    ks_all = torch.tensor([tot["ks"], raw_k], dtype=torch.float64, device="cuda")
    if world > 1:
        dist.all_reduce(vec, op=dist.ReduceOp.MAX)
        dist.all_reduce(ks_all, op=dist.ReduceOp.SUM)
    dev_ms, wall_max, ev_max, _ = vec.tolist()
    ks_total, raw_total = ks_all.tolist()

    # plain one-K-per-launch-sequence form over the rank's 64-K range once
    plain = None
    if not args.no_plain:
        barrier()
        pms, pk, t0 = 0.0, 0, time.perf_counter()
        for K in range(kmin, kmin + RANGE_K):
            if will_search(K):
                _, _, st = ctx.search_k_sol(K, SHIFT)
                pms += st.device_ms
                pk += 1
        pwall = time.perf_counter() - t0
        pv = torch.tensor([pms, pwall], dtype=torch.float64, device="cuda")
        pkt = torch.tensor([pk], dtype=torch.float64, device="cuda")
        if world > 1:
            dist.all_reduce(pv, op=dist.ReduceOp.MAX)
            dist.all_reduce(pkt, op=dist.ReduceOp.SUM)
        progress("plain form done")
        plain = {"value": pkt.item() / (pv[0].item() / 1000.0), "unit": "K/s",
                 "e2e": pkt.item() / pv[1].item(), "searched_k": int(pkt.item()),
                 "form": "ap26_search_k_sol per K over the 64-K range (search + ReportSolution "
                         "on the device), device time and wall clock"}

    secondary = {}
    if rank == 0 and world == 1 and not args.no_secondary:
        def keep(name, fn):
            # a failing secondary key is reported in the line, not fatal
            try:
                secondary[name] = fn()
            except Exception as e:          # noqa: BLE001
                secondary[name] = {"error": f"{type(e).__name__}: {e}"}
            progress(f"{name} done")

        with ClockSampler(local) as clk2:
            keep("batched", lambda: measure_batched(ctx, A, n_items=args.batched_items))
            cap = (statistics.mean(secondary["batched"]["batched"]["device_kps"])
                   if "error" not in secondary["batched"] else
                   ks_total / (dev_ms / 1000.0))
            keep("serve", lambda: measure_serve(ctx, A, cap, roofline_kps, args.serve_units,
                                                args.serve_max_k))
            keep("sieve_pair", lambda: measure_sieve_pair(ctx, A, smem_gbs, args.sieve_k))
            keep("sprp", lambda: measure_sprp(ctx, A, int_tops, args.prp_log2))
        secondary["clocks"] = clk2.summary()

    if rank == 0:
        sieve_launch_ms = tot["sieve_ms"] / max(1, tot["launches"])
        cells_per_launch = tot["cells"] / max(1, tot["launches"])
        alg_bytes = cells_per_launch * ROW_BYTES_PER_CELL
        achieved = alg_bytes / (sieve_launch_ms / 1000.0) / 1e9
        hash_par = {"items": 0, "ok": True}
        for h, a, b in item_hash.values():
            exp = []
            for K in range(a, b + 1):
                if will_search(K):
                    f = ref_fixture(K, SHIFT)
                    exp = None if f is None or exp is None else exp + f
            if exp is not None:
                hash_par["items"] += 1
                hash_par["ok"] = hash_par["ok"] and h == host_hash(A, exp)
        line = {
            "metric": "K/s, 10-shift search", "value": ks_total / (dev_ms / 1000.0),
            "unit": "K/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": dev_ms / args.steps, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "int64", "data": "synthetic (seeded K range)",
            "config": {"workload": f"64 consecutive K from KMIN={KMIN_SEEDED} (seed 26) per "
                                   f"rank, SHIFT=0, steps of {STEP_K} K via the batched "
                                   "persistent pipeline",
                       "kmin": KMIN_SEEDED, "k_per_rank": RANGE_K, "shift": SHIFT,
                       "searched_k": int(ks_total), "raw_k": int(raw_total),
                       "parallelism": f"replicas x{world} (disjoint K ranges)",
                       "l2": "row tables in shared memory, a 15 MB plan per K built on the "
                             "device; no HBM-resident inputs to flush",
                       "autotuned": tuned},
            "raw_kps": raw_total / (dev_ms / 1000.0),
            "e2e": {"value": ks_total / wall_max, "unit": "K/s",
                    "raw_kps": raw_total / wall_max,
                    "h2d_bytes_per_step": tot["h2d"] // args.steps,
                    "d2h_bytes_per_step": tot["d2h"] // args.steps,
                    "includes": "C-ABI calls (ap26_search_batch + ap26_report_batch), job "
                                "H2D, report/result D2H, device-side ReportSolution and hash"},
            "roofline": {"bound": "smem", "achieved": achieved, "peak": smem_gbs,
                         "unit": "GB/s", "frac": achieved / smem_gbs,
                         "traffic": cells_per_launch * SIEVE_DRAM_BYTES_PER_CELL,
                         "traffic_unit": "DRAM bytes per launch",
                         "kernel": "class_sieve_kernel",
                         "note": "algorithmic bytes = cells x 46.3 B of the 20 dense moduli's rows; peak = "
                                 "measured conflict-free LDS.128 bandwidth of this GPU "
                                 "(ap26_probe_peaks); HBM and tensor cores are not on the path",
                         "launch_ms": sieve_launch_ms, "int_tops_peak": int_tops,
                         "roofline_kps": roofline_kps},
            "gpu_launches": tot["kernels"],
            "torch_event_ms": ev_max,
            "clocks": clk.summary(),
        }
        if plain:
            line["plain"] = plain
        line["parity"] = parity_check(seen, kmin)
        line["parity"]["item_hash"] = hash_par
        line["parity"]["ok"] = line["parity"]["ok"] and hash_par["ok"]
        line.update(secondary)
        if world == 1 and not args.no_cpu_baseline:
            ks = [k for k in range(KMIN_SEEDED, KMIN_SEEDED + RANGE_K) if will_search(k)]
            cb = cpu_baseline_value(ks, 6)
            progress("cpu baseline done")
            cb["extrapolated"] = ("per-pass time per lattice value from a bounded sample, "
                                  "times the 10840 lattice values of a pass, plus set-up; "
                                  "checked once against a whole K (591 s estimated, 614 s "
                                  "measured on one core)")
            line["cpu_baseline"] = cb
            comp = avx512_companion(ks[0])
            if comp:
                line["cpu_avx512"] = comp
        print(json.dumps(line), flush=True)
    ctx.close()
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
