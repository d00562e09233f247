"""The work of this framework that is timed: its calls, from the smallest to the largest.

A case names one public call and its sizes.  listed() gives the fixed ones,
draw() more from the same ranges; prepare() makes a case's inputs, run() is
one pass through the call, work() what the pass cannot do without, exact()
its answer without this library.

Two kinds of call.  The whole searches (search_k, search_batch, the serving
loop, sieve_count) are what the library is for: a workunit is a range of K,
each K costs the same 4.8e9 lattice values, and the host sends and receives
almost nothing.  The kernel-level calls (sieve_range, sprp_batch, sprp_bases,
chain_batch, report_batch) take host arrays, from a handful of values to
2^24, and their small sizes are bound by latency.
"""
import numpy as np

import ap26_b200 as A

PRIM23 = 223092870
STARTS_PER_N43 = 12673          # n53 starts of one n43 value
CELLS_PER_START = 35 * 10       # 35 n59 values of 10 shift words each
CONSULTS_PER_CELL = 16.62       # mean table lookups per word, ascending primes, stop at zero
SURVIVORS_PER_START = 0.283     # after the sieve and the 7..23 filter
MOST_SURVIVORS_PER_START = 2    # of the densest K (1.5), rounded up
REPORTS = 150                   # raw reports of an ordinary K
MOST_REPORTS_PER_K = 1024       # of the densest K (734), rounded up
BASES = np.array([2, 3, 5, 7, 11, 13, 17, 19, 23], np.uint32)

_CTX = None


def _context():
    """The device context: a program makes one and keeps it."""
    global _CTX
    if _CTX is None:
        _CTX = A.Context(0)
    return _CTX


def listed():
    return [
        # one n43 value's starts: the smallest slice anyone checks
        {"name": "sieve-one-n43", "call": "sieve_range", "starts": STARTS_PER_N43, "shift": 0},
        # a ragged slice of the middle of the lattice, as a spot check of a K
        {"name": "sieve-ragged", "call": "sieve_range", "starts": 600011, "shift": 640},
        # a few values to test, as from an interactive program
        {"name": "sprp-few", "call": "sprp_batch", "count": 61},
        # a list of candidates to test
        {"name": "sprp-1m", "call": "sprp_batch", "count": 1 << 20},
        # the roofline set of the strong-PRP test
        {"name": "sprp-16m", "call": "sprp_batch", "count": 1 << 24},
        # validation of some thousand terms with the nine bases
        {"name": "sprp-bases", "call": "sprp_bases", "count": 50021},
        # chain walks of the survivors of a slice
        {"name": "chain-slice", "call": "chain_batch", "count": 20011, "shift": 0},
        # ReportSolution of one K's raw reports
        {"name": "report-k", "call": "report_batch", "copies": 1, "shift": 0},
        # survivor counts (no chain walk) of K at another SHIFT
        {"name": "count-2k", "call": "sieve_count", "ks": 2, "shift": 640},
        # the plain command: one K searched
        {"name": "search-k", "call": "search_k", "shift": 0},
        # a batch of items of different lengths and SHIFT in one call
        {"name": "batch-4k", "call": "search_batch", "lengths": "2,1,1", "shifts": "0,640,1280"},
        # units served together until all are done
        {"name": "serve-4k", "call": "serve", "lengths": "1,2,1", "shifts": "1280,0,640"},
    ]


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi], odd more often than not."""
    n = int(round(lo * (hi / lo) ** rng.random()))
    return min(hi, n | 1) if rng.random() < 0.7 else n


def draw(rng):
    call = rng.choice(["sieve_range", "sieve_range", "sprp_batch", "sprp_batch", "sprp_bases",
                       "chain_batch", "report_batch", "sieve_count", "search_k", "search_batch",
                       "serve"])
    shift = 64 * rng.randrange(1, 240)
    if call == "sieve_range":
        return {"call": call, "starts": _log(rng, 200, 1000000), "shift": shift}
    if call in ("sprp_batch", "sprp_bases"):
        return {"call": call, "count": _log(rng, 16, 1 << (23 if call == "sprp_batch" else 18))}
    if call == "chain_batch":
        return {"call": call, "count": _log(rng, 16, 100000), "shift": shift}
    if call == "report_batch":
        return {"call": call, "copies": _log(rng, 1, 60), "shift": shift}
    if call == "sieve_count":
        return {"call": call, "ks": rng.randrange(1, 4), "shift": shift}
    if call == "search_k":
        return {"call": call, "shift": shift}
    n = rng.randrange(2, 4)
    lengths, left = [], 4
    for i in range(n):
        lengths.append(rng.randrange(1, left - (n - 1 - i) + 1))
        left -= lengths[-1]
    shifts = [640 * rng.randrange(25) for _ in range(n)]
    return {"call": call, "lengths": ",".join(map(str, lengths)),
            "shifts": ",".join(map(str, shifts))}


# ---- inputs -------------------------------------------------------------------
def _searchable_k(rng):
    while True:
        k = int(rng.integers(1_000_000, 50_000_000))
        if A.will_search(k):
            return k


def _item_range(rng, length):
    """[kmin, kmax] with `length` searchable K, starting at a seeded one."""
    kmin = k = _searchable_k(rng)
    left = length - 1
    while left:
        k += 1
        left -= A.will_search(k)
    return kmin, k


def _items(case, rng):
    lengths = [int(x) for x in case["lengths"].split(",")]
    shifts = [int(x) for x in case["shifts"].split(",")]
    return [(i + 1,) + _item_range(rng, n) + (s,) for i, (n, s) in enumerate(zip(lengths, shifts))]


def _test_values(rng, count):
    """Values to test for primality: in [2^40, 2^63), log-uniform, without a
    factor up to 23, as the 7..23 filter leaves them."""
    q = np.exp2(rng.uniform(40.0, 63.0, count)).astype(np.uint64) // np.uint64(PRIM23)
    q = np.clip(q, (1 << 40) // PRIM23 + 1, (1 << 63) // PRIM23 - 2).astype(np.uint64)
    pool = rng.integers(0, PRIM23, max(4096, min(count, 1 << 18) * 8), dtype=np.int64)
    ok = pool % 2 != 0
    for p in (3, 5, 7, 11, 13, 17, 19, 23):
        ok &= pool % p != 0
    pool = pool[ok].astype(np.uint64)
    return q * np.uint64(PRIM23) + pool[rng.integers(0, len(pool), count)]


def prepare(case, seed):
    rng = np.random.default_rng([seed, len(case["call"])])
    ctx = _context()
    s = {"call": case["call"], "ctx": ctx}
    if case["call"] == "sieve_range":
        q0 = int(rng.integers(0, A.N53_PER_K - case["starts"]))
        s.update(K=_searchable_k(rng), shift=case["shift"], q0=q0, q1=q0 + case["starts"])
    elif case["call"] == "sprp_batch":
        s.update(N=_test_values(rng, case["count"]))
    elif case["call"] == "sprp_bases":
        s.update(N=_test_values(rng, case["count"]), a=BASES[rng.integers(0, 9, case["count"])])
    elif case["call"] == "chain_batch":
        K, count = _searchable_k(rng), case["count"]
        q0 = int(rng.integers(0, A.N53_PER_K // 2))
        n = np.sort(ctx.sieve_range(K, case["shift"], q0, q0 + 4 * count + 12673)[0])
        s.update(K=K, n=rng.permutation(n)[:count].copy())
    elif case["call"] == "report_batch":
        aps, _ = ctx.search_k(_searchable_k(rng), case["shift"])
        aps = (aps * REPORTS)[:REPORTS] * case["copies"]
        s.update(aps=aps)
    elif case["call"] == "sieve_count":
        s.update(Ks=[_searchable_k(rng) for _ in range(case["ks"])], shift=case["shift"])
    elif case["call"] == "search_k":
        s.update(K=_searchable_k(rng), shift=case["shift"])
    else:
        s.update(items=_items(case, rng))
    return s


# ---- one pass -----------------------------------------------------------------
def _reports(aps, ks):
    """The reports in an array with room for any K's, the rest zero."""
    out = np.zeros((MOST_REPORTS_PER_K * ks, 4), np.int64)
    out[:len(aps)] = np.array(aps, np.int64).reshape(-1, 4)
    return out


def _serve(ctx, items):
    for it in items:
        rc = ctx.serve_submit(*it)
        if rc != A.OK:
            raise A.AP26Error(rc, "ap26_serve_submit")
    out = {}
    while True:
        active = ctx.serve_step()
        while True:
            r = ctx.serve_poll()
            if r is None:
                break
            out[r[0].id] = r
        if active == 0:
            return [out[it[0]] for it in items]
        ctx.serve_wait(10.0)


def run(state):
    ctx, call = state["ctx"], state["call"]
    if call == "sieve_range":
        # the call's candidates come in no order: a caller sorts them
        cand, _ = ctx.sieve_range(state["K"], state["shift"], state["q0"], state["q1"])
        out = np.zeros(MOST_SURVIVORS_PER_START * (state["q1"] - state["q0"]), np.int64)
        out[:len(cand)] = np.sort(cand)
        return out, len(cand)
    if call == "sprp_batch":
        return ctx.sprp_batch(state["N"])[0]
    if call == "sprp_bases":
        return ctx.sprp_bases(state["N"], state["a"])[0]
    if call == "chain_batch":
        k, first, _ = ctx.chain_batch(state["K"], state["n"])
        return k, first
    if call == "report_batch":
        rc, fin, h = ctx.report_batch(state["aps"], result_hash=0)
        f = np.ctypeslib.as_array((A.Final * len(fin))(*fin)) if fin else np.zeros(0)
        return rc, h, f["hash_add"], f["status"], f["n_sol"], f["sol_len"], f["sol_first"]
    if call == "sieve_count":
        return ctx.sieve_count(state["Ks"], state["shift"])[0]
    if call == "search_k":
        aps, st = ctx.search_k(state["K"], state["shift"])
        return _reports(aps, 1), st.candidates, len(aps)
    if call == "search_batch":
        per, res, _ = ctx.search_batch(state["items"])
    else:
        got = _serve(ctx, state["items"])
        per, res = [aps for _, aps in got], [r for r, _ in got]
    return [(_reports(aps, r.ks_searched), len(aps), r.result_hash, r.candidates, r.ks_searched)
            for aps, r in zip(per, res)]


# ---- what a pass cannot do without ------------------------------------------------
def _sieve_work(starts):
    # one 64-bit AND per table consult; the survivors are the output
    return {"bytes": 8.0 * SURVIVORS_PER_START * starts,
            "flops": CONSULTS_PER_CELL * CELLS_PER_START * starts}


def _sprp_ops(tests, bits):
    return tests * bits * 12.0      # a Montgomery square: 12 32-bit multiply-adds


def work(case):
    call = case["call"]
    if call == "sieve_range":
        return _sieve_work(case["starts"])
    if call in ("sprp_batch", "sprp_bases"):
        return {"bytes": case["count"] * (9.0 if call == "sprp_batch" else 13.0),
                "flops": _sprp_ops(case["count"], 51)}
    if call == "chain_batch":
        return {"bytes": case["count"] * 20.0, "flops": _sprp_ops(1.4 * case["count"], 57)}
    if call == "report_batch":      # 10.4 terms a report, nine bases
        n = float(REPORTS) * case["copies"]
        return {"bytes": n * 80.0, "flops": _sprp_ops(n * 10.4 * 9, 57)}
    ks = {"sieve_count": case.get("ks"), "search_k": 1}.get(call)
    if ks is None:
        ks = sum(int(x) for x in case["lengths"].split(","))
    w = _sieve_work(float(A.N53_PER_K) * ks)
    if call == "sieve_count":
        return {"bytes": 12.0 * ks, "flops": w["flops"]}
    return {"bytes": 24.0 * REPORTS * ks,
            "flops": w["flops"] + _sprp_ops(1.4 * SURVIVORS_PER_START * A.N53_PER_K * ks, 57)}


# ---- answers without this library --------------------------------------------------
def _sprp(n, a):
    """Strong probable prime to base a, plain integers."""
    if n <= a or n % 2 == 0:
        return False
    t = ((n - 1) & (1 - n)).bit_length() - 1
    x = pow(a, (n - 1) >> t, n)
    if x in (1, n - 1):
        return True
    for _ in range(t - 1):
        x = x * x % n
        if x == n - 1:
            return True
    return False


def exact(case, seed):
    if case["call"] == "sprp_batch" and case["count"] <= 1 << 17:
        return np.array([_sprp(int(n), 2) for n in prepare(case, seed)["N"]], np.uint8)
    if case["call"] == "sprp_bases":
        s = prepare(case, seed)
        return np.array([_sprp(int(n), int(a)) for n, a in zip(s["N"], s["a"])], np.uint8)
    if case["call"] == "chain_batch":
        s = prepare(case, seed)
        S = s["K"] * PRIM23
        ks, firsts = [], []
        for n in map(int, s["n"]):
            k, m = 0, n + 5 * S
            while _sprp(m, 2):
                k, m = k + 1, m + S
            if k >= 10:
                m = n + 4 * S
                while m > 0 and _sprp(m, 2):
                    k, m = k + 1, m - S
            ks.append(k)
            firsts.append(m + S)
        return np.array(ks, np.int32), np.array(firsts, np.int64)
    return None
