"""Inputs that no search meets, and that cost as little as others.

Times are the least of several calls, compared with those of an ordinary input
of the same size on the same device.
"""
import time

import numpy as np
import pytest

import ap26_b200 as A

pytestmark = pytest.mark.gpu

K = 366384


def _least(call, n=15):
    times = []
    for _ in range(n):
        t = time.perf_counter()
        call()
        times.append(time.perf_counter() - t)
    return min(times)


@pytest.mark.parametrize("n", [20_011, 1_000_000])
def test_walks_outside_the_domain_cost_no_more_than_others(ctx, n):
    """Each such walk raises the call's error: once a warp, not once a walk over
    the bus.  They end at their first term, before any test."""
    cand, _ = ctx.sieve_range(K, 0, 0, 4_000_000)
    good = np.resize(cand, n)
    bad = -good
    k, first = np.empty(n, np.int32), np.empty(n, np.int64)

    def walk(c, rc):                             # the call alone, without the binding's exception
        assert A.lib.ap26_chain_batch(ctx.h, K, A._ptr(c), n, A._ptr(k), A._ptr(first), None) == rc
    assert _least(lambda: walk(bad, A.E_DOMAIN)) < 3 * _least(lambda: walk(good, A.OK))


def test_one_walk_of_many_outside_the_domain_is_an_error(ctx):
    cand, _ = ctx.sieve_range(K, 0, 0, 4_000_000)
    for n in (1, 33, 20_011, 1_000_000):
        c = np.resize(cand, n)
        ctx.chain_batch(K, c)
        for at in {0, n // 2, n - 1}:
            bad = c.copy()
            bad[at] = -1 - c[at]
            with pytest.raises(A.AP26Error) as e:
                ctx.chain_batch(K, bad)
            assert e.value.code == A.E_DOMAIN
        ctx.chain_batch(K, c)


def _report(ctx, rows):
    arr = np.array(rows, A._AP)
    fin = (A.Final * len(arr))()
    rc = A.lib.ap26_report_batch(ctx.h, A._ptr(arr), len(arr), fin, None, None)
    return rc, [f.status for f in fin]


def test_a_long_report_of_composites_costs_no_more_than_a_real_one(ctx):
    """The most terms a report can have, none of them a probable prime: one base
    shows it, the other eight have nothing to add."""
    real = [(25, 366384, 6171054912832631, 0)]       # the golden solution of this K
    none = [(128, K, (1 << 57) + 9, 0)]
    assert _report(ctx, real)[0] == A.OK
    assert _report(ctx, none)[0] == A.E_INVALID
    assert _least(lambda: _report(ctx, none), 40) < 2 * _least(lambda: _report(ctx, real), 40)


@pytest.mark.parametrize("k", [31, 32, 33, 95, 96, 97, 127, 128])
def test_long_reports_equal_the_host_restatement(ctx, k):
    """Statuses where the terms are tested to base 2 first (above 32) and where they
    are not: an AP that goes on past its 25 primes, composites, an even start, and
    terms that leave the domain of 2^62 within the report."""
    rows = [(k, 366384, 6171054912832631, 0), (k, K, (1 << 57) + 9, 0), (k, K, 1 << 57, 0),
            (k, 400_000_000 - 1, (1 << 62) - 12 * 399_999_999 * A.PRIM23 + 1, 0),
            (k, 1, 1_000_003, 0)]
    want = []
    for r in rows:
        try:
            A.Reporter().report(*r[:3])
            want.append(A.OK)
        except A.AP26Error as e:
            want.append(e.code)
    assert _report(ctx, rows)[1] == want
    assert A.OK not in want
