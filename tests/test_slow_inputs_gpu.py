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
