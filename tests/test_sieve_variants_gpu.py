"""Every compiled variant of the window sieve over long ranges, and the class
sieve's candidates against the window sieve's.

test_gpu_parity.py checks each variant on a short slice, whose starts are split
over 35 tiles; a whole-K count is the class sieve's whatever the variant.  Here
the variants sieve the whole lattice of a K with a known count in long ranges
(one tile a start, queues that fill and carry over many tiles), and ranges of
each other split.  Everything is integers: equal.
"""
import numpy as np
import pytest

import ap26_b200 as A

pytestmark = pytest.mark.gpu

VARIANTS = A.list_variants()
SLICES = 16


def _lattice(ctx, K, shift):
    step = -(-A.N53_PER_K // SLICES)
    for q0 in range(0, A.N53_PER_K, step):
        yield ctx.sieve_range(K, shift, q0, min(q0 + step, A.N53_PER_K), cap=1 << 25)[0]


@pytest.mark.parametrize("vi", range(len(VARIANTS)))
def test_variant_counts_a_whole_lattice(ctx, vi):
    ctx.set_opts(**VARIANTS[vi])
    try:
        # the reference's known answer (src/opencl/AP26.h:343)
        assert sum(len(c) for c in _lattice(ctx, 366384, 0)) == 38838420
    finally:
        ctx.set_opts(**VARIANTS[0])


@pytest.mark.parametrize("starts", [140_003, 300_001, 1_000_003])   # 7, 5 and 1 parts
def test_variants_give_the_same_candidates(ctx, starts):
    K, shift, q0 = 28686653, 640, 61_234_567                        # 61 * 67 | K
    want = None
    try:
        for v in VARIANTS:
            ctx.set_opts(**v)
            got = np.sort(ctx.sieve_range(K, shift, q0, q0 + starts)[0])
            if want is None:
                want = got
            assert np.array_equal(got, want), v
    finally:
        ctx.set_opts(**VARIANTS[0])


@pytest.mark.parametrize("K,shift", [
    (43241061, 15360),           # an ordinary K: four rows a class
    (42700061, 1280),            # 61 | K: seven
    (28686653, 640),             # 61 * 67 | K: ten
    (71 * 700009, 0),            # the prime that quarter rows are skipped by
])
def test_class_sieve_candidates_by_their_walks(ctx, K, shift):
    """A search's candidates stay on the device: those with a long walk come out
    as reports, with their n, and all of them are counted.  The window sieve's
    candidates, walked one batch after the other, give the same."""
    aps, st = ctx.search_k(K, shift)
    seen, reports = 0, []
    for cand in _lattice(ctx, K, shift):
        seen += len(cand)
        k, first, _ = ctx.chain_batch(K, cand)
        reports += [(int(k[i]), K, int(first[i]), int(cand[i])) for i in np.flatnonzero(k >= 10)]
    assert seen == st.candidates == st.chain_walks
    assert aps and sorted(reports) == sorted(aps)
