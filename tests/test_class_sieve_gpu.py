"""The class sieve (every whole-K run) against the window sieve, which
test_gpu_parity.py checks against the oracle: survivors of the whole lattice.

The K are the ones where the class sieve's shapes change: a class prime (61,
67) dividing K lets more (b, j) through, so a class has more than four rows;
a dense or tail prime dividing K keeps almost every candidate to the stages
behind it; the smallest and largest K and SHIFT; and launches of a single
unit's classes and of the whole K at once.  The counts are integers: equal.
"""
import pytest

import ap26_b200 as A

pytestmark = pytest.mark.gpu

SLICES = 16


def _window_count(ctx, K, shift):
    step = -(-A.N53_PER_K // SLICES)
    return sum(len(ctx.sieve_range(K, shift, q0, min(q0 + step, A.N53_PER_K), cap=1 << 25)[0])
               for q0 in range(0, A.N53_PER_K, step))


@pytest.mark.parametrize("K,shift,chunk_tiles", [
    (1, 0, 131072),
    (400_000_000, 640, 131072),          # AP26_KMAX_SAFE
    (43241061, 15360, 1 << 20),          # one launch; near the SHIFT limit
    (42700061, 1280, 131072),            # 61 | K: seven rows a class
    (67 * 700009, 0, 131072),            # 67 | K
    (28686653, 640, 60000),              # 61 * 67 | K: ten rows a class
    (71 * 700009, 0, 4099),              # a dense modulus's prime, small launches
    (179 * 200003, 1344, 131072),        # a tail product's prime
    (541 * 70001, 0, 131072),            # the last single prime
])
def test_whole_k_survivors_equal_the_window_sieves(K, shift, chunk_tiles):
    assert A.will_search(K)
    with A.Context(0, chunk_tiles=chunk_tiles) as ctx:
        counts, _ = ctx.sieve_count([K, K - 31 if K > 31 else K + 31], shift)
        assert counts[0] == _window_count(ctx, K, shift)
        aps, st = ctx.search_k(K, shift)
        assert st.candidates == st.chain_walks == counts[0]
        assert st.error_flags == 0


@pytest.mark.parametrize("K,ring,sieves", [
    (43241061, 27, 1),                   # 36.9 M fit with a quarter to spare
    (43241061, 25, 2),                   # 33.5 M entries: two launches
    (61 * 7019, 26, 2),                  # 61 | K: 59.8 M, too near to 67.1 M
    (21182921, 26, 4),                   # the densest K: 201 M
    (43241061, 22, 5),                   # never more launches than chunk_tiles asks for
])
def test_launches_of_a_k_by_the_survivors_a_ring_holds(K, ring, sieves):
    with A.Context(0, cand_ring_log2=ring) as ctx:
        counts, st = ctx.sieve_count([K], 0)
        assert st.launches == 1 + 5 + 3              # counts alone: one launch
        aps, st = ctx.search_k(K, 0)
        assert st.candidates == st.chain_walks == counts[0]
        if ring > 22:                                # there a chunk overflows and is redone
            assert st.launches == 1 + 5 + 4 * sieves + 1
            assert st.error_flags == 0
    with A.Context(0, chunk_tiles=131071) as ctx:    # a set size bounds the launches
        want, st = ctx.search_k(K, 0)
        assert st.launches == 1 + 5 + 4 * 5 + 1
        assert aps == want
