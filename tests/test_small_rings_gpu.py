"""A candidate ring that is smaller than the class sieve's smallest launch.

A K that 61 or 67 divides has units of up to 4850 survivors, the densest K of
15200: more than the smallest ring of 4096.  There the window sieve, whose
chunks can be a few tiles, searches the K: same reports, same survivors.
"""
import pytest

import ap26_b200 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,opts", [
    (42700061, {"cand_ring_log2": 12}),                    # 61 | K
    (67 * 700009, {"cand_ring_log2": 12, "chunk_tiles": 32, "use_graphs": -1}),   # 67 | K
    (61 * 67 * 71 * 73, {"cand_ring_log2": 13, "chunk_tiles": 20}),   # the densest K
])
def test_a_ring_below_a_unit(ctx, K, opts):
    want, st = ctx.search_k(K, 0)
    with A.Context(0, **opts) as small:
        got, small_st = small.search_k(K, 0)
        assert got == want
        assert small_st.candidates == small_st.chain_walks == st.candidates
        assert small_st.error_flags == 1                   # redone
        assert small.opts["chunk_tiles"] == opts.get("chunk_tiles", 131072)


def test_a_batch_with_one_dense_k(ctx):
    """The K of a run are redone together: the ordinary ones keep their results."""
    items = [(1, 42700060, 42700061, 0)]
    want, res, _ = ctx.search_batch(items)
    with A.Context(0, cand_ring_log2=12, chunk_tiles=32) as small:
        got, small_res, st = small.search_batch(items)
        assert got == want and st.error_flags == 1
        assert [(r.result_hash, r.candidates, r.ks_searched) for r in small_res] == \
            [(r.result_hash, r.candidates, r.ks_searched) for r in res]
