"""ap26_sieve_range splits each start's 35 n59 values into 35, 7, 5 or 1 tiles
by the length of the range.  A range of each split gives the candidates of its
pieces, which are short enough for the finest split; that one is checked
against the oracle in test_gpu_parity.py."""
import numpy as np
import pytest

import ap26_b200 as A

pytestmark = pytest.mark.gpu

PIECE = 40_000          # starts: 35 parts whatever the variant


@pytest.mark.parametrize("starts", [90_001, 130_003, 640_007])
@pytest.mark.parametrize("vi", [0, 1])          # CTAs of 256 and of 384 starts
def test_range_equals_its_pieces(ctx, starts, vi):
    variants = A.list_variants()
    ctx.set_opts(**variants[vi])
    try:
        q0 = A.N53_PER_K - starts                # ends with the lattice
        got, _ = ctx.sieve_range(43241061, 1280, q0, q0 + starts)
        pieces = [ctx.sieve_range(43241061, 1280, q, min(q + PIECE, q0 + starts))[0]
                  for q in range(q0, q0 + starts, PIECE)]
        assert np.array_equal(np.sort(got), np.sort(np.concatenate(pieces)))
    finally:
        ctx.set_opts(**variants[0])
