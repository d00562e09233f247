"""The kernel-level calls at the sizes and values where their paths change.

Sizes: a call of up to 1 MB of values is one kernel on pinned memory, a longer
one goes through sets of 8 MB in slices, by several host threads.  A long
call's results are those of short calls on its pieces (which the other files
check against the oracle and the reference's vectors).

Values: the base-2 test has a form for 2^33 <= N < 2^60 with an odd part of
N - 1 of at least six bits, and one for every other odd N; both against the
oracle at those limits.
"""
import ctypes

import numpy as np
import pytest

import ap26_b200 as A

pytestmark = pytest.mark.gpu

PIECE = 30_000          # one kernel on pinned memory for every call


def _values(rng, n):
    N = np.exp2(rng.uniform(2, 63, n)).astype(np.uint64)
    N[:8] = [0, 1, 2, 3, 4, 9, (1 << 63) - 25, 1 << 63]
    odd = rng.random(n) < 0.95
    N[odd] |= np.uint64(1)
    return rng.permutation(N)


@pytest.mark.parametrize("n", [1, 31, 131_072, 131_073, 1_048_576, 1_048_577, 4_300_001])
def test_long_sprp_batches_equal_their_pieces(ctx, n):
    N = _values(np.random.default_rng(n), max(8, n))[:n]
    got, st = ctx.sprp_batch(N)
    parts = [ctx.sprp_batch(N[i:i + PIECE]) for i in range(0, n, PIECE)]
    assert np.array_equal(got, np.concatenate([v for v, _ in parts]))
    assert st.late_items == sum(s.late_items for _, s in parts)     # modular squarings
    assert st.prp_tests == n


@pytest.mark.parametrize("n", [87_382, 700_001])
def test_long_base_batches_equal_their_pieces(ctx, n):
    rng = np.random.default_rng(n)
    N, a = _values(rng, n), rng.integers(2, 32, n, dtype=np.uint32)
    got, _ = ctx.sprp_bases(N, a)
    assert np.array_equal(got, np.concatenate(
        [ctx.sprp_bases(N[i:i + PIECE], a[i:i + PIECE])[0] for i in range(0, n, PIECE)]))


@pytest.mark.parametrize("n", [87_400, 750_003])
def test_long_chain_batches_equal_their_pieces(ctx, n):
    cand, _ = ctx.sieve_range(366384, 0, 0, 40 * 12673)
    c = np.resize(np.sort(cand), n)
    k, f, _ = ctx.chain_batch(366384, c)
    parts = [ctx.chain_batch(366384, c[i:i + PIECE]) for i in range(0, n, PIECE)]
    assert np.array_equal(k, np.concatenate([p[0] for p in parts]))
    assert np.array_equal(f, np.concatenate([p[1] for p in parts]))


@pytest.mark.parametrize("n", [18_725, 160_001])
def test_long_report_batches_equal_their_pieces(ctx, n):
    aps, _ = ctx.search_k(366384, 0)
    reps = (aps * (n // len(aps) + 1))[:n]
    rc, fin, h = ctx.report_batch(reps, result_hash=5)
    one, onefin, _ = ctx.report_batch(aps, result_hash=0)
    assert rc == one == 0
    assert all(bytes(f) == bytes(onefin[i % len(aps)]) for i, f in enumerate(fin))
    total = 5 + sum(onefin[i % len(aps)].hash_add for i in range(n))
    assert h == (total - 1) % 2_000_000_000 + 1


def test_sprp_forms_at_their_limits(ctx, oracle):
    N = []
    for e in (33, 34, 59, 60, 61, 62):
        N += [(1 << e) + d for d in range(-301, 301, 2)]
    N += list(range(3, 2000, 2)) + [(1 << 63) - d for d in range(1, 301, 2)]
    for e in range(3, 63):                       # N - 1 with a small odd part
        N += [m * (1 << e) + 1 for m in (1, 3, 5, 31, 33, 63, 65) if m << e < 1 << 62]
    N = np.array(N, np.uint64)
    got, _ = ctx.sprp_batch(N)
    exp = np.array([oracle.ao_sprp(ctypes.c_int64(int(n)), ctypes.c_int64(2)) for n in N], np.uint8)
    assert np.array_equal(got, exp)
    for a in (2, 3, 23, 31):
        M = N[N > a]
        got, _ = ctx.sprp_bases(M, np.full(len(M), a, np.uint32))
        exp = np.array([oracle.ao_sprp(ctypes.c_int64(int(n)), ctypes.c_int64(a)) for n in M],
                       np.uint8)
        assert np.array_equal(got, exp), a


@pytest.mark.parametrize("n", [1, 31, 33, 64, 65, 255, 257, 18_943, 131_072, 131_073,
                               606_208, 606_209])
def test_sprp_batches_of_mixed_lengths_keep_their_order(ctx, oracle, n):
    """Values are tested in the order of their length, a block's batch at a
    time: verdicts and squarings belong to their values at the edges of warps,
    batches and grids, with values that are not tested among them."""
    rng = np.random.default_rng(7)
    some = np.exp2(rng.uniform(1, 63.9, 2000)).astype(np.uint64) | np.uint64(1)
    some[::7] += np.uint64(1)                    # even
    some[:4] = 0, 1, 2, 3
    some[4:400] = [p for p in range(1 << 40, (1 << 40) + 20000) if _is_prime(p)][:396]
    tested = (some & np.uint64(1) > 0) & (some >= 3) & (some < np.uint64(1 << 63))
    exp = np.array([t and oracle.ao_sprp(ctypes.c_int64(int(x)), ctypes.c_int64(2))
                    for x, t in zip(some, tested)], np.uint8)
    assert 300 < exp.sum() < 800
    each = np.array([ctx.sprp_batch(some[i:i + 1])[1].late_items for i in range(len(some))])
    pick = rng.integers(0, len(some), n)
    got, st = ctx.sprp_batch(some[pick])
    assert np.array_equal(got, exp[pick])
    assert st.late_items == each[pick].sum()


def _is_prime(n):
    return all(n == p or (n % p and _strong(n, p)) for p in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37))


def _strong(n, a):
    d, t = n - 1, 0
    while d % 2 == 0:
        d, t = d // 2, t + 1
    x = pow(a, d, n)
    return x in (1, n - 1) or any((x := x * x % n) == n - 1 for _ in range(t - 1))


@pytest.mark.parametrize("bits", [35, 59, 61])
def test_sprp_over_the_powers_of_two_in_n_minus_one(ctx, bits):
    """2^-d and the squares after it are looked for in the last squares of one
    loop: primes and composites with every 2^t in N - 1 on both sides of that
    length, and products p(2p - 1) and p(3p - 2), many of which are
    pseudoprimes whose square roots of 1 decide."""
    rng = np.random.default_rng(bits)
    N, psp = [], 0
    for t in range(1, 24 if bits < 40 else 40):
        primes = 0
        while primes < 12:
            n = (int(rng.integers(1 << (bits - t - 1), 1 << (bits - t))) | 1) << t | 1
            N.append(n)
            primes += _is_prime(n)
    for m in (2, 3):
        p = int(2 ** (bits / 2)) // m | 1
        while psp < 40 * (m - 1):
            p += 2
            if _is_prime(p) and _is_prime(m * (p - 1) + 1):
                N.append(p * (m * (p - 1) + 1))
                psp += 1
    exp = np.array([_strong(n, 2) for n in N], np.uint8)
    got, _ = ctx.sprp_batch(np.array(N, np.uint64))
    assert np.array_equal(got, exp)
    assert np.array_equal(ctx.sprp_bases(np.array(N, np.uint64), np.full(len(N), 2, np.uint32))[0],
                          exp)


def test_chain_terms_past_the_end_of_a_walk_do_not_count(ctx):
    """Terms are tested ahead of a walk: one at 2^62 or beyond is an error only
    where the walk reaches it (2^62 is the domain of the reference's PrimeQ)."""
    K = 50_000_001
    S = K * A.PRIM23
    top = (1 << 62) - 1
    n = next(m for m in range(top, top - 12, -1) if m % 3 == 0 and m % 2) - 5 * S
    k, f, _ = ctx.chain_batch(K, np.array([n], np.int64))
    assert (k[0], f[0]) == (0, n + 6 * S)        # n + 5S composite, n + 6S beyond 2^62
    for bad in (n + S, n + 4):
        with pytest.raises(A.AP26Error) as e:
            ctx.chain_batch(K, np.array([bad], np.int64))
        assert e.value.code == A.E_DOMAIN
