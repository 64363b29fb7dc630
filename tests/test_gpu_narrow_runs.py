"""Narrow runs (GPU): where the sieving primes past the tiles (less three
million) are five or more per integer of the run, what the tiles leave is tested for primality number by
number. The maps equal those of the read-before-mark sieve bit for bit, on both
sides of that line, in batches with wide runs, and at strong base-2
pseudoprimes, which only the test's second half turns away."""
import numpy as np
import pytest

import gbc
import oracle

pytestmark = pytest.mark.gpu
TUNED = dict(p_mid=1703936, tile_bits=1835008)


def maps(segs, limits, limit, **kw):
    with gbc.Context(limit=limit, max_batch=max(8, len(segs)), **kw) as c:
        c.enqueue_segments(0, segs, limits, [gbc.SEG_VERIFY if i % 2 else 0 for i in range(len(segs))])
        res, t = c.collect(0, len(segs))
        out = [(b, n, [np.array(w[k * wpc:k * wpc + n // 32]) for k in range(8)],
                [int(w[k * wpc + n // 32]) & ((1 << n % 32) - 1) if n % 32 else 0 for k in range(8)])
               for b, n, wpc, w in (c.map(0, r) for r in range(t.runs))]
        return out, [(list(r.primes30), list(r.twins), list(r.ghist), r.ntail, r.gmax_key) for r in res], c.stats()


def same(segs, limits, limit, knobs, **general):
    got, res, st = maps(segs, limits, limit, selfcheck_every=1, **knobs)
    want, ref, _ = maps(segs, limits, limit, **general, **knobs)
    assert res == ref and len(got) == len(want) and st.selfchecks == 1
    for (b, n, w, e), (b2, n2, w2, e2) in zip(got, want):
        assert (b, n, e) == (b2, n2, e2)
        for k in range(8):
            assert np.array_equal(w[k], w2[k]), (b, k)
    return st, got


@pytest.mark.parametrize("a,width,knobs,narrow", [
    (10**16, 400_000, dict(p_mid=128), True),      # tiles of 31 primes: many more bits a word are tested
    (10**16, 600_000, dict(p_mid=128), False),
    (10**16, 30, {}, True),
    (10**16, 500_000, TUNED, True),
    (10**16, 540_000, TUNED, False),
    (25 * 10**14, 2, TUNED, False),                # less than three million primes
    (4 * 10**18, 2, TUNED, True),
    (4 * 10**18 + 2, 8 * 30 * 32 * 3, {}, True),   # list words of a warp: full, and a rest of one
    (4 * 10**18, 3_333_332, TUNED, True),          # several words a warp
    (4 * 10**18, 17_000_000, TUNED, True),
    (4 * 10**18, 20_000_000, TUNED, False),
    (gbc.MAX_LIMIT - 2_000_000, 2_000_000, {}, True),
])
def test_maps_on_both_sides_of_the_line(a, width, knobs, narrow):
    st, _ = same([(a, a + width)], [a + width], a + width, knobs, hl_mode=2)
    # lists on (a batch this wide): their multiplier table is built where a run needs it
    assert st.mtab_builds == (0 if narrow else 1)


def test_narrow_and_wide_runs_in_one_batch():
    h = 4 * 10**18
    segs = [(h, h + 100_000), (h + 10**12, h + 10**12 + 40_000_000), (h + 2 * 10**12, h + 2 * 10**12 + 999_998),
            (10**10, 10**10 + 50_000), (h + 2 * 10**12 + 10**6, h + 2 * 10**12 + 2 * 10**6),
            (10**16, 10**16 + 400_000), (h + 3 * 10**12, h + 3 * 10**12 + 2), (4, 20_000)]
    same(segs, [b for _, b in segs], h + 4 * 10**12, TUNED, hl_mode=2)


def strong_base2(n):
    d, s = n - 1, 0
    while d % 2 == 0:
        d, s = d // 2, s + 1
    x = pow(2, d, n)
    return x in (1, n - 1) or any((x := x * x % n) == n - 1 for _ in range(s - 1))


def test_strong_base2_pseudoprimes():
    """(k + 1)(2 k + 1) of two primes past the tile primes, strong to base 2."""
    found, k = [], 1_414_213_562
    while len(found) < 12:
        k += 2
        n = (k + 1) * (2 * k + 1)
        if strong_base2(n) and oracle.is_prime(k + 1) and oracle.is_prime(2 * k + 1):
            found.append(n)
            k += 10_000
    segs = [((n - 500) // 2 * 2, (n + 500) // 2 * 2) for n in found]
    _, got = same(segs, [b for _, b in segs], segs[-1][1], {}, hl_mode=2)
    unit = (1, 7, 11, 13, 17, 19, 23, 29)
    for n, (base, nblk, words, rest) in zip(found, got):
        t, k = (n - base) // 30, unit.index(n % 30)
        assert not ((int(words[k][t // 32]) if t // 32 < len(words[k]) else rest[k]) >> (t % 32)) & 1, n
