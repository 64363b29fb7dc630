"""Hit lists of one run and of several (GPU): runs at heights that few or many
sieving primes reach, in no order, binned and (more runs than the bins take)
marked directly; the maps equal the rebuild without hit lists."""
import random

import pytest

import gbc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 20, 150])
def test_runs_of_uneven_heights(n):
    rnd = random.Random(n)
    segs = []
    for i in range(n):
        a = int(10 ** rnd.uniform(13, 18.6)) // 2 * 2
        segs.append((a, a + int(10 ** rnd.uniform(3, 8 if i % 5 == 0 else 6)) // 2 * 2))
    limit = max(b for _, b in segs)
    with gbc.Context(limit=limit, segment_even=200_000_000, max_batch=n, max_runs=n, hl_mode=1, selfcheck_every=1, mtab_max_gb=8,
                     p_mid=1703936, tile_bits=1835008) as c:
        for s in (segs, segs[::-1]):
            c.enqueue_segments(0, s, [b for _, b in s], [gbc.SEG_VERIFY] * n)
            res, _ = c.collect(0, n)  # raises where a map word differs
            assert all(r.err == 0 for r in res)
        assert c.stats().selfchecks == 2
