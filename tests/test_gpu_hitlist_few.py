"""Hit lists of few primes in a wide batch (GPU): at 1e13 with the tile primes
to 1.7e6 the hit-listed primes are fewer than the harvest's threads; the
harvest CTAs' region bins must hold their marks, and the maps equal the
rebuild without hit lists."""
import pytest

import gbc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("height", [10**13, 3 * 10**13, 10**14])
def test_few_hit_listed_primes(height):
    seg = gbc.DEFAULT_SEGMENT
    segs = [(height + i * seg, height + (i + 1) * seg - 2) for i in range(58)]
    limit = segs[-1][1]
    with gbc.Context(limit=limit, max_batch=58, p_mid=1703936, tile_bits=1835008, hl_mode=1, selfcheck_every=1) as c:
        c.enqueue_batch(0, segs, limit, [gbc.SEG_VERIFY] * 58)
        res, _ = c.collect(0, 58)  # raises when the overflow list is full or a map word differs
        assert c.stats().selfchecks == 1 and all(r.err == 0 for r in res)
