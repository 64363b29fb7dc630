"""Hit lists of the widest run a context takes (2^31 class bits and the
checkers' margin) for a prime below 2^31 whose position in the run and the run's
width add up to more than 2^32 (GPU): each segment's map is that of the same
segments in two runs of half the width."""
import ctypes as C

import pytest

import gbc

pytestmark = pytest.mark.gpu

P = 2**31 - 1


def is_prime(n):
    d, s = n - 1, 0
    while d % 2 == 0:
        d, s = d // 2, s + 1
    for a in (2, 3, 5, 7, 11, 13):
        x = pow(a, d, n)
        if x in (1, n - 1):
            continue
        for _ in range(s - 1):
            x = x * x % n
            if x == n - 1:
                break
        else:
            return False
    return True


@pytest.mark.parametrize("back", [1, 100, 300])
def test_widest_run_against_two_halves(back):
    # blocks of 30 below P * b that start the run `back` blocks early; several multipliers of b's block are prime
    b = 77_600_000
    while sum(is_prime(30 * b + u) for u in (1, 7, 11, 13, 17, 19, 23, 29)) < 4:
        b += 1
    base = 30 * (P * b - back)
    start = base + 9796  # even; its map starts at base
    n, seg = 30, 2**31
    segs = [(start + i * seg, start + (i + 1) * seg - 2) for i in range(n)]
    end = segs[-1][1]
    with gbc.Context(limit=end, segment_even=seg, max_batch=n, ridge_min=9000) as c:
        flags = [gbc.SEG_VERIFY] * n

        def run(part):
            c.enqueue_batch(0, part, end, flags[:len(part)])
            return [(s.map_primes, s.map_hash, s.pending) for s in c.collect(0, len(part))[0]]
        whole = run(segs)
        at, nblk = C.c_uint64(), C.c_uint32()
        c._check(c.lib.gbc_map_run(c.h, 0, 0, C.byref(at), C.byref(nblk), None, None, 0))
        assert at.value == base and P - back + nblk.value - 1 >= 2**32
        assert run(segs[:n // 2]) + run(segs[n // 2:]) == whole

