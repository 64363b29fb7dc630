"""The tile sieve's largest prime (kMaxTilePrime): the marks' 32-bit arithmetic
(clear_stride in goldbach-l0_gb300/csrc/k_sieve.cu), restated, leaves the tile
for larger ones; and a context whose p_mid lies above it sieves the same map (GPU)."""
import os
import re

import pytest

import gbc
from conftest import ROOT

M32 = 2**32 - 1
END = 8 * 233472 + 1835008  # the last bit of the largest tile, as marks address it, at shared memory's end


def clear_stride(b, st, end):
    """The bits a lane clears."""
    out = []
    while (b + 3 * st) & M32 < end:
        out += [(b + i * st) & M32 for i in range(4)]
        b = (b + 4 * st) & M32
    while b < end:
        out.append(b)
        b = (b + st) & M32
    return out


def test_marks_stay_in_the_tile():
    src = open(os.path.join(ROOT, "goldbach-l0_gb300", "csrc", "gbc_common.cuh")).read()
    m = re.search(r"kMaxTilePrime = uint32_t\(\(\(1ull << 32\) - \(1u << 22\)\) / 3\)", src)
    assert m, "no bound on the tile sieve's primes"
    largest = (2**32 - 2**22) // 3
    for p in [97, 14321, 1703941, 2**22 + 15, largest // 2, largest - 1, largest]:
        for b in {0, 1, p % END, END - 1}:
            assert clear_stride(b, p, END) == list(range(b, END, p))
    over = 2**32 // 3 + 7  # four marks far outside the tile
    assert max(clear_stride(0, over, END)) > END


@pytest.mark.gpu
@pytest.mark.parametrize("p_mid", [2**32 - 1, 1_500_000_000])
def test_large_p_mid(p_mid):
    a = 9_200_000_000_000_000_000
    seg = (a, a + 200_000)

    def run(**kw):
        with gbc.Context(limit=seg[1], segment_even=1_000_000, max_batch=1, **kw) as c:
            c.enqueue_batch(0, [seg], seg[1])
            s = c.collect(0, 1)[0][0]
            return s.map_primes, s.map_hash, list(s.primes30), list(s.hist[0])
    assert run(p_mid=p_mid, hl_mode=2) == run()
