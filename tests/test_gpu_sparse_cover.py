"""The sparse checker's entries (GPU): the evens it leaves are those without a
witness in the plan, for plans cut within a group of the word form, within a
later group and between groups, and for candidate limits with the fewest and
the most window words (all pattern rows and fewer of them)."""
import numpy as np
import pytest

import gbc

pytestmark = pytest.mark.gpu
M = 30030


@pytest.mark.parametrize("pmax,cap", [(100_000, 0), (100_000, 2), (40_000_000, 3), (40_000_000, 5), (40_000_000, 8),
                                      (40_000_000, 0), (200_000_000, 4)])
def test_leftovers_are_the_evens_without_a_witness(pmax, cap):
    start, count = 4 * 10**18 + 13 * M + 777778, 1_000_003 if pmax > 100_000 else 60_001
    with gbc.Sparse(limit=4 * 10**18 + 10**12, dlt_log2=16, pmax=pmax, group_cap=cap) as sp:
        r = sp.verify(start, start + 2 * (count - 1))
        w = np.array(sp.witness(start, count))
        assert r.evens == count
        assert sp.pending() == [start + 2 * int(j) for j in np.flatnonzero(w == 0)]


def test_leftovers_of_whole_chunks():
    """A segment of two chunks: every class whole, every word of a lane."""
    start = 4 * 10**18 - 4 * 10**18 % M
    with gbc.Sparse(limit=4 * 10**18 + 10**12, dlt_log2=14, group_cap=14) as sp:
        r = sp.verify(start, start + M * 2**14 - 2)
        assert r.evens == M // 2 * 2**14 and r.segments == 1
        pend = sp.pending()
        for i0 in (0, 4090, 8191, 16320):  # the first, a middle, both sides of the chunks' seam, the last words
            a, n = start + M * i0, M // 2 * 60
            w = np.array(sp.witness(a, n))
            assert [x for x in pend if a <= x < a + 2 * n] == [a + 2 * int(j) for j in np.flatnonzero(w == 0)]
