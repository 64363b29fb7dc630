"""The funnel verify at the edges of its words and chunks (GPU): segments of
one even to a few chunks of words, starting and ending at every residue mod
30, against the plan restated here: the pending evens are exactly those no
plan member settles, their words and their p(n)."""
import numpy as np
import pytest

import gbc

pytestmark = pytest.mark.gpu

U30 = (1, 7, 11, 13, 17, 19, 23, 29)


def odd_primes_upto(n):
    s = np.ones(n + 1, dtype=bool)
    s[:2] = False
    for i in range(2, int(n ** 0.5) + 1):
        if s[i]:
            s[i * i::i] = False
    return [int(p) for p in np.nonzero(s)[0] if p > 2]


CAND = odd_primes_upto(9781)


def is_prime_window(lo, hi):
    s = np.ones(hi - lo + 1, dtype=bool)
    s[lo % 2::2] = False
    for p in odd_primes_upto(int(hi ** 0.5) + 1):
        s[max(p * p, -(-lo // p) * p) - lo::p] = False
    return s


def plan(r, funnels):
    """Members of the class's plan: each uncovered useful candidate below 3000,
    ascending, opens a funnel of the uncovered primes p + 30 d, d < 32."""
    useful = [p for p in CAND if (r - p) % 30 in U30]
    known, covered, opened = set(useful), set(), 0
    for p in useful:
        if opened == funnels or p >= gbc.TAIL_T:
            break
        if p in covered:
            continue
        covered |= {p + 30 * d for d in range(32) if p + 30 * d in known and p + 30 * d < gbc.TAIL_T} - covered
        opened += 1
    return useful, covered


BASE = 10**9 + 2
CASES = [(BASE + 2 * i, w) for i, w in enumerate(
    [2, 4, 30, 32, 60, 958, 960, 962, 1920, 3838, 3840, 3842, 4 * 960, 128 * 960 - 2, 128 * 960, 128 * 960 + 2,
     512 * 960 + 14, 1_000_000 - 6, 3_999_994])]


@pytest.mark.parametrize("funnels", [1, 4, 5, 8, 32])
def test_pending_evens_are_the_plans(funnels):
    with gbc.Context(limit=BASE + 10**7, segment_even=4_000_000, max_batch=1, plan_funnels=funnels) as c:
        for a, w in CASES:
            if funnels < 5 and w > 10_000:  # few funnels leave more words than the list holds
                continue
            b = a + w - 2
            c.enqueue_batch(0, [(a, b)], b, [gbc.SEG_VERIFY])
            (s,), _ = c.collect(0, 1)
            lo = a - 9790
            prime = is_prime_window(lo, b)
            pend = words = 0
            hist = np.zeros((15, gbc.NCAND), dtype=np.int64)
            for r in range(0, 30, 2):
                n0 = a + (r - a) % 30
                if n0 > b:
                    continue
                n = np.arange(n0, b + 1, 30)
                useful, members = plan(r, funnels)
                open_ = np.ones(len(n), dtype=bool)
                for p in members:
                    open_ &= ~prime[n - p - lo]
                idx = np.nonzero(open_)[0]
                pend += len(idx)
                words += len(set((idx >> 5).tolist()))
                for e in n[idx].tolist():
                    p = next(p for p in useful if prime[e - p - lo])
                    hist[r // 2, CAND.index(p)] += 1
            assert (s.pending, s.npend, s.nleft, s.err) == (pend, words, 0, 0), (a, w)
            assert np.array_equal(np.frombuffer(s.hist, dtype=np.uint32).reshape(15, -1), hist), (a, w)


@pytest.mark.parametrize("want_pn", [False, True])
def test_exact_checker_edges(want_pn):
    """p(n) of every even on the same segments: the histogram by class, the
    first occurrences, the ridges from a low floor, and the p(n) array."""
    floor = 500
    for a, w in CASES:
        b = a + w - 2
        with gbc.Context(limit=BASE + 10**7, segment_even=4_000_000, max_batch=1, want_pn=want_pn,
                         ridge_min=floor if w < 10_000 else 3000) as c:
            c.enqueue_batch(0, [(a, b)], b)
            (s,), _ = c.collect(0, 1)
            got_pn = np.frombuffer(c.copy_pn(0, 0, w // 2), dtype=np.uint16) if want_pn else None
        prime = is_prime_window(a - 9790, b)
        n = np.arange(a, b + 1, 2)
        pn = np.zeros(len(n), dtype=np.int64)
        open_ = np.arange(len(n))
        for p in CAND:
            hit = prime[n[open_] - p - (a - 9790)]
            pn[open_[hit]] = p
            open_ = open_[~hit]
        assert not len(open_)
        index = {p: i for i, p in enumerate(CAND)}
        hist = np.zeros((15, gbc.NCAND), dtype=np.int64)
        first = np.full(gbc.NCAND, 0xFFFFFFFF, dtype=np.int64)
        ci = np.array([index[p] for p in pn])
        np.add.at(hist, (n % 30 // 2, ci), 1)
        np.minimum.at(first, ci, np.arange(len(n)))
        assert np.array_equal(np.frombuffer(s.hist, dtype=np.uint32).reshape(15, -1), hist), (a, w)
        assert np.array_equal(np.frombuffer(s.first, dtype=np.uint32), first), (a, w)
        ridges = sorted(zip(s.ridge_n[:s.nridge], s.ridge_p[:s.nridge]))
        at = pn >= (floor if w < 10_000 else 3000)
        assert ridges == list(zip(n[at].tolist(), pn[at].tolist())), (a, w)
        if want_pn:
            assert np.array_equal(got_pn, pn), (a, w)
