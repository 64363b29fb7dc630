"""How the hit-listed primes are dealt out to the harvest's CTAs (hl_deal in
goldbach-l0_gb300/csrc/k_sieve.cu): a CTA's marks stay within a bin's quota, the
mean and 45%, but for a few primes, whose marks the overflow list holds. The
choice is taken from the built library; the shares are computed here, prime by
prime. And wide batches whose shares differed most pass their map self-check (GPU)."""
import ctypes as C
import math
import os

import numpy as np
import pytest

import gbc

CTAS, THREADS, ROUNDS = 304, 768, 512
BLOCKS, WARPS, LANES = 0, 1, 2


@pytest.fixture(scope="module")
def primes():
    n = math.isqrt(10**16)
    s = np.ones(n // 2 + 1, dtype=bool)
    s[0] = False
    for i in range(3, math.isqrt(n) + 1, 2):
        if s[i // 2]:
            s[i * i // 2::i] = False
    return (2 * np.nonzero(s)[0] + 1).astype(np.uint32)


@pytest.fixture(scope="module")
def lib():
    if not os.path.exists(gbc.LIB_PATH):
        pytest.skip("the library is not built")
    lib = C.CDLL(gbc.LIB_PATH)
    lib._ZN3gbh9hl_sharesEPKjjjjPNS_8HlSharesE.argtypes = [C.c_void_p, C.c_uint32, C.c_uint32, C.c_uint32, C.c_void_p]
    lib._ZN3gbh9hl_sharesEPKjjjjPNS_8HlSharesE.restype = None
    f = lib._ZN3gbh7hl_dealEPKNS_8HlSharesEPKjjjjb
    f.argtypes, f.restype = [C.c_void_p, C.c_void_p, C.c_uint32, C.c_uint32, C.c_uint32, C.c_bool], C.c_uint32
    return lib


def cta_of(deal, n):
    i = np.arange(n)
    return (i // THREADS if deal == BLOCKS else i // 32 if deal == WARPS else i) % CTAS


def excess(p, q, deal):
    """The part of the marks above 1.45 times the mean of the CTAs."""
    p = p.astype(float)
    s = np.bincount(cta_of(deal, len(p)), 1 / (p * np.log(q / p)), CTAS)
    return np.maximum(s / s.mean() - 1.45, 0).sum() / CTAS


def first_share(p, deal):
    s = np.bincount(cta_of(deal, len(p)), 1 / p.astype(float), CTAS)
    return s[0] / s.mean()


@pytest.mark.parametrize("first", [2156, 10001, 16411, 65537, 262147, 1048583, 1703941, 4194319, 16777259])
def test_no_cta_above_a_bin_s_quota(lib, primes, first):
    lo = int(np.searchsorted(primes, first))
    pr = primes.ctypes.data
    for q in (10**10, 10**11, 10**12, 10**13, 18 * 10**12, 10**14, 10**15, 4 * 10**15, 10**16):
        hi = int(np.searchsorted(primes, math.isqrt(q), side="right"))
        if hi - lo < 3 * CTAS or first**3 < q:
            continue
        # a context of this height and a lower batch of a context that reaches 1e16
        for top in {hi, len(primes)}:
            shares = (C.c_double * (2 * (ROUNDS + 1)))()
            lib._ZN3gbh9hl_sharesEPKjjjjPNS_8HlSharesE(pr, lo, top, CTAS, shares)
            deal = lib._ZN3gbh7hl_dealEPKNS_8HlSharesEPKjjjjb(shares, pr, lo, hi, CTAS, True)
            few = hi - lo < 8 * THREADS * CTAS
            assert excess(primes[lo:hi], q, deal) < 0.005, (first, q, deal)
            # and no finer than the first CTA's share of 1 / p asks for (1.40, the sums' ends aside)
            assert deal == BLOCKS or few or first_share(primes[lo:hi], BLOCKS) > 1.38, (first, q)
            assert deal != LANES or first_share(primes[lo:hi], WARPS) > 1.38, (first, q)
            # marks that go straight to the map take no bin: as before
            assert lib._ZN3gbh7hl_dealEPKNS_8HlSharesEPKjjjjb(shares, pr, lo, hi, CTAS, False) == (WARPS if few else BLOCKS)


@pytest.mark.gpu
@pytest.mark.parametrize("height,p_mid,n", [(10**15, 1 << 18, 24), (10**12, 9000, 16), (18 * 10**12, 1 << 22, 24),
                                            (10**16, 1 << 18, 16)])
def test_wide_batches(height, p_mid, n):
    seg = gbc.DEFAULT_SEGMENT
    segs = [(height + i * seg, height + (i + 1) * seg - 2) for i in range(n)]
    limit = segs[-1][1]
    with gbc.Context(limit=limit, max_batch=n, p_mid=p_mid, hl_mode=1, selfcheck_every=1) as c:
        c.enqueue_batch(0, segs, limit, [gbc.SEG_VERIFY] * n)
        res, _ = c.collect(0, n)  # raises when the overflow list is full or a map word differs
        assert c.stats().selfchecks == 1 and all(r.err == 0 for r in res)
