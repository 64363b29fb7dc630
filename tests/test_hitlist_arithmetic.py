"""The hit-list harvest's placement of a prime's multiples (k_hitlist in
goldbach-l0_gb300/csrc/k_sieve.cu), restated in exact float32 and integer
arithmetic and compared with the general definition: the multiples q = p m of
a run, m coprime to 30, as class bits, for runs narrower than p / 4 bits (a few
candidate multipliers), primes from 2^31 on (64-bit bits) and the word loop
(32-bit bits). A CPU test of the algorithm; the GPU tests check the kernel
through every map bit."""
import math
import random
from fractions import Fraction as F

import pytest

from test_modulo_emulation import f2i_rn, f2u_rz, rn32

U30 = (1, 7, 11, 13, 17, 19, 23, 29)
M32, M64 = 2**32 - 1, 2**64 - 1


def recip64(p):
    rp = rn32(F(1, int(rn32(F(p)))))
    if p < 1 << 20:
        return M64 // p
    q1 = f2u_rz(rn32(rp * 2**52))
    d = 2**52 - q1 * p
    assert abs(d) < 2**33
    c = f2i_rn(rn32(rn32(F(d >> 2)) * rn32(rp * 2**14)))
    return (q1 << 12) + c - 2


def recip64_exact(p):
    inv = recip64(p)
    e = 2**64 - inv * p
    assert 0 <= e < 5 * p
    for step in (2, 1):
        if e >= p * step:
            e -= p * step
            inv += step
    return inv + 1 if e >= p else inv


def divmod_recip(x, p, recip=recip64):
    q = x * recip(p) >> 64
    r = x - q * p
    assert 0 <= r < 2 * p
    return (q + 1, r - p) if r >= p else (q, r)


def marks(base, nblk, p, several=False):
    """(class residue, bit) of every multiple p m in the run, m coprime to 30,
    by the kernel's steps (several: of a batch of several runs), every table
    bit taken as set."""
    rp = rn32(F(1, int(rn32(F(p)))))
    span = min(30 * nblk - 1, M32)
    if several and span < p >> 6 and not p >> 31:
        r = ((base - 1) - ((base - 1) * recip64_exact(p) >> 64) * p) & M32
        assert r < 2 * p
        r = min(r, (r - p) & M32)
        if r < p - 1 - span:
            return None, set()
    b0, rho = divmod_recip(base // 30, p, recip64_exact if several else recip64)
    pq, pr = divmod(p, 30)
    out = set()

    def v(u):
        return pq * u + pr * u // 30

    one = nblk <= p >> 5
    if one or (nblk <= p >> 2 and not p >> 31):
        a = rn32(rn32(F(rho)) * rn32(30 * rp))
        j0 = math.ceil(max(rn32(a - rn32(F(1, 100))), 0))
        n = 1 if one else f2u_rz(rn32(rn32(F(nblk)) * rn32(30 * rp))) + 3
        assert j0 <= 30 and n <= 10
        for j in range(j0, j0 + n):
            nxt, j = j >= 30, j % 30
            if j not in U30 or (nxt and one):
                continue
            t = ((p if nxt else 0) + pq * j + ((pr * j * 2185) >> 16) - rho) & M32
            if t < nblk:
                out.add((p * j % 30, t))
        return b0, out
    if p >> 31:
        for nb in range(2 if rho + nblk > p else 1):
            out |= {(p * u % 30, nb * p + v(u) - rho) for u in U30 if 0 <= nb * p + v(u) - rho < nblk}
        return b0, out
    x = rho + nblk - 1
    assert x <= M32
    nb = f2u_rz(rn32(rn32(F(x)) * rp))
    if nb * p > x:
        nb -= 1
    elif x - nb * p >= p:
        nb += 1
    assert nb == x // p
    f30 = rn32(30 * rp)
    ja = math.ceil(max(rn32(rn32(rn32(F(rho)) * f30) - rn32(F(1, 100))), 0))
    jb = f2u_rz(rn32(rn32(rn32(F(x - nb * p + 1)) * f30) + rn32(F(1, 100))))
    assert ja <= 30 and jb <= 30
    for b in range(nb + 1):
        for u in U30:
            if (b == 0 and u < ja) or (b == nb and u > jb):  # outside the end bytes' masks
                continue
            t = (b * p + v(u) - rho) & M32
            if t < nblk:
                out.add((p * u % 30, t))
    return b0, out


def general(base, nblk, p):
    m, out = -(-base // p), set()
    while p * m < base + 30 * nblk:
        if m % 30 in U30:
            out.add((p * m % 30, (p * m - base) // 30))
        m += 1
    return out


PRIMES = [131, 1009, 65537, 1048573, 1048583, 1703941, 4194319, 16777259, 99999989, 499999993,
          1999999973, 2147483647, 2147483659, 2236067969, 4294967291]


@pytest.mark.parametrize("p", PRIMES)
def test_division_by_the_reciprocal(p):
    rnd = random.Random(p)
    assert recip64_exact(p) == 2**64 // p and 0 <= 2**64 - recip64(p) * p < 6 * p
    top = (2**64 - 2**40) // 30
    for x in [0, 1, p - 1, p, top, top // p * p, top // p * p - 1] + [rnd.randrange(top) for _ in range(200)]:
        assert divmod_recip(x, p) == divmod(x, p)


@pytest.mark.parametrize("p", PRIMES)
def test_marks_equal_the_general_form(p):
    rnd = random.Random(p + 1)
    widths = {1, 2, 33, max(p >> 5, 1), (p >> 5) + 1, p // 30 + 1, p // 8, max(p >> 2, 1), (p >> 2) + 1, p // 2 + 1, p - 1,
              p, p + 1, 40 * p}
    for nblk in sorted(w for w in widths if 0 < w < 2**31 and w < 4096 * p):
        if nblk // p > 50:
            continue
        for _ in range(12):
            # bases whose first multiple sits at either end of the run or anywhere
            m = rnd.randrange(p, max(p + 1, min(2**63 // p, 1 << 42)))
            off = rnd.choice((0, 30, -30, 30 * nblk, 30 * (nblk - 1), rnd.randrange(30 * p)))
            base = max(30, p * m - off) // 30 * 30
            want = general(base, nblk, p)
            assert marks(base, nblk, p)[1] == want and marks(base, nblk, p, True)[1] == want, (p, nblk, base)


def test_small_product_division_by_30():
    assert all((x * 2185) >> 16 == x // 30 for x in range(900))
