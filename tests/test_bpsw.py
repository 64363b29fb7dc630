"""The primality test of narrow runs (struct Bpsw in
goldbach-l0_gb300/csrc/k_sieve.cu), its own source compiled for the CPU with the
device intrinsics restated: the Lucas parameter is the first P from 3 on whose
P^2 - 4 has Jacobi symbol -1, a symbol of 0 before it (a common factor) makes
the number composite, and the test tells primes from composites."""
import os
import random
import re
import subprocess

import pytest

from conftest import ROOT

SHIM = """
#include <cstdint>
#include <cstdio>
#define __device__
#define __forceinline__ inline
#define __noinline__
static uint64_t __umul64hi(uint64_t a, uint64_t b) { return uint64_t((unsigned __int128)a * b >> 64); }
static int __ffs(int x) { return __builtin_ffs(x); }
static int __ffsll(long long x) { return __builtin_ffsll(x); }
static int __clz(int x) { return __builtin_clz(x); }
static int __clzll(long long x) { return __builtin_clzll(x); }
%s
int main()
{
    unsigned long long n;
    while (std::scanf("%%llu", &n) == 1) {
        const Bpsw t(n);
        std::printf("%%u %%d %%d\\n", t.lucas_p(), int(t.base2()), int(t.lucas()));
    }
}
"""


@pytest.fixture(scope="module")
def bpsw(tmp_path_factory):
    src = open(os.path.join(ROOT, "goldbach-l0_gb300", "csrc", "k_sieve.cu")).read()
    body = re.search(r"^struct Bpsw \{.*?^\};", src, re.S | re.M).group(0)
    d = tmp_path_factory.mktemp("bpsw")
    (d / "t.cpp").write_text(SHIM % body)
    subprocess.run(["g++", "-std=c++20", "-O1", "-w", "-o", str(d / "t"), str(d / "t.cpp")], check=True)

    def run(ns):
        r = subprocess.run([str(d / "t")], input="".join(f"{n}\n" for n in ns), capture_output=True, text=True, check=True)
        return [tuple(map(int, x.split())) for x in r.stdout.splitlines()]
    return run


def jacobi(a, n):
    a, s = a % n, 1
    while a:
        while a % 2 == 0:
            a //= 2
            s = -s if n % 8 in (3, 5) else s
        a, n = n, a
        s = -s if a % 4 == n % 4 == 3 else s
        a %= n
    return s if n == 1 else 0


def parameter(n):
    p = 3
    while jacobi(p * p - 4, n) == 1:
        p += 1
    return p if jacobi(p * p - 4, n) == -1 else 0


def strong(n, a):
    d, s = n - 1, 0
    while d % 2 == 0:
        d, s = d // 2, s + 1
    x = pow(a, d, n)
    return x in (1, n - 1) or any((x := x * x % n) == n - 1 for _ in range(s - 1))


def is_prime(n):
    return all(strong(n, a) for a in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37))


def small_factor(n):
    return any(n % f == 0 for f in range(3, 128, 2))


# every prime below 128 a quadratic residue: the first P is past 126, where a
# factor of P^2 - 4 can be one of these numbers' own (131, 137, 149)
FAR = [131 * 65851211, 131 * 67721891, 137 * 62791073, 137 * 63908993, 149 * 59325989, 149 * 61221269]


def test_a_common_factor_makes_the_number_composite(bpsw):
    assert all(parameter(n) == 0 for n in FAR)
    for n, (p, _, lucas) in zip(FAR, bpsw(FAR)):
        assert (p, lucas) == (0, 0), n


def test_parameter_and_answer(bpsw):
    rnd = random.Random(3)
    ns = []
    while len(ns) < 4000:
        n = int(2 ** rnd.uniform(33.1, 63.999)) | 1
        if not small_factor(n):
            ns.append(n)
    for n, (p, base2, lucas) in zip(ns, bpsw(ns)):
        assert p == parameter(n) and base2 == strong(n, 2), n
        assert (base2 and lucas) == is_prime(n), n
