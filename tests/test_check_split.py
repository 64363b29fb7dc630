"""How the exact checker's words are split over its CTAs (check_split in
goldbach-l0_gb300/csrc/k_check.cu), called in the built library without a GPU:
every split covers its segment in chunks of at most the 501 words a CTA stages
and no more chunks an item than the kernel's counters are asserted for, also in
a batch without words for the checker. Each call runs in a process of its own:
an integer division by zero ends one on x86."""
import os
import random
import subprocess
import sys

import pytest

import gbc
from conftest import ROOT

CALL = """
import ctypes as C, sys
f = C.CDLL(sys.argv[1])._ZN3gbh11check_splitEmmmiPjS0_
f.restype, f.argtypes = None, [C.c_uint64, C.c_uint64, C.c_uint64, C.c_int, C.POINTER(C.c_uint32), C.POINTER(C.c_uint32)]
for q in sys.stdin:
    cw, vbx = C.c_uint32(), C.c_uint32()
    f(*map(int, q.split()), C.byref(cw), C.byref(vbx))
    print(cw.value, vbx.value)
"""
SM, WORDS, WARPS = 152, 501, 16  # multiprocessors; words of a full chunk; warps of a CTA (a word each at least)
MAX_CHUNKS = 18


def splits(queries):
    text = "".join("%d %d %d %d\n" % q for q in queries)
    r = subprocess.run([sys.executable, "-c", CALL, gbc.LIB_PATH], input=text, capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr[-300:])
    return [tuple(map(int, x.split())) for x in r.stdout.splitlines()]


def class_words(evens):
    return (2 * evens - 2) // 960 + 2


def chunks_per_item(evens, cw, vbx):
    """The most chunks an item takes, by the kernel's own division, at either end of its words' range."""
    most = 0
    for words in (max(1, (evens - 1) // 480), class_words(evens)):
        nch = (words - 1) // cw + 1
        most = max([most] + [nch * (b + 1) // vbx - nch * b // vbx for b in range(vbx)])
    return most


@pytest.fixture(scope="module", autouse=True)
def built():
    if not os.path.exists(gbc.LIB_PATH):
        pytest.skip("the library is not built")


@pytest.mark.parametrize("evens", [1, 9999, 32768, 233750000, 2**32])
def test_a_batch_without_words_for_the_checker(evens):
    ((cw, vbx),) = splits([(evens, 0, 2**64 - 1, SM)])
    assert WARPS <= cw <= WORDS and vbx >= 1


def test_every_split_covers_its_segment_in_the_kernel_s_bounds():
    rnd = random.Random(1)
    queries = [(70196 * 480, 2433211, 2**64 - 1, SM)]
    for _ in range(400):
        segs = [rnd.randrange(2, int(2 * 10 ** rnd.uniform(2, 8.67))) // 2 for _ in range(rnd.choice((1, 1, 2, 3, 8, 48, 256)))]
        words = [class_words(e) for e in segs]
        queries += [(e, sum(words), min(words), SM) for e in rnd.sample(segs, min(len(segs), 3))]
    for (evens, *_), (cw, vbx) in zip(queries, splits(queries)):
        assert WARPS <= cw <= WORDS and vbx >= 1
        assert chunks_per_item(evens, cw, vbx) <= MAX_CHUNKS, (evens, cw, vbx)


def test_the_counters_are_asserted_for_the_split_s_bound():
    src = open(os.path.join(ROOT, "goldbach-l0_gb300", "csrc", "k_check.cu")).read()
    assert f"kCkMaxChunks = {MAX_CHUNKS};" in src
    assert "static_assert(kCkMaxChunks * " in src and "m <= gbk::kCkMaxChunks" in src
