"""How the exact checker's words are split over its CTAs (GPU): one, two or
three equal items per CTA or many of 16 chunks, alone or beside small
segments. Each segment's statistics are those of the same evens cut into many
small segments (or, for whole batches, of the segment alone)."""
import numpy as np
import pytest

import gbc

pytestmark = pytest.mark.gpu
SEG = gbc.DEFAULT_SEGMENT


def run(c, segs):
    c.enqueue_segments(0, segs, [max(b for _, b in segs)] * len(segs))
    return c.collect(0, len(segs))[0]


def fields(r):
    return np.array(r.hist), np.array(r.first), r.nleft


@pytest.mark.parametrize("height,width", [
    (10**12, 4_650_000),        # below 16 words a CTA
    (10**12, 4_700_000),        # from there on as many items as CTAs
    (10**12 + 2, 146_000_002),  # a chunk a CTA, and two
    (10**12, 147_000_000),
    (4 * 10**18, 300_000_014),
])
def test_one_segment_against_its_pieces(height, width):
    step = width // 47 // 2 * 2
    parts = [(a, min(a + step - 2, height + width)) for a in range(height, height + width + 1, step)]
    with gbc.Context(limit=height + 2 * width, max_batch=len(parts), max_runs=len(parts)) as c:
        whole = run(c, [(height, height + width)])[0]
        pieces = run(c, parts)
    hist, first, nleft = fields(whole)
    assert np.array_equal(hist, sum(np.array(p.hist) for p in pieces)) and hist.sum() + nleft == width // 2 + 1
    assert nleft == sum(p.nleft for p in pieces)
    want = np.full(len(first), 0xFFFFFFFF, dtype=np.uint32)
    for (a, _), p in zip(parts, pieces):
        f = np.array(p.first)
        seen = f != 0xFFFFFFFF
        want[seen] = np.minimum(want[seen], f[seen] + (a - height) // 2)
    assert np.array_equal(first, want)


@pytest.mark.parametrize("n", [5, 11, 16])  # two and three items per CTA, and items of 16 chunks
def test_batch_against_its_segments(n):
    segs = [(10**12 + i * SEG, 10**12 + (i + 1) * SEG - 2) for i in range(n)]
    with gbc.Context(limit=10**12 + 20 * SEG, max_batch=16) as c:
        together = run(c, segs)
        for s, r in zip(segs, together):
            for x, y in zip(fields(r), fields(run(c, [s])[0])):
                assert np.array_equal(x, y)


def test_large_segments_beside_small_ones():
    h = 10**12
    segs = [(h, h + 400_000_000), (h + 10**10, h + 10**10 + 20_000), (h + 2 * 10**10, h + 2 * 10**10 + 460_000_000),
            (h + 3 * 10**10, h + 3 * 10**10 + 2), (h + 4 * 10**10, h + 4 * 10**10 + 30_000_000)]
    with gbc.Context(limit=h + 5 * 10**10, max_batch=8) as c:
        together = run(c, segs)
        for s, r in zip(segs, together):
            for x, y in zip(fields(r), fields(run(c, [s])[0])):
                assert np.array_equal(x, y)
