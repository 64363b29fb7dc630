"""A verify plan of fewer than five funnels (GPU), which lacks some of the word
form's: the batch's statistics at the edges of words are the plan's
(test_gpu_verify_edges); here that its words are taken word by word too, by its
device time against a plan of five funnels, which holds the word form's."""
import pytest

import gbc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("height", [10**12, 4 * 10**18])
def test_time_of_small_plans(height):
    seg = (height, height + 20_000_000 - 2)

    def batch(funnels):
        with gbc.Context(limit=seg[1], max_batch=1, plan_funnels=funnels) as c:
            best = 1e9
            for _ in range(6):
                c.enqueue_batch(0, [seg], seg[1], [gbc.SEG_VERIFY])
                (s,), t = c.collect(0, 1)
                best = min(best, t.ms_check)
            return best, (s.map_hash, s.evens)
    (t5, want), (t4, got4), (t3, got3) = batch(5), batch(4), batch(3)
    assert got3 == got4 == want
    # two or three funnels by their members cost two to three times the compiled ones; even by even 20 times
    assert t4 < 6 * t5 and t3 < 8 * t5, (t3, t4, t5)
