"""Figures of the bench line that it works out from the library's counters."""
import types


def test_sparse_entries_per_warp_task():
    """A warp's task of the sparse checker is 8192 evens of a class; the
    library counts the plan entries that it takes word by word."""
    import bench

    class Sparse:
        def __init__(self, **kw):
            pass

        def __enter__(self):
            return self

        def __exit__(self, *a):
            pass

        def verify(self, a, b):
            return types.SimpleNamespace(evens=8192 * 1000, groups=3030, segments=2, pending=0, map_primes=1,
                                         ms_sieve=1.0, ms_large=1.0, ms_check=1.0, ms_total=4.0)
    out = bench.sparse_leg(types.SimpleNamespace(Sparse=Sparse))
    assert out["word_entries_per_warp_task"] == 3.03 and "entries_per_warp_task" not in out
