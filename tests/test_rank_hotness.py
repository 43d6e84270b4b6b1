"""Hotness ranking (ugc_rank_hotness): ids by descending count, ties by ascending id, against
numpy's stable sort.  Whole numbers: equal or wrong."""
import numpy as np
import pytest


# sizes around one thread's share (32768 ids) and value ranges around the digit widths: one pass up
# to 11 bits, two up to 22, three beyond; a constant array and a single huge count among zeros
@pytest.mark.parametrize("n", [0, 1, 2, 32767, 32768, 32769, 300_001])
@pytest.mark.parametrize("bits", [0, 1, 11, 12, 22, 23, 32])
def test_rank_matches_stable_sort(built_lib, n, bits):
    from ugache_b200 import runtime as rt
    counts = np.random.default_rng(n + bits).integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    if n > 2 and bits == 1:
        counts[:] = 0
        counts[n // 2] = 0xFFFFFFFF
    ids, freqs = rt.Cache.rank_hotness(counts)
    want = np.argsort(-counts.astype(np.int64), kind="stable").astype(np.uint32)
    assert np.array_equal(ids, want) and np.array_equal(freqs, counts[want])


def test_more_ids_than_the_library_ranks(built_lib, monkeypatch):
    """Longer arrays go through numpy, with the same result."""
    from ugache_b200 import runtime as rt
    counts = np.array([3, 0, 7, 3, 7, 1], dtype=np.uint32)
    want = rt.Cache.rank_hotness(counts)
    monkeypatch.setattr(rt, "_RANK_MAX", 5)
    monkeypatch.setattr(rt._lib, "lib", lambda: pytest.fail("the library refuses these"))
    for a, b in zip(rt.Cache.rank_hotness(counts), want):
        assert a.dtype == b.dtype and np.array_equal(a, b)
