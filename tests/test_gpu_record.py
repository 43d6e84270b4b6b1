"""Hotness counters on the GPU (ugc_record, ugc_hotness_read) against a host bincount, at the sizes
where the kernel's shapes change.  Whole numbers: equal or wrong."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# 1024 keys a CTA, 32 a warp; read-out parts of 131,072 counters.  "one" = every key the same id,
# "few" = 5 ids, "wide" = about as many ids as keys, so that the CTA's counters collide
@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024, 1025, 100_003])
@pytest.mark.parametrize("spread", ["one", "few", "wide"])
@pytest.mark.parametrize("N", [1000, 131_072, 300_001])
def test_counts_match_bincount(built_lib, n, spread, N):
    from ugache_b200 import runtime as rt
    table = torch.zeros((N, 4), dtype=torch.float32).pin_memory()
    cache = rt.Cache(1, N, 16, 0.1, max_batch=1024)
    cache.set_placement(rt.solve_placement("rep", 1, np.arange(N, dtype=np.uint32), None, 10.0))
    cache.build(0, 0, table.data_ptr())
    r = np.random.default_rng(n)
    hi = {"one": 1, "few": 5, "wide": N}[spread]
    keys = (N - 1 - r.integers(0, hi, n)).astype(np.int64)
    want = np.bincount(keys, minlength=N) + np.bincount(keys, minlength=N)
    k = torch.from_numpy(keys).cuda()
    cache.record(0, k)
    cache.record(0, k.to(torch.int32))
    out_of_range = torch.tensor([-1, N, 1 << 40], device="cuda")
    cache.record(0, out_of_range)                       # counts nothing
    stream = torch.cuda.current_stream().cuda_stream
    assert np.array_equal(cache.hotness_read(0, reset=True, stream=stream), want)
    assert not cache.hotness_read(0, stream=stream).any()
    cache.close()
