"""The process' staging block: whoever holds it waits for its own copies, never for a caller's stream."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def make_cache(N):
    from ugache_b200 import runtime as rt
    table = torch.arange(N * 4, dtype=torch.float32).view(N, 4).pin_memory()
    cache = rt.Cache(1, N, 16, 0.1, max_batch=1024)
    ids = np.arange(N, dtype=np.uint32)
    first = rt.solve_placement("rep", 1, ids, None, 10.0)
    cache.set_placement(first)
    cache.build(0, 0, table.data_ptr())
    cache._keep.append(table)
    return cache, [first, rt.solve_placement("rep", 1, ids[::-1].copy(), None, 10.0)]


@pytest.mark.parametrize("slow", ["read", "refresh"])
@pytest.mark.parametrize("quick", ["read", "refresh"])
def test_a_busy_stream_holds_nobody_up(built_lib, slow, quick):
    N = 300_000
    caches = [make_cache(N) for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    keys = torch.arange(1000, device="cuda")
    counts = [None, None]

    def step(i, what):
        cache, placements = caches[i]
        if what == "read":
            counts[i] = cache.hotness_read(0, reset=True, stream=streams[i].cuda_stream)
        else:
            cache.refresh_all_local(placements.pop(), [0], streams[i].cuda_stream)

    for i in range(2):                       # first use makes the block, the streams, counters and lists
        caches[i][0].record(0, keys, stream=streams[i].cuda_stream)
        step(i, "read")
        step(i, "refresh")
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        torch.cuda._sleep(int(1.2e9))        # 0.6 s and more, at any clock of the card
        caches[0][0].record(0, keys)
    busy = threading.Thread(target=step, args=(0, slow))
    t0 = time.perf_counter()
    busy.start()
    time.sleep(0.1)
    caches[1][0].record(0, keys, stream=streams[1].cuda_stream)
    step(1, quick)
    took = time.perf_counter() - t0
    assert not streams[0].query(), "the first stream was to be busy all the time"
    busy.join()
    assert took < 0.4, took
    for i, what in ((0, slow), (1, quick)):
        if what == "read":
            assert counts[i][:1000].tolist() == [1] * 1000 and counts[i].sum() == 1000
        got = caches[i][0].lookup(0, keys).view(torch.float32)
        assert torch.equal(got.cpu(), torch.arange(4000, dtype=torch.float32).view(1000, 4))
    for cache, _ in caches:
        cache.close()
