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


@pytest.mark.parametrize("call", ["record", "lookup", "unique", "pool"])
@pytest.mark.parametrize("programmatic", [0, 3])
def test_programmatic_launch_is_a_choice(built_lib, call, programmatic):
    """The edge between two launches of a captured stream is programmatic only where the tuning says so."""
    import ctypes as C

    from ugache_b200 import _lib, runtime as rt
    table = torch.zeros((1000, 32)).pin_memory()
    cache = rt.Cache(1, 1000, 128, 0.1, max_batch=1024)
    cache.set_placement(rt.solve_placement("rep", 1, np.arange(1000, dtype=np.uint32), None, 10.0))
    cache.build(0, 0, table.data_ptr())
    cache.tune(0, programmatic_launch=programmatic, extract_mode=_lib.EXTRACT_DIRECT)
    keys = torch.arange(100, device="cuda")
    run = {"record": lambda: cache.record(0, keys), "lookup": lambda: cache.lookup(0, keys),
           "unique": lambda: cache.lookup_unique(0, keys), "pool": lambda: cache.lookup_pool(0, keys, bag_size=10)}[call]
    run()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        run()
        run()
    edges = C.CDLL("libcuda.so.1").cuGraphGetEdges_v2
    n = C.c_size_t(0)
    graph = C.c_void_p(g.raw_cuda_graph())
    assert edges(graph, None, None, None, C.byref(n)) == 0 and n.value > 0
    ends, data = ((C.c_void_p * n.value)(), (C.c_void_p * n.value)()), (C.c_uint8 * (8 * n.value))()
    assert edges(graph, ends[0], ends[1], data, C.byref(n)) == 0
    kinds = [data[8 * i + 2] for i in range(n.value)]        # from port, to port, type, reserved
    assert any(kinds) == (programmatic != 0), kinds
    cache.close()
