"""Launches of one stream that overlap see what the ones before them wrote: calls are enqueued without a
synchronisation in between, all outputs are kept and compared at the end, byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def build(table, share, max_batch, table_kind=0):
    from ugache_b200 import runtime as rt
    N = len(table)
    row = table.nbytes // N
    cache = rt.Cache(1, N, row, share, max_batch=max_batch, table_kind=table_kind)
    cache.set_placement(rt.solve_placement("rep", 1, np.arange(N, dtype=np.uint32), None, share * 100.0))
    host = torch.from_numpy(table.view(np.uint8).reshape(N, row)).pin_memory()
    cache.build(0, 0, host.data_ptr())
    cache._keep.append(host)
    return cache


# Rows of one lookup are the keys of the next, in one cache and across two on the same stream, with a
# long extraction ahead; batches of one CTA, of one wave and of several
@pytest.mark.parametrize("mode", ["direct", "grouped"])
@pytest.mark.parametrize("n", [200, 13_000, 300_000])
def test_rows_are_the_next_keys(built_lib, mode, n):
    from ugache_b200 import _lib
    N = 400_000
    r = np.random.default_rng(n)
    steps = [r.permutation(N).astype(np.int64) for _ in range(2)]
    caches = [build(t, 0.9, n) for t in steps]
    for c in caches:
        c.tune(0, extract_mode=_lib.EXTRACT_DIRECT if mode == "direct" else _lib.EXTRACT_GROUPED)
    batches = [r.integers(0, N, n) for _ in range(3)]
    keys = [torch.from_numpy(b).cuda() for b in batches]
    torch.cuda.synchronize()
    got, want = [], []
    for it in range(30):
        k, w = keys[it % 3], batches[it % 3]
        for hop in range(4):
            which = (it >> hop) & 1          # both caches, in changing order, also one after itself
            k = caches[which].lookup(0, k).view(torch.int64).view(-1)
            w = steps[which][w]
        got.append(k)
        want.append(w)
    for g, w in zip(got, want):
        assert np.array_equal(g.cpu().numpy(), w)
    for c in caches:
        c.close()


# The key buffer is written by an ordinary kernel right ahead of each lookup, and the host table by a copy
@pytest.mark.parametrize("mode", ["auto", "direct", "grouped"])
@pytest.mark.parametrize("n", [200, 13_000])
def test_keys_written_just_ahead(built_lib, mode, n):
    from ugache_b200 import _lib
    N, dim = 200_000, 32
    r = np.random.default_rng(n)
    table = r.integers(0, 1 << 30, (N, dim)).astype(np.int32)
    cache = build(table, 0.9, n)
    cache.tune(0, extract_mode={"auto": 0, "direct": _lib.EXTRACT_DIRECT, "grouped": _lib.EXTRACT_GROUPED}[mode])
    batches = [r.integers(0, N, n) for _ in range(8)]
    source = [torch.from_numpy(b).cuda() for b in batches]
    keys = torch.empty(n, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    got = []
    for it in range(64):
        torch.add(source[it % 8], 0, out=keys)
        got.append(cache.lookup(0, keys))
        if it % 3 == 0:                      # and once with the lookup's own output as the one ahead
            got[-1] = cache.lookup(0, keys, out=got[-1])
    for it, g in enumerate(got):
        assert np.array_equal(g.view(torch.int32).cpu().numpy(), table[batches[it % 8]])
    cache.close()


# Every kind of call, in changing order and size, over the flat and the probing table
@pytest.mark.parametrize("kind", ["flat", "hashed"])
def test_mixed_calls(built_lib, kind):
    from oracle import oracle as orc
    from ugache_b200 import _lib
    N, dim, big = 60_000, 16, 40_000
    r = np.random.default_rng(7)
    table = r.standard_normal((N, dim)).astype(np.float32)
    cache = build(table, 0.4, big, _lib.TABLE_FLAT if kind == "flat" else _lib.TABLE_HASHED)
    cache.tune(0, host_order_min_rows=100)   # the grouped lookups order their host rows
    calls, recorded = [], np.zeros(N, dtype=np.int64)
    ops = ["unique", "direct", "pool", "record", "grouped"]
    plan = []
    for it in range(60):
        n = int(r.choice([1, 33, 1025, 7000, big]))
        plan.append((ops[int(r.integers(0, 5))], torch.from_numpy(r.integers(0, N, n)).cuda()))
    torch.cuda.synchronize()
    for op, k in plan:
        if op in ("direct", "grouped"):
            cache.tune(0, extract_mode=_lib.EXTRACT_DIRECT if op == "direct" else _lib.EXTRACT_GROUPED)
            calls.append(cache.lookup(0, k))
        elif op == "unique":
            rows, uniq, inverse, nu = cache.lookup_unique(0, k)
            calls.append((rows, uniq, inverse, nu, cache.lookup(0, inverse)))
        elif op == "pool":
            calls.append(cache.lookup_pool(0, k, bag_size=1 + k.numel() // 50))
        else:
            calls.append(cache.record(0, k))
    for (op, k), got in zip(plan, calls):
        k = k.cpu().numpy()
        if op in ("direct", "grouped"):
            assert np.array_equal(got.view(torch.float32).cpu().numpy(), table[k])
        elif op == "unique":
            rows, uniq, inverse, nu, again = got
            nu, inverse = int(nu), inverse.cpu().numpy()
            assert nu == len(np.unique(k)) and np.array_equal(uniq.cpu().numpy()[:nu][inverse], k)
            assert np.array_equal(rows.view(torch.float32).cpu().numpy()[:nu][inverse], table[k])
            assert np.array_equal(again.view(torch.float32).cpu().numpy(), table[inverse])
        elif op == "pool":
            want = orc.pool(table, k, bag_size=1 + len(k) // 50, mean=False)
            assert np.array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32))
        else:
            recorded += np.bincount(k, minlength=N)
    assert np.array_equal(cache.hotness_read(0, stream=torch.cuda.current_stream().cuda_stream), recorded)
    assert cache.stats(0)["err_key_range"] == 0
    cache.close()


# The same chains captured into a graph and launched on new keys
@pytest.mark.parametrize("mode", ["direct", "grouped"])
def test_captured_chain(built_lib, mode):
    from ugache_b200 import _lib
    N, n = 100_000, 5000
    r = np.random.default_rng(1)
    step = r.permutation(N).astype(np.int64)
    cache = build(step, 0.9, n)
    cache.tune(0, extract_mode=_lib.EXTRACT_DIRECT if mode == "direct" else _lib.EXTRACT_GROUPED)
    keys = torch.zeros(n, dtype=torch.int64, device="cuda")
    other = torch.randint(0, N, (n,), device="cuda")
    cache.lookup(0, keys)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        a = cache.lookup(0, keys)
        b = cache.lookup(0, other)               # beside the first one
        c = cache.lookup(0, a.view(torch.int64).view(-1))
        k = c.view(torch.int64).view(-1) + 1     # an ordinary kernel between two lookups
        d = cache.lookup(0, k.clamp_(max=N - 1))
    batches = [r.integers(0, N, n) for _ in range(10)]
    got = []
    for batch in batches:
        keys.copy_(torch.from_numpy(batch).pin_memory(), non_blocking=True)
        g.replay()
        got.append([x.clone() for x in (a, b, c, d)])
        cache.lookup(0, other)
    o = other.cpu().numpy()
    for batch, outs in zip(batches, got):
        second = step[step[batch]]
        want = (step[batch], step[o], second, step[np.minimum(second + 1, N - 1)])
        for x, w in zip(outs, want):
            assert np.array_equal(x.view(torch.int64).view(-1).cpu().numpy(), w)
    cache.close()
