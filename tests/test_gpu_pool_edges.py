"""Pooled lookup at the sizes where the kernel's shapes change, bit for bit against the sequential
fp32 oracle (each output element is one chain of additions in key order, so there is no tolerance)."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# rows of one and three 16-byte pieces (several lane groups a warp), of one column, of ten and of
# twelve columns of 4-byte pieces (two CTAs a tile)
@pytest.mark.parametrize("dim,dtype", [(4, "float32"), (24, "float16"), (64, "float16"), (320, "float32"), (384, "float32")])
@pytest.mark.parametrize("piece", [0, 4, 16])
def test_pool_edges(built_lib, dim, dtype, piece):
    from ugache_b200 import runtime as rt, workload as wl
    N, n = 5000, 6000
    dt = np.dtype(dtype)
    table = wl.table(3, N, dim, dt)
    ids, freqs = wl.analytic_hotness(N, 1.1)
    cache = rt.Cache(1, N, dim * dt.itemsize, 0.5, max_batch=n)
    cache.set_placement(rt.solve_placement("intuitive", 1, ids, freqs, 50.0))
    host = torch.from_numpy(table).pin_memory()
    cache.build(0, 0, host.data_ptr())
    cache.tune(0, pool_vec_bytes=piece)
    keys = wl.zipf_keys(9, n, N, 1.1)
    keys[[0, 70, n - 1]] = -1, N, N + 7
    k = torch.from_numpy(keys).cuda()
    lists = {
        "one": [0, n],                                                     # one bag, many chunks of keys
        "edges": np.cumsum([0, 63, 64, 65, 1, 0, 7, 8, 9, 127, 128, 129, 255, 256, 257]),
        "empty": np.concatenate([np.zeros(300), [5], np.full(400, 5), [n]]),  # more bags than a tile holds
        "single": np.arange(n + 1),
    }
    for name, off in lists.items():
        off = np.asarray(off, dtype=np.int64)
        for mode in ("sum", "mean"):
            got = cache.lookup_pool(0, k, offsets=torch.from_numpy(off).cuda(), elem="f16" if dt.itemsize == 2 else "f32",
                                    mode=mode).cpu().numpy()
            want = orc.pool(table, keys, offsets=off, mean=mode == "mean")
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (name, mode)
    assert cache.stats(0)["err_key_range"] > 0
    cache.close()


@pytest.mark.parametrize("piece", [4, 16])
def test_pool_over_the_probing_table(built_lib, piece):
    from ugache_b200 import _lib, runtime as rt, workload as wl
    N, dim, n = 50_000, 64, 6000
    table = wl.table(3, N, dim)
    cache = rt.Cache(1, N, dim * 4, 0.05, max_batch=n, table_kind=_lib.TABLE_HASHED)
    cache.set_placement(rt.solve_placement("rep", 1, np.arange(N, dtype=np.uint32), None, 5.0))
    host = torch.from_numpy(table).pin_memory()
    cache.build(0, 0, host.data_ptr())
    cache.tune(0, pool_vec_bytes=piece)
    keys = wl.zipf_keys(9, n, N, 1.1)
    k = torch.from_numpy(keys).cuda()
    off = np.array([0, 0, 5, 700, 701, n], dtype=np.int64)
    for mode in ("sum", "mean"):
        got = cache.lookup_pool(0, k, offsets=torch.from_numpy(off).cuda(), mode=mode).cpu().numpy()
        want = orc.pool(table, keys, offsets=off, mean=mode == "mean")
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    cache.close()
