"""The rules that pick a load width, a path and a number of CTAs: whatever they pick, rows are equal or wrong."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def build(table, share, max_batch, **kw):
    from ugache_b200 import runtime as rt
    N, row = len(table), table.nbytes // len(table)
    cache = rt.Cache(1, N, row, share, max_batch=max_batch, **kw)
    cache.set_placement(rt.solve_placement("rep", 1, np.arange(N, dtype=np.uint32), None, share * 100.0))
    host = torch.from_numpy(table.view(np.uint8).reshape(N, row)).pin_memory()
    cache.build(0, 0, host.data_ptr())
    cache._keep.append(host)
    return cache


@pytest.mark.parametrize("kind", [1, 2])           # direct-index and probing table
def test_load_width_is_a_choice_again(built_lib, kind):
    from ugache_b200 import _lib
    table = np.random.default_rng(1).integers(0, 1 << 30, (20_000, 32)).astype(np.int32)
    cache = build(table, 0.2, 8192, table_kind=kind)
    assert cache.get_tuning(0)["gather_vec_bytes"] == 16
    keys = torch.randint(0, 20_000, (8000,), device="cuda")
    want = table[keys.cpu().numpy()]
    for vec in (16, 32):
        for mode in (_lib.EXTRACT_DIRECT, _lib.EXTRACT_GROUPED):
            for early in (1, 2):
                cache.tune(0, gather_vec_bytes=vec, extract_mode=mode, direct_early_host=early)
                assert cache.get_tuning(0)["gather_vec_bytes"] == vec
                for _ in range(2):
                    got = cache.lookup(0, keys).view(torch.int32).cpu().numpy()
                    assert np.array_equal(got, want), (vec, mode)
    with pytest.raises(_lib.UgcError):
        cache.tune(0, gather_vec_bytes=8)
    cache.close()
    wide = build(table, 0.2, 8192, gather_vec_bytes=32)
    assert wide.get_tuning(0)["gather_vec_bytes"] == 32
    wide.close()


# rows of more than 128 bytes over at most 1.5 GB go grouped from 4096 host rows on, others from 8192
@pytest.mark.parametrize("row,nbytes,line", [(512, 1 << 26, 4096), (128, 1 << 26, 8192), (132, 1 << 26, 4096),
                                             (512, 3 << 29, 4096), (512, (3 << 29) + 512, 8192)])
def test_line_between_direct_and_grouped(built_lib, row, nbytes, line):
    from ugache_b200 import runtime as rt
    N = nbytes // row
    host, _ = rt.host_alloc(N * row)
    cache = rt.Cache(1, N, row, 0.001, max_batch=1024)
    cache.set_placement(rt.solve_placement("rep", 1, np.arange(N, dtype=np.uint32), None, 0.1))
    cache.build(0, 0, host)
    assert cache.get_tuning(0)["direct_max_host_rows"] == line
    cache.close()
    rt.host_free(host)


# host lists in address order: rows that move in 4-byte pieces, in odd numbers of 16-byte ones, in whole
# ones; with and without rows in the slice
@pytest.mark.parametrize("dim", [1, 25, 50, 100, 128, 256])
@pytest.mark.parametrize("share", [0.0, 0.3])
def test_ordered_host_lists(built_lib, dim, share):
    from ugache_b200 import _lib
    N, n = 30_000, 20_000
    table = np.random.default_rng(dim).integers(0, 1 << 30, (N, dim)).astype(np.int32)
    cache = build(table, share, n)
    cache.tune(0, extract_mode=_lib.EXTRACT_GROUPED, host_order_min_rows=1)
    batches = [torch.randint(0, N, (k,), device="cuda") for k in (n, 1, n - 7, 33)]
    cache.lookup(0, batches[0])
    torch.cuda.synchronize()                   # from here on the last lookup's host rows are known
    got = [cache.lookup(0, k) for k in batches * 3]
    for k, g in zip(batches * 3, got):
        assert np.array_equal(g.view(torch.int32).cpu().numpy(), table[k.cpu().numpy()])
    assert cache.stats(0)["lookups_host_ordered"] > 0
    cache.close()
