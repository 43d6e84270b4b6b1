"""Host-buffer lookups on both sides of the line between rows written in place and rows staged: the
rows are copies, so they are equal or wrong, and nothing beyond them is touched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# 512-byte rows: 4 MB are 8192 keys; 200-byte rows, or 512-byte ones in a buffer 4 bytes off: 512 KB
# are 2621 and 1024
@pytest.mark.parametrize("dim,shift,ns", [(128, 0, [1, 8192, 8193]), (50, 0, [1, 2621, 2622]), (128, 4, [1, 1024, 1025])])
@pytest.mark.parametrize("key_dtype", [np.int64, np.uint32])
def test_host_lookup_edges(built_lib, dim, shift, ns, key_dtype):
    from ugache_b200 import runtime as rt, workload as wl
    N, row = 20000, dim * 4
    table = wl.table(2, N, dim)
    ids, freqs = wl.analytic_hotness(N, 1.1)
    cache = rt.Cache(1, N, row, 0.5, max_batch=1 << 14)
    cache.set_placement(rt.solve_placement("intuitive", 1, ids, freqs, 50.0))
    host = torch.from_numpy(table).pin_memory()
    cache.build(0, 0, host.data_ptr())
    stream = torch.cuda.current_stream().cuda_stream
    for n in ns:
        keys = wl.zipf_keys(n, n, N, 1.1).astype(key_dtype)
        k = torch.from_numpy(keys.view(np.int64 if key_dtype == np.int64 else np.int32)).pin_memory()
        out = torch.full((shift + n * row + 64,), 7, dtype=torch.uint8).pin_memory()
        for keys_ptr in (k.data_ptr(), keys.ctypes.data):     # pinned and pageable keys
            out.fill_(7)
            cache.lookup_host_ptr(0, keys_ptr, keys.itemsize, n, out.data_ptr() + shift, stream)
            got = out.numpy()
            assert np.array_equal(got[shift:shift + n * row].view(np.uint8).reshape(n, row),
                                  table[keys.astype(np.int64)].view(np.uint8).reshape(n, row)), n
            assert (got[:shift] == 7).all() and (got[shift + n * row:] == 7).all()
    cache.close()


# fp16 rows at an odd element, and at odd bytes: the kernels store 4-byte words, so these are staged
@pytest.mark.parametrize("shift", [1, 2, 3, 6])
@pytest.mark.parametrize("zero_copy", [1, 3])
def test_host_rows_at_any_byte(built_lib, shift, zero_copy):
    from ugache_b200 import runtime as rt, workload as wl
    N, dim, n = 5000, 50, 300
    row = dim * 2
    table = wl.table(4, N, dim, np.dtype(np.float16))
    ids, freqs = wl.analytic_hotness(N, 1.1)
    cache = rt.Cache(1, N, row, 0.5, max_batch=1024)
    cache.set_placement(rt.solve_placement("intuitive", 1, ids, freqs, 50.0))
    host = torch.from_numpy(table).pin_memory()
    cache.build(0, 0, host.data_ptr())
    cache.tune(0, host_zero_copy=zero_copy)
    keys = torch.from_numpy(wl.zipf_keys(3, n, N, 1.1)).pin_memory()
    out = torch.full((shift + n * row + 64,), 7, dtype=torch.uint8).pin_memory()
    cache.lookup_host_ptr(0, keys.data_ptr(), 8, n, out.data_ptr() + shift, torch.cuda.current_stream().cuda_stream)
    got = out.numpy()
    assert got[shift:shift + n * row].tobytes() == table[keys.numpy()].tobytes()
    assert (got[:shift] == 7).all() and (got[shift + n * row:] == 7).all()
    cache.close()


def test_an_error_is_reported_once(built_lib):
    """CUDA refuses to copy to a buffer that is pinned in part; the calls after that one succeed."""
    import ctypes as C
    import mmap

    from ugache_b200 import _lib, runtime as rt
    N, dim, page = 5000, 32, 4096
    table = np.arange(N * dim, dtype=np.float32).reshape(N, dim)
    host = torch.from_numpy(table).pin_memory()
    keys = torch.arange(200).pin_memory()
    area = mmap.mmap(-1, 8 * page)
    base = C.addressof(C.c_char.from_buffer(area))
    stream = torch.cuda.current_stream().cuda_stream
    cudart = torch.cuda.cudart()
    assert int(cudart.cudaHostRegister(base, page, 0)) == 0
    for _ in range(2):
        cache = rt.Cache(1, N, dim * 4, 0.5, max_batch=1024)
        cache.set_placement(rt.solve_placement("rep", 1, np.arange(N, dtype=np.uint32), None, 50.0))
        cache.build(0, 0, host.data_ptr())
        cache.tune(0, host_zero_copy=0)
        with pytest.raises(_lib.UgcError, match="cudaMemcpyAsync"):
            cache.lookup_host_ptr(0, keys.data_ptr(), 8, 200, base, stream)
        cache.record(0, keys.cuda())
        assert cache.hotness_read(0, stream=stream).sum() == 200
        cache.close()
    cudart.cudaHostUnregister(base)

# Buffers pinned at both ends with a pageable hole between, and at the start only, are not used in place
# (CUDA refuses to copy them); ones pinned in two pieces are
@pytest.mark.parametrize("pinned,whole", [(((0, 1), (6, 8)), False), (((0, 3),), False), (((0, 4), (4, 8)), True)])
@pytest.mark.parametrize("zero_copy", [1, 3])
def test_host_buffers_pinned_in_part(built_lib, pinned, whole, zero_copy):
    import ctypes as C
    import mmap

    from ugache_b200 import _lib, runtime as rt, workload as wl
    N, dim, page = 5000, 32, 4096
    row, n = dim * 4, 8 * page // (dim * 4)
    table = wl.table(4, N, dim)
    ids, freqs = wl.analytic_hotness(N, 1.1)
    cache = rt.Cache(1, N, row, 0.5, max_batch=8192)
    cache.set_placement(rt.solve_placement("intuitive", 1, ids, freqs, 50.0))
    host = torch.from_numpy(table).pin_memory()
    cache.build(0, 0, host.data_ptr())
    cache.tune(0, host_zero_copy=zero_copy)
    areas = [mmap.mmap(-1, 8 * page) for _ in range(2)]
    base = [C.addressof(C.c_char.from_buffer(m)) for m in areas]
    cudart = torch.cuda.cudart()
    for b in base:
        for lo, hi in pinned:
            assert int(cudart.cudaHostRegister(b + lo * page, (hi - lo) * page, 0)) == 0
    stream = torch.cuda.current_stream().cuda_stream
    area, key_area = (np.frombuffer(m, dtype=np.uint8) for m in areas)
    k = wl.zipf_keys(3, 8 * page // 8, N, 1.1)
    key_area.view(np.int64)[:] = k
    own_keys = torch.from_numpy(k).pin_memory()
    own_out = torch.zeros((len(k), dim)).pin_memory()
    calls = [(own_keys.data_ptr(), n, base[0], area), (base[1], len(k), own_out.data_ptr(), own_out.numpy())]
    for keys_ptr, count, out_ptr, out in calls:      # as many rows, or keys, as the area holds
        if whole:
            cache.lookup_host_ptr(0, keys_ptr, 8, count, out_ptr, stream)
            assert out.tobytes() == table[k[:count]].tobytes()
        else:
            with pytest.raises(_lib.UgcError):
                cache.lookup_host_ptr(0, keys_ptr, 8, count, out_ptr, stream)
    cache.lookup_host_ptr(0, own_keys.data_ptr(), 8, len(k), own_out.data_ptr(), stream)
    assert own_out.numpy().tobytes() == table[k].tobytes()
    for b in base:
        for lo, hi in pinned:
            cudart.cudaHostUnregister(b + lo * page)
    cache.close()


# Keys at an address that is not a multiple of their size are staged
@pytest.mark.parametrize("key_bytes,shift", [(8, 1), (8, 4), (4, 1), (4, 2)])
def test_host_keys_at_any_byte(built_lib, key_bytes, shift):
    from ugache_b200 import runtime as rt
    N, dim, n = 5000, 32, 300
    table = np.arange(N * dim, dtype=np.float32).reshape(N, dim)
    cache = rt.Cache(1, N, dim * 4, 0.5, max_batch=1024)
    cache.set_placement(rt.solve_placement("rep", 1, np.arange(N, dtype=np.uint32), None, 50.0))
    host = torch.from_numpy(table).pin_memory()
    cache.build(0, 0, host.data_ptr())
    keys = np.random.default_rng(1).integers(0, N, n).astype(np.int64 if key_bytes == 8 else np.int32)
    raw = torch.zeros(shift + keys.nbytes, dtype=torch.uint8).pin_memory()
    raw.numpy()[shift:] = keys.view(np.uint8)
    out = torch.zeros((n, dim)).pin_memory()
    cache.lookup_host_ptr(0, raw.data_ptr() + shift, key_bytes, n, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert np.array_equal(out.numpy(), table[keys])
    cache.close()
