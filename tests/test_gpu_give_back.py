"""Device memory that the library gives back to a caller's allocator is idle by then, also where a
build or a refresh is refused: such an allocator may hand a block on at once."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


class Pool:
    """Allocator callbacks over torch's caching allocator; notes frees while `stream` is busy."""

    def __init__(self, stream):
        from ugache_b200 import _lib
        self.blocks, self.busy_frees, self.frees, self.stream = {}, [], 0, stream
        self.alloc_cb, self.free_cb = _lib.ALLOC_FN(self._alloc), _lib.FREE_FN(self._free)

    def _alloc(self, nbytes, user):
        t = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        self.blocks[t.data_ptr()] = t
        return t.data_ptr()

    def _free(self, ptr, user):
        idle = self.stream.query()
        self.frees += 1
        t = self.blocks.pop(ptr)
        if not idle:
            self.busy_frees.append(t.numel())


def make_cache(pool, N, row, share):
    from ugache_b200 import _lib, runtime as rt
    cache = rt.Cache(1, N, row, share, max_batch=4096)
    cache.close()
    cache.cfg.alloc, cache.cfg.free = pool.alloc_cb, pool.free_cb
    _lib.check(_lib.lib().ugc_create(C.byref(cache.cfg), C.byref(cache._h)))
    cache._ctx = cache._h.value
    return cache


# 18 M listed keys: 72 MB of lists, which are given back; 2 M: kept for the next refresh
@pytest.mark.parametrize("N", [2_000_000, 20_000_000])
def test_refused_refresh_and_build(built_lib, N):
    from ugache_b200 import _lib, runtime as rt
    row = 4
    table = torch.arange(N, dtype=torch.int32).pin_memory()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    pool = Pool(a)
    ids = np.arange(N, dtype=np.uint32)
    small = rt.solve_placement("rep", 1, ids, None, 10.0)
    moved = rt.solve_placement("rep", 1, ids[::-1].copy(), None, 10.0)
    everything = rt.solve_placement("rep", 1, ids, None, 100.0)

    cache = make_cache(pool, N, row, 0.1)
    cache.set_placement(everything)             # ten times what the slice holds
    with pytest.raises(_lib.UgcError, match="slice holds"):
        cache.build(0, 0, table.data_ptr(), a.cuda_stream)
    assert pool.frees > 0 and not pool.busy_frees and not pool.blocks

    cache.set_placement(small)
    cache.build(0, 0, table.data_ptr(), a.cuda_stream)
    keys = torch.randint(0, N, (4096,), device="cuda")
    torch.cuda.synchronize()
    for _ in range(3):
        cache.refresh_set_placement(everything)
        with pytest.raises(_lib.UgcError, match="slice holds"):
            cache.refresh_evict(0, a.cuda_stream)
        assert a.query()
        for p in (moved, small):                # at once, on another stream
            cache.refresh_all_local(p, [0], b.cuda_stream)
            got = cache.lookup(0, keys).view(torch.int32).view(-1)
            assert torch.equal(got.long(), keys)
            src = cache.table_words(0, torch.arange(N, device="cuda", dtype=torch.int32))
            held = torch.nonzero(src.view(torch.int32) != -1).view(-1).cpu().numpy()
            want = np.nonzero(p.nid_to_block == 0)[0]
            assert np.array_equal(held, want)
    assert not pool.busy_frees
    cache.close()
    assert not pool.blocks
