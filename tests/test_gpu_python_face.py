"""The Python face's per-step calls: errors are those torch raises for the same thing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# outputs of 16 TB or more: the allocation fails before anything is launched
@pytest.mark.parametrize("call", ["lookup", "unique", "pool"])
def test_out_of_memory(built_lib, call):
    from ugache_b200 import runtime as rt
    table = torch.zeros((1000, 4096), dtype=torch.float32).pin_memory()
    cache = rt.Cache(1, 1000, 4096 * 4, 0.1, max_batch=1024)
    cache.set_placement(rt.solve_placement("rep", 1, np.arange(1000, dtype=np.uint32), None, 10.0))
    cache.build(0, 0, table.data_ptr())
    keys = torch.zeros(1, dtype=torch.int64, device="cuda").expand(1 << 30)   # one element in memory
    with pytest.raises(torch.OutOfMemoryError):
        if call == "lookup":
            cache.lookup(0, keys)
        elif call == "unique":
            cache.lookup_unique(0, keys)
        else:
            cache.lookup_pool(0, keys, bag_size=1)
    assert cache.lookup(0, torch.zeros(8, dtype=torch.int64, device="cuda")).numel() == 8 * 4096 * 4  # and goes on
    cache.close()
