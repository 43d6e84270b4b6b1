"""Deduplicated lookup at the sizes where its kernels' shapes change: the distinct ids, the index of
every key and the rows are exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# 1024 keys a claim CTA; 592 extraction CTAs write two indices a thread before their rows (303,104
# keys) and the rest after them; tiles of 4 to 32 keys by the number found
@pytest.mark.parametrize("n", [1, 1023, 1025, 30_000, 303_105])
@pytest.mark.parametrize("spread", ["one", "few", "wide"])
def test_unique_edges(built_lib, n, spread):
    from ugache_b200 import runtime as rt, workload as wl
    N, dim = 400_000, 4
    table = wl.table(5, N, dim)
    ids, freqs = wl.analytic_hotness(N, 1.2)
    cache = rt.Cache(1, N, dim * 4, 0.5, max_batch=n)
    cache.set_placement(rt.solve_placement("intuitive", 1, ids, freqs, 50.0))
    host = torch.from_numpy(table).pin_memory()
    cache.build(0, 0, host.data_ptr())
    rows_of = torch.from_numpy(table).cuda()
    r = np.random.default_rng(n)
    hi = {"one": 1, "few": 3000, "wide": N}[spread]
    calls = 260 if n <= 1025 else 3   # past the last epoch of the stamps where that is quick
    for it in range(calls):
        k = torch.from_numpy((N - 1 - r.integers(0, hi, n)).astype(np.int64)).cuda()
        kk = k if it % 2 else k.to(torch.int32)
        rows, uniq, inverse, n_unique = cache.lookup_unique(0, kk)
        # the index is the next launch's keys: it must be complete by then
        again = cache.lookup(0, inverse).view(torch.float32)
        nu = int(n_unique)
        assert nu == int(torch.unique(k).numel())
        assert torch.equal(uniq[:nu][inverse.long()].long(), k)
        assert torch.equal(rows.view(torch.float32)[:nu][inverse.long()], rows_of[k])
        assert torch.equal(again, rows_of[inverse.long()])
    cache.close()


def test_capture_between_calls(built_lib):
    """Calls captured into graphs -- never launched, launched once, launched again on other keys -- and
    ordinary calls between them, over the turn of the epochs."""
    from ugache_b200 import runtime as rt, workload as wl
    N, dim, n = 50_000, 4, 3000
    table = wl.table(6, N, dim)
    ids, freqs = wl.analytic_hotness(N, 1.2)
    cache = rt.Cache(1, N, dim * 4, 0.5, max_batch=n)
    cache.set_placement(rt.solve_placement("intuitive", 1, ids, freqs, 50.0))
    host = torch.from_numpy(table).pin_memory()
    cache.build(0, 0, host.data_ptr())
    rows_of = torch.from_numpy(table).cuda()
    r = np.random.default_rng(3)
    draw = lambda: torch.from_numpy(r.integers(0, N, n)).cuda()

    def check(result, k):
        rows, uniq, inverse, n_unique = result
        nu = int(n_unique)
        assert nu == int(torch.unique(k).numel())
        assert int(inverse.min()) >= 0 and int(inverse.max()) < nu
        assert torch.equal(uniq[:nu][inverse.long()], k)
        assert torch.equal(rows.view(torch.float32)[:nu][inverse.long()], rows_of[k])

    def eager():
        k = draw()
        check(cache.lookup_unique(0, k), k)

    eager()
    static = draw()
    graphs = []
    for _ in range(90):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            result = cache.lookup_unique(0, static)
        graphs.append((g, result))
        eager()                          # the captured call has not run
        for g, result in graphs[-2:]:
            for _ in range(2):
                static.copy_(draw())
                g.replay()
                check(result, static)
        eager()
        if len(graphs) > 3:
            graphs.pop(0)
    cache.close()
