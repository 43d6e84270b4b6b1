"""Performance cases of the embedding-extraction path, all through ``ugache_b200.runtime``.

What a program does with the cache, and how often:

* every step it looks a key batch up (``Cache.lookup``), or looks its distinct keys up once
  (``Cache.lookup_unique``), or looks up and pools (``Cache.lookup_pool``);
* a program whose consumer sits on the host takes the same batch through host buffers
  (``Cache.lookup_host``);
* it counts the keys of its batches (``Cache.record``) and reads the counters once per hotness
  window (``Cache.hotness_read``);
* at the end of a window it ranks the counters, solves for a new placement and moves the cache to
  it (``Cache.rank_hotness``, ``solve_placement``, ``Cache.refresh_all_local``).

One GPU, one replica: rows come from the replica's slice in HBM and from the pinned host table.
Tables hold 0.5 to 1 GB instead of the tens of GB of a deployment, so that they are quickly made;
slices stay larger than the L2 wherever a deployment's would decide the time.  Keys follow the
bounded-Pareto Zipf law and the rank-to-id bijection of ``ugache_b200.workload``.

A case: ``op``; ``rows`` x ``dim`` x ``elem`` = the table; ``cached`` = share of the rows in the
slice; ``keys`` = batch size, ``key_bits`` = 64 (int64) or 32 (int32); ``alpha`` = Zipf exponent;
and what its ``op`` needs besides.
"""
import functools
import math

import numpy as np
import torch

from ugache_b200 import runtime as rt
from ugache_b200 import workload as wl

_ELEM_BYTES = {"f32": 4, "f16": 2}
_TORCH_ELEM = {"f32": torch.float32, "f16": torch.float16}


# ---- cases ---------------------------------------------------------------------------------
def _case(name, op, rows, dim, elem, cached, keys, key_bits, alpha, **more):
    c = {"op": op, "rows": rows, "dim": dim, "elem": elem, "cached": cached, "keys": keys,
         "key_bits": key_bits, "alpha": alpha}
    if name is not None:
        c["name"] = name
    c.update(more)
    return c


def listed():
    return [
        # an online request: 8 samples x 26 sparse fields; launch and host time are what it costs
        _case("lookup_request", "lookup", 1_000_000, 128, "f32", 0.8, 208, 64, 1.2),
        # a serving batch of 512 samples with 32-bit ids over half-precision rows
        _case("lookup_serving_f16", "lookup", 2_000_000, 64, "f16", 0.5, 512 * 26, 32, 1.2),
        # the recommendation training step: 8192 samples x 26 fields, a tenth of the rows cached
        _case("lookup_train_10pct", "lookup", 2_000_000, 128, "f32", 0.1, 8192 * 26, 64, 1.2),
        # the same step with what eight such caches hold together: nearly every row is in HBM
        _case("lookup_train_80pct", "lookup", 2_000_000, 128, "f32", 0.8, 8192 * 26, 64, 1.2),
        # a large flat-skew batch, 65,536 x 26 fields over half-precision rows, one row in twelve
        # to fifteen from the host
        _case("lookup_flat_f16", "lookup", 8_000_000, 64, "f16", 0.2, 65536 * 26, 64, 1.05),
        # feature extraction of a sampled GNN mini-batch: distinct node ids, an odd number of them
        _case("lookup_gnn", "lookup_distinct", 2_000_000, 128, "f32", 0.9, 500_009, 64, 1.2),
        # the training step's batch deduplicated on the GPU, rows put back in batch order by the
        # consumer's index
        _case("unique_train", "unique", 2_000_000, 128, "f32", 0.8, 8192 * 26, 64, 1.2),
        # multi-hot feature: ragged bags (26 ids on average, some empty) summed
        _case("pool_sum_ragged", "pool", 2_000_000, 128, "f32", 0.8, 8192 * 26, 64, 1.2, bags=8192,
              ragged=True, mode="sum"),
        # behaviour-sequence feature: short bags of equal length averaged, half-precision rows
        _case("pool_mean_f16", "pool", 2_000_000, 64, "f16", 0.8, 65536 * 5, 32, 1.2, bags=65536,
              ragged=False, mode="mean"),
        # inference whose consumer is on the host: pinned keys in, pinned rows out, one call
        _case("host_inference", "host", 2_000_000, 128, "f32", 0.8, 16384, 64, 1.2),
        # a hotness window: the keys of 64 steps counted, the counters read and reset
        _case("record_window", "record", 2_000_000, 64, "f16", 0.2, 8192 * 26, 64, 1.2, steps=64),
        # end of a window: counters -> ranking -> placement -> cache moved, then the next step's
        # lookup; a tenth of the cached rows changes
        _case("refresh_window", "refresh", 2_000_000, 64, "f16", 0.2, 8192 * 26, 64, 1.2, drift=0.1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["lookup", "lookup", "lookup", "lookup_distinct", "unique", "pool", "pool", "host",
                     "record", "refresh"])
    elem = rng.choice(["f32", "f16"])
    # widths of embedding tables and of node features; 50 and 100 leave rows that no 32-byte (or no
    # 16-byte) piece divides
    dim = rng.choice([16, 32, 50, 64, 100, 128, 256] if op != "pool" else [16, 32, 64, 128, 256])
    row_bytes = dim * _ELEM_BYTES[elem]
    rows = min(_log_int(rng, 500_000, 8_000_000), 1_000_000_000 // row_bytes)
    cached = rng.choice([0.1, 0.2, 0.5, 0.8, 0.9, 1.0])
    alpha = round(rng.uniform(1.05, 1.4), 3)
    key_bits = rng.choice([64, 64, 32])
    cap = 500_000_000 // row_bytes  # keys: no more output than the largest listed batch
    if op == "lookup":
        return _case(None, op, rows, dim, elem, cached, _log_int(rng, 1, min(1_700_000, cap)), key_bits, alpha)
    if op == "lookup_distinct":
        return _case(None, op, rows, dim, elem, rng.choice([0.8, 0.9, 1.0]),
                     _log_int(rng, 10_000, min(500_000, rows // 4, cap)), key_bits, alpha)
    if op == "unique":
        return _case(None, op, rows, dim, elem, cached, _log_int(rng, 1000, min(500_000, cap // 2)), key_bits, alpha)
    if op == "pool":
        bags = _log_int(rng, 16, 65536)
        bag = _log_int(rng, 1, max(2, min(1000, 800_000 // bags)))
        return _case(None, op, rows, dim, elem, cached, bags * bag, key_bits, alpha, bags=bags,
                     ragged=rng.random() < 0.5, mode=rng.choice(["sum", "mean"]))
    if op == "host":
        return _case(None, op, rows, dim, elem, cached, _log_int(rng, 16, min(250_000, cap // 2)), key_bits, alpha)
    if op == "record":
        return _case(None, op, min(rows, 2_000_000), dim, elem, cached, _log_int(rng, 1000, 212_992), key_bits,
                     alpha, steps=rng.randint(8, 64))
    return _case(None, op, min(rows, 2_000_000, 256_000_000 // row_bytes), dim, elem, rng.choice([0.1, 0.2, 0.4]),
                 _log_int(rng, 1000, 212_992), key_bits, alpha, drift=round(rng.uniform(0.01, 0.1), 3))


# ---- inputs --------------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _hotness(rows, alpha):
    return wl.analytic_hotness(rows, alpha)


@functools.lru_cache(maxsize=4)
def _placement(rows, alpha, cached):
    ids, freqs = _hotness(rows, alpha)
    return rt.solve_placement("intuitive", 1, ids, freqs, cached * 100.0)


def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((seed * 1_000_003 + salt) & 0x7FFFFFFFFFFFFFFF)
    return g


def _ids(rank0, rows):
    a, b = wl.bijection(rows)
    return (rank0 * a + b) % rows


def _zipf(g, shape, rows, alpha):
    """Zipf ids: the reference generator's bounded-Pareto inverse CDF (``workload.zipf_ranks``)."""
    u = torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)
    a = alpha - 1.0
    ha = float(rows) ** a
    x = torch.pow(-ha / (u * (ha - 1.0) - ha), 1.0 / a)
    return _ids((x.to(torch.int64) - 1).clamp_(0, rows - 1), rows)


def _distinct(g, n, rows, alpha):
    """n different ids drawn without replacement with weights rank^-alpha, in random order."""
    w = torch.arange(1, rows + 1, device="cuda", dtype=torch.float32).log_().mul_(-alpha)
    u = torch.rand(rows, generator=g, device="cuda").clamp_(1e-30, 1.0 - 1e-7)
    top = torch.topk(w - torch.log(-torch.log(u)), n).indices
    return _ids(top[torch.randperm(n, generator=g, device="cuda")], rows)


class _State:
    """The cache, its host table, and the inputs of a pass.  Gives everything back when dropped."""

    def __init__(self):
        self.cache = None
        self.host = None

    def __del__(self):
        if self.cache is not None:
            self.cache.close()
        if self.host is not None:
            rt.host_free(self.host)


def prepare(case, seed):
    c, s = case, _State()
    rows, dim, n, alpha = c["rows"], c["dim"], c["keys"], c["alpha"]
    elem = _ELEM_BYTES[c["elem"]]
    s.case = c
    s.dtype = _TORCH_ELEM[c["elem"]]
    s.host, host_dev = rt.host_alloc(rows * dim * elem)
    rt.gen_table(host_dev, seed & 0x7FFFFFFF, 0, rows, dim, elem)
    s.cache = rt.Cache(1, rows, dim * elem, c["cached"], max_batch=max(n, 1024))
    s.cache.set_placement(_placement(rows, alpha, c["cached"]))
    torch.cuda.synchronize()  # the table is complete before it is read
    s.cache.build(0, torch.cuda.current_device(), s.host)

    g = _generator(seed, 7)
    kdtype = torch.int64 if c["key_bits"] == 64 else torch.int32
    if c["op"] == "lookup_distinct":
        s.keys = _distinct(g, n, rows, alpha).to(kdtype)
    elif c["op"] == "record":
        s.keys = list(_zipf(g, (c["steps"], n), rows, alpha).to(kdtype).unbind(0))
    else:
        s.keys = _zipf(g, (n,), rows, alpha).to(kdtype)

    if c["op"] == "pool":
        if c["ragged"]:  # bag lengths of random cut points: geometric-like, some bags empty
            cuts = torch.randint(0, n + 1, (c["bags"] - 1,), generator=g, device="cuda")
            ends = torch.tensor([0, n], device="cuda")
            s.offsets = torch.cat([ends[:1], torch.sort(cuts).values, ends[1:]]).to(torch.int64)
        else:
            s.offsets = None
    elif c["op"] == "host":
        s.keys_pinned = s.keys.cpu().pin_memory()
        s.out_pinned = torch.empty((n, dim), dtype=s.dtype, pin_memory=True)
        s.keys_np, s.out_np = s.keys_pinned.numpy(), s.out_pinned.numpy()
    elif c["op"] == "refresh":
        # two counter arrays as two windows would leave them: the second exchanges the counts of
        # `drift` of the cached ids with those of ids that are not cached
        ids, freqs = _hotness(rows, alpha)
        cap = int(rows * c["cached"])
        m = max(1, int(cap * c["drift"]))
        r = np.random.default_rng(seed & 0x7FFFFFFF)
        first = np.empty(rows, dtype=np.uint32)
        first[ids] = freqs
        out = ids[r.choice(cap, m, replace=False)]
        into = ids[cap + r.choice(rows - cap, m, replace=False)]
        second = first.copy()
        second[out], second[into] = first[into], first[out]
        s.counts = [second, first]
        s.window = 0
        s.all_ids = torch.arange(rows, device="cuda", dtype=torch.int32)
    return s


# ---- one pass ------------------------------------------------------------------------------
def run(s):
    c, cache = s.case, s.cache
    op = c["op"]
    if op in ("lookup", "lookup_distinct"):
        return cache.lookup(0, s.keys).view(s.dtype)
    if op == "unique":
        rows, _, inverse, n_unique = cache.lookup_unique(0, s.keys)
        # distinct rows come in order of discovery: the consumer's index puts the batch together
        return {"batch": rows.view(s.dtype).index_select(0, inverse), "n_unique": n_unique}
    if op == "pool":
        bag = 0 if c["ragged"] else c["keys"] // c["bags"]
        return cache.lookup_pool(0, s.keys, offsets=s.offsets, bag_size=bag, elem=c["elem"], mode=c["mode"])
    if op == "host":
        return cache.lookup_host(0, s.keys_np, s.out_np)
    if op == "record":
        for k in s.keys:
            cache.record(0, k)
        stream = torch.cuda.current_stream().cuda_stream
        return cache.hotness_read(0, reset=True, stream=stream)
    stream = torch.cuda.current_stream().cuda_stream
    rank_ids, rank_freqs = cache.rank_hotness(s.counts[s.window])
    s.window ^= 1
    placement = rt.solve_placement("intuitive", 1, rank_ids, rank_freqs, c["cached"] * 100.0)
    cache.refresh_all_local(placement, [0], stream)
    rows = cache.lookup(0, s.keys).view(s.dtype)
    return {"rank_ids": rank_ids, "rank_freqs": rank_freqs, "blocks": placement.nid_to_block,
            "table_words": cache.table_words(0, s.all_ids), "batch": rows}


# ---- what a pass cannot do without -----------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _expected_distinct(n, rows, alpha):
    """Expected number of different ids in a batch: sum over ranks of 1 - (1 - p)^n."""
    a = alpha - 1.0
    edges = np.arange(1, rows + 1, dtype=np.float64)
    mass = -np.diff(np.append(np.power(edges, -a), float(rows) ** -a)) / (1.0 - float(rows) ** -a)
    mass[-1] = max(mass[-1], 0.0)
    return float(-np.expm1(n * np.log1p(-np.minimum(mass, 1.0 - 1e-12))).sum())


def work(case):
    """Bytes of one pass: every different input row, key and offset read once, every output written
    once.  Nothing on the path is a contraction; pooled sums are the only arithmetic."""
    c = case
    n, kb = c["keys"], c["key_bits"] // 8
    row = c["dim"] * _ELEM_BYTES[c["elem"]]
    distinct = n if c["op"] == "lookup_distinct" else _expected_distinct(n, c["rows"], c["alpha"])
    flops = 0
    if c["op"] == "unique":  # rows, ids and index of the deduplicated lookup, then the batch
        nbytes = n * kb + distinct * (2 * row + kb) + n * 4 + n * row
    elif c["op"] == "pool":
        nbytes = n * kb + distinct * row + c["bags"] * c["dim"] * 4 + (c["bags"] * 8 if c["ragged"] else 0)
        flops = n * c["dim"]
    elif c["op"] == "record":  # keys of the window; the counters read out and reset
        nbytes = c["steps"] * n * kb + c["rows"] * 8
    elif c["op"] == "refresh":  # counters in; ranking, placement and table words out; moved rows; the batch
        moved = int(c["rows"] * c["cached"]) * c["drift"]
        nbytes = c["rows"] * (4 + 8 + 4 + 4) + 2 * moved * row + n * kb + distinct * row + n * row
    else:
        nbytes = n * kb + distinct * row + n * row
    return {"bytes": int(nbytes), "flops": int(flops)}


def tolerance(case):
    """Rows are copied, counts are whole numbers, and a pooled sum is defined addition by addition
    (fp32, key order), so every output is the same bit for bit."""
    return "exact"
