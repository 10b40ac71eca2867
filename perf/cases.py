"""The work that a user of this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values.  Its "kind" is the public interface that it goes through:

  serve    Runner: batches of the device-resident seed list, enqueued one behind the other and waited for
           (a single one goes through RunOnce); the consumer then reads the hand-off buffers
  infer    Runner.submit_host / collect_host: seeds from host memory, the batch stays on the GPU
  host     Runner.submit_host_to / collect_host: seeds from host memory, block structure back to host arrays
  ops      the five operators in the reference's order on the caller's stream (run_batch)
  gather   gather_rows_noalloc: one id list, rows out
  encode   quantize_table: fp32 rows into compressed rows (the way back, the decoding gather, is in the serve cases)

A batch has as many nodes and edges as its seeds happen to reach.  The consumer here pads it with zeros to the size
of its model's captured step, as a program that replays one graph for every batch does.

Graphs are R-MAT with the densities of the benchmark configurations, scaled so that the topology, the caches and
the tables of one state are hundreds of megabytes to a few gigabytes: far above the L2 cache, quick to make.
"""
import functools
import importlib.util
import math
import os
import sys

import numpy as np
import torch


@functools.lru_cache(maxsize=None)
def _package():
    """The package directory is `legion-ibp_b200` (beside this folder's parent); it is imported as legion_ibp_b200."""
    if "legion_ibp_b200" in sys.modules:
        return sys.modules["legion_ibp_b200"]
    pkg = os.path.join(os.getcwd(), "legion-ibp_b200")
    spec = importlib.util.spec_from_file_location("legion_ibp_b200", os.path.join(pkg, "__init__.py"),
                                                  submodule_search_locations=[pkg])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["legion_ibp_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


# ---- the cases ---------------------------------------------------------------------------------------------------

def _batch_case(kind, nodes, pairs, feat, batch, fanout, batches, elt="f32", cached=1.0, codec="raw", host_codec=False,
                lru=False, slots=4, edge_counts=False):
    """cached: share of the rows that the GPU's cache holds (the others stay in pinned host memory)."""
    return dict(kind=kind, nodes=nodes, pairs=pairs, feat=feat, elt=elt, batch=batch, fanout=fanout, batches=batches,
                cached=cached, codec=codec, host_codec=host_codec, lru=lru, slots=slots, edge_counts=edge_counts)


def listed():
    def named(name, case):
        return dict(case, name=name)

    return [
        # one small batch and the wait for it: online inference, and the floor that every batch pays in launches
        named("infer-small", _batch_case("infer", 500000, 5000000, 128, 32, "10,5", 1)),
        # products-shaped training batches, whole table cached, sampled ahead of the two hand-off slots that the
        # trainers' segment has: the sampling_server's steady state
        named("products-train", _batch_case("serve", 2449029, 34000000, 100, 800, "25,10", 8, slots=2)),
        # the same with the int8 cache: rows are decoded inside the gather
        named("products-int8", _batch_case("serve", 2449029, 34000000, 100, 800, "25,10", 4, codec="int8")),
        # paper100M-shaped batches scaled down: a degree-ordered cache of 20% of the rows, the others by zero-copy
        # and by staged seed rows from pinned host memory
        named("paper-train", _batch_case("serve", 8000000, 64000000, 128, 8000, "25,10", 4, cached=0.2)),
        # the same through the host-buffer calls: seeds in, block structure out over the host link
        named("paper-host", _batch_case("host", 8000000, 64000000, 128, 8000, "25,10", 4, cached=0.2)),
        # compressed rows in the cache and in the host table (fp8), so that a miss moves a quarter of the bytes
        named("paper-fp8", _batch_case("serve", 8000000, 64000000, 128, 8000, "25,10", 4, cached=0.2, codec="e4m3",
                                       host_codec=True)),
        # MAG240M-shaped rows (768 x fp16), whole table in the cache
        named("mag-train", _batch_case("serve", 2000000, 16000000, 768, 1024, "25,15", 4, elt="f16")),
        # LRU stress: three hops, Zipf seeds, 8-way cache of 10% of the rows, thousands of insertions per batch
        named("lru-stress", _batch_case("serve", 8000000, 33600000, 128, 4096, "15,10,5", 2, cached=0.1, lru=True,
                                        slots=2)),
        # validation through the operators, ragged sizes: 75 floats are not a multiple of 16 bytes
        named("ops-ragged", _batch_case("ops", 1000003, 12000000, 75, 1237, "15,10", 1)),
        # a trainer that asks for the rows of a short list of its own
        named("gather-short", dict(kind="gather", nodes=300000, feat=128, elt="f32", rows=1000, cached=1.0)),
        # and of a long one, wide rows
        named("gather-long", dict(kind="gather", nodes=1000000, feat=768, elt="f16", rows=250000, cached=1.0)),
        # a table is compressed before it is served
        named("encode-int8", dict(kind="encode", rows=1000000, feat=128, codec="int8")),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["serve", "serve", "serve", "serve", "infer", "host", "ops", "gather", "encode"])
    if kind == "encode":
        feat = 4 * rng.randint(8, 192)
        return dict(kind=kind, rows=_spread(rng, 10000, 100000000 // feat), feat=feat, codec=rng.choice(["int8", "e4m3"]))
    elt, feat = rng.choice([("f32", 128), ("f32", 100), ("f16", 768), ("f32", 4 * rng.randint(8, 128)),
                            ("f32", rng.randint(17, 512)), ("f32", 602)])
    width = feat * (2 if elt == "f16" else 4)
    if kind == "gather":
        return dict(kind=kind, nodes=_spread(rng, 100000, min(2000000, 3000000000 // width)), feat=feat, elt=elt,
                    rows=_spread(rng, 100, min(262144, 380000000 // width)), cached=rng.choice([1.0, 1.0, 1.0, 0.9]))
    nodes = _spread(rng, 200000, min(8000000, 4000000000 // width))
    pairs = int(nodes * rng.uniform(4, 14))
    batch = _spread(rng, 16, 8000)
    hops = rng.choice([1, 2, 2, 2, 3])
    while True:
        fan = [rng.choice([5, 10, 15, 25]) if rng.random() < 0.8 else rng.randint(2, 32) for _ in range(hops)]
        worst = batch * np.prod([1.0 + k for k in fan])
        if worst * width < 1.3e9 and worst < 3.2e6:
            break
        batch = max(16, batch * 3 // 4)
    more = {}
    what = rng.choice(["whole", "whole", "part", "codec", "lru"])
    if what == "part" and kind != "ops":
        more = dict(cached=rng.choice([0.2, 0.5]))
    elif what == "codec" and elt == "f32" and feat % 4 == 0:
        part = rng.choice([1.0, 0.2])
        more = dict(codec=rng.choice(["int8", "e4m3"]), cached=part, host_codec=part < 1.0)
    elif what == "lru" and kind in ("serve", "ops") and width % 16 == 0 and width <= 2048:
        more = dict(lru=True, cached=0.1, slots=2)
    batches = 1 if kind in ("ops", "infer") else min(rng.choice([1, 2, 4, 4, 8]), 2 if more.get("lru") else 4 if kind == "host" else 8)
    if kind == "serve" and not more.get("lru") and rng.random() < 0.4:
        more = dict(more, slots=2)
    if kind == "host" and rng.random() < 0.4:
        more = dict(more, edge_counts=True)
    while True:
        case = _batch_case(kind, nodes, pairs, feat, batch, ",".join(map(str, fan)), batches, elt=elt, **more)
        # no dearer than the listed ones: an LRU cache fetches a large share of its rows over the host link
        if work(case)["bytes"] < (300e6 if more.get("lru") else 400e6 if more.get("cached", 1.0) < 1.0 else 600e6):
            return case
        batch = batch * 2 // 3


# ---- what a pass needs -----------------------------------------------------------------------------------------

_DTYPE = {"f32": torch.float32, "f16": torch.float16}
_SIZE = {"f32": 4, "f16": 2}


def _fanout(case):
    return [int(k) for k in case["fanout"].split(",")]


def _slot_bytes(feat):
    return (feat + 4 + 15) // 16 * 16


class _Handles:
    """The framework's objects of one state, closed in order when the last output that lies in them is gone."""

    def __init__(self):
        self.close, self.keep = [], []

    def __del__(self):
        for fn in self.close:
            fn()


class _Buffer:
    """One of the framework's device buffers, for torch.as_tensor."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=typestr, data=(ptr, False), version=2)


def _view(owner, ptr, shape, typestr):
    return torch.as_tensor(_Buffer(owner, ptr, shape, typestr), device="cuda")


class _State:
    pass


def _generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed(seed * 1000 + salt)


def _normal_rows(nodes, feat, elt, seed, place):
    """N(0,1) rows in chunks: place(first_row, device rows)."""
    g = _generator(seed, 1)
    step = max(1, (1 << 26) // feat)
    for r0 in range(0, nodes, step):
        place(r0, torch.randn(min(step, nodes - r0), feat, device="cuda", generator=g, dtype=_DTYPE[elt]))


def _host_table(nodes, feat, elt, seed):
    table = torch.empty((nodes, feat), dtype=_DTYPE[elt], pin_memory=True)
    _normal_rows(nodes, feat, elt, seed, lambda r0, rows: table[r0:r0 + rows.shape[0]].copy_(rows, non_blocking=True))
    torch.cuda.synchronize()
    return table


def _zipf_batches(nodes, batch, count, seed):
    """`count` batches of distinct nodes, each in the order in which Zipf(1.1) draws over the node id meet them."""
    g = _generator(seed, 2)
    rank = torch.arange(1, nodes + 1, device="cuda", dtype=torch.float32).pow_(1.1)
    out = []
    for _ in range(count):
        key = torch.empty(nodes, device="cuda").exponential_(generator=g).mul_(rank)
        out.append(torch.topk(key, batch, largest=False).indices.to(torch.int32))
    return torch.cat(out)


def _prepare_batches(case, seed):
    L = _package()
    from legion_ibp_b200 import synth
    n, feat, elt, batch, fan = case["nodes"], case["feat"], case["elt"], case["batch"], _fanout(case)
    row_bytes = feat * _SIZE[elt]
    codec = {"raw": L.CODEC_RAW, "int8": L.CODEC_INT8, "e4m3": L.CODEC_E4M3}[case["codec"]]
    s, h = _State(), _Handles()
    s.L, s.case, s.handles = L, case, h
    s.run = {"serve": _run_serve, "infer": _run_infer, "host": _run_host, "ops": _run_ops}[case["kind"]]
    indptr, indices = synth.rmat_csr(n, case["pairs"], seed=seed, device="cuda")
    if case["lru"]:
        train = _zipf_batches(n, batch, 16, seed)
        s.n_batches = 16
    else:
        # eight batches, the last one ragged as the end of a training list is
        train = torch.randperm(n, device="cuda", generator=_generator(seed, 3))[: batch * 7 + (batch + 2) // 3].to(torch.int32)
        s.n_batches = (train.numel() + batch - 1) // batch
    labels = torch.randint(0, 172, (train.numel(),), device="cuda", generator=_generator(seed, 4), dtype=torch.int32)

    capacity = min(n, int(n * case["cached"]))
    if case["lru"]:
        ways = 8
        sets = max(1, capacity // ways)
        cache = L.UnifiedCache(0, n, row_bytes, 0, lru=(sets, ways))
        table = _host_table(n, feat, elt, seed)
        cache.set_host_table(table)
        keys, stamps, _ = cache.lru_state()
        s.lru = (_view(h, keys, (sets * ways,), "<i4"), _view(h, stamps, (sets * ways,), "<i4"))
    else:
        s.lru = ()
        order = torch.empty(n, dtype=torch.int32, device="cuda")
        L.UnifiedCache.degree_order(0, indptr, order)
        cache = L.UnifiedCache(0, n, row_bytes, capacity, codec=codec)
        if elt == "f16" and case["cached"] >= 1.0:
            # the table exists in the caches only
            table = None
            cache.place_static(order)
            _normal_rows(n, feat, elt, seed, cache.write_partition_rows)
        else:
            table = _host_table(n, feat, elt, seed)
            # the server's layout: rows of the uncached nodes by falling degree, cached rows last
            row_of = torch.empty(n, dtype=torch.int32, device="cuda")
            L.UnifiedCache.pack_order(0, order, capacity, row_of)
            if case["host_codec"]:
                stored = torch.empty((n, _slot_bytes(feat)), dtype=torch.uint8, pin_memory=True)
                L.quantize_table(0, codec, table, n, feat, stored)
                cache.set_host_codec(codec)
                table = stored
            cache.fill_static(order, table, row_of_id=row_of)
    graph = L.GraphStorage(0, indptr, indices)
    features = L.FeatureStorage(0, n, row_bytes, table)
    features.set_split(L.TRAINMODE, train, labels)
    pipes = 1 if case["kind"] == "ops" else 2 if case["lru"] else 4
    s.pipes, s.slots = pipes, min(pipes, case["slots"])
    pool = L.MemoryPool(0, batch, fan, row_bytes, pipes, slots=s.slots)
    pool.set_rng(seed, 64)
    runner = None
    if case["kind"] != "ops":
        runner = L.Runner(0, graph, features, cache, pool, None)
        h.close.append(runner.Finalize)
    h.close += [pool.close, cache.close, features.close, graph.close]
    h.keep += [indptr, indices, train, labels, table]
    s.graph, s.features, s.cache, s.pool, s.runner = graph, features, cache, pool, runner

    s.hops, s.at = len(fan), 0
    s.room = _room(case, pool)
    s.out = []
    for slot in range(s.slots):
        b = lambda which: pool.buffer(which, slot)[0]  # noqa: E731
        s.out.append(dict(
            ids=_view(h, b(L.BUF_IDS), (pool.max_nodes,), "<i4"),
            features=_view(h, b(L.BUF_FEATURES), (pool.max_nodes, feat), "<f%d" % _SIZE[elt]),
            feature_words=_view(h, b(L.BUF_FEATURES), (pool.max_nodes, row_bytes // 4), "<i4"),
            labels=_view(h, b(L.BUF_LABELS), (batch,), "<i4"),
            agg_src=_view(h, b(L.BUF_AGG_SRC), (pool.max_edges,), "<i4"),
            agg_dst=_view(h, b(L.BUF_AGG_DST), (pool.max_edges,), "<i4"),
            nc=_view(h, b(L.BUF_NODE_COUNTER), (16,), "<i4"), ec=_view(h, b(L.BUF_EDGE_COUNTER), (16,), "<i4")))
    stageable = table is not None and not case["lru"] and codec == L.CODEC_RAW and case["cached"] < 1.0
    if case["kind"] == "serve" and stageable:
        runner.stage_seeds(L.TRAINMODE)
    if case["kind"] in ("infer", "host"):
        pinned = lambda count, dtype=torch.int32: torch.empty(count, dtype=dtype, pin_memory=True)  # noqa: E731
        t = pinned(train.numel())
        t.copy_(train)
        s.seeds = t.numpy()
        t2 = pinned(train.numel())
        t2.copy_(labels)
        s.seed_labels = t2.numpy()
        h.keep += [t, t2]
        s.counters = [np.zeros(16, np.int32), np.zeros(16, np.int32)]
        if case["edge_counts"]:
            runner.set_edge_counts(True)
        if stageable:
            runner.register_host_seeds(s.seeds)
        s.host = []
        for _ in range(case["batches"] if case["kind"] == "host" else 0):
            arrays = [pinned(pool.max_nodes), pinned(batch), pinned(pool.max_edges),
                      pinned(len(fan) * pool.max_nodes, torch.uint8) if case["edge_counts"] else pinned(pool.max_edges)]
            h.keep.append(arrays)
            s.host.append([a.numpy() for a in arrays] + [np.zeros(16, np.int32), np.zeros(16, np.int32)])
    torch.cuda.synchronize()
    return s


def _padded(s, slot, nc, ec, tails):
    """The hand-off buffers of a finished batch up to the captured step's size; what has to be zeroed goes to `tails`."""
    o = s.out[slot]
    n, e = min(s.room[0], int(nc[9 + s.hops])), min(s.room[1], int(ec[0]) + int(ec[1]))
    rows, words, edges, seeds = s.room[0], o["feature_words"], s.room[1], int(nc[9])
    tails += [o["ids"][n:rows], words[n:rows], o["agg_src"][e:edges], o["agg_dst"][e:edges], o["labels"][seeds:]]
    return dict(ids=o["ids"][:rows], features=o["features"][:rows], labels=o["labels"], agg_src=o["agg_src"][:edges],
                agg_dst=o["agg_dst"][:edges], node_counter=o["nc"], edge_counter=o["ec"])


def _on_device(s, slots):
    """Finished batches as their consumer in this process takes them: sizes from the counters (all of them by one
    copy), padding by one launch."""
    words = torch.cat([s.out[k][c] for k in slots for c in ("nc", "ec")]).tolist()
    tails = []
    out = [_padded(s, k, words[32 * i:32 * i + 16], words[32 * i + 16:32 * i + 32], tails) for i, k in enumerate(slots)]
    torch._foreach_zero_(tails)
    return out, s.lru


def _give_back():
    """The consumer's work on the batches before is over: their buffers may be written again."""
    torch.cuda.current_stream().synchronize()


def _run_serve(s):
    _give_back()
    r, L, count, first = s.runner, s.L, s.case["batches"], s.at
    s.at = first + count
    if count == 1:
        r.RunOnce(first, L.TRAINMODE, first % s.n_batches)
    else:
        for i in range(first, first + count):
            r.enqueue(i, L.TRAINMODE, i % s.n_batches)
        r.sync()
    # the batches that the hand-off slots hold now
    return _on_device(s, [(i % s.pipes) % s.slots for i in range(first + max(0, count - s.slots), first + count)])


def _seeds_of(s, i):
    lo = i % s.n_batches * s.case["batch"]
    hi = min(len(s.seeds), lo + s.case["batch"])
    return s.seeds[lo:hi], s.seed_labels[lo:hi]


def _run_infer(s):
    _give_back()
    i, s.at = s.at, s.at + 1
    nc, ec = s.counters
    s.runner.submit_host(*_seeds_of(s, i), i)
    s.runner.collect_host(None, None, None, None, nc, ec)
    tails = []
    out = _padded(s, i % s.pipes, nc, ec, tails)
    torch._foreach_zero_(tails)
    return dict(out, node_counter=nc, edge_counter=ec)


def _run_host(s):
    _give_back()
    r, first = s.runner, s.at
    s.at = first + len(s.host)
    for i, a in enumerate(s.host):
        r.submit_host_to(*_seeds_of(s, first + i), first + i, a[0], a[1], a[2], a[3])
    out, tails = [], []
    rows, edges, inputs = s.room
    for i, (ids, labels, src, dst, nc, ec) in enumerate(s.host):
        n, e = r.collect_host(None, None, None, None, nc, ec)
        o = s.out[(first + i) % s.pipes]
        tails.append(o["feature_words"][n:rows])
        d, room_d = (int(nc[9:9 + s.hops].sum()), inputs) if s.case["edge_counts"] else (e, edges)
        ids[n:rows] = 0
        labels[nc[9]:] = 0
        src[e:edges] = 0
        dst[d:room_d] = 0
        out.append(dict(ids=ids[:rows], labels=labels, agg_src=src[:edges], agg_dst=dst[:room_d], node_counter=nc,
                        edge_counter=ec, features=o["features"][:rows]))
    torch._foreach_zero_(tails)
    return out


def _run_ops(s):
    it, s.at = s.at, s.at + 1
    s.pool.set_batch(it % s.n_batches, s.L.TRAINMODE, 0, it)
    s.L.run_batch(None, s.graph, s.features, s.cache, s.pool, 0)
    return _on_device(s, [0])


def _prepare_gather(case, seed):
    L = _package()
    n, feat, elt = case["nodes"], case["feat"], case["elt"]
    row_bytes = feat * _SIZE[elt]
    s, h = _State(), _Handles()
    s.L, s.handles, s.run = L, h, _run_gather
    g = _generator(seed, 5)
    capacity = int(n * case["cached"])
    order = torch.randperm(n, device="cuda", generator=g).to(torch.int32)
    cache = L.UnifiedCache(0, n, row_bytes, capacity)
    table = None
    if capacity < n:
        table = _host_table(n, feat, elt, seed)
        cache.fill_static(order, table)
    else:
        cache.place_static(order)
        _normal_rows(n, feat, elt, seed, cache.write_partition_rows)
    # nodes that the trainer asks for: each once, in no order
    ids = torch.randperm(n, device="cuda", generator=g)[: case["rows"]].to(torch.int32)
    s.ids = ids if ids.numel() == case["rows"] else torch.randint(0, n, (case["rows"],), device="cuda", generator=g, dtype=torch.int32)
    s.table, s.n, s.row_bytes, s.capacity = table, n, row_bytes, capacity
    s.lut, s.partitions = cache.lut_ptr(), [cache.partition()[0]]
    s.out = torch.zeros((case["rows"], feat), dtype=_DTYPE[elt], device="cuda")
    h.close.append(cache.close)
    torch.cuda.synchronize()
    return s


def _run_gather(s):
    s.L.gather_rows_noalloc(None, 0, s.ids, s.lut, s.capacity, 1, 0, s.partitions, s.table, s.n, s.row_bytes, s.out)
    return s.out


def _prepare_encode(case, seed):
    L = _package()
    s = _State()
    s.L, s.run, s.n, s.feat = L, _run_encode, case["rows"], case["feat"]
    s.codec = {"int8": L.CODEC_INT8, "e4m3": L.CODEC_E4M3}[case["codec"]]
    s.rows = torch.randn(s.n, s.feat, device="cuda", generator=_generator(seed, 6))
    s.out = torch.zeros((s.n, _slot_bytes(s.feat)), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    return s


def _run_encode(s):
    s.L.quantize_table(0, s.codec, s.rows, s.n, s.feat, s.out)
    return s.out


def prepare(case, seed):
    torch.cuda.set_device(0)
    if case["kind"] == "gather":
        return _prepare_gather(case, seed)
    if case["kind"] == "encode":
        return _prepare_encode(case, seed)
    return _prepare_batches(case, seed)


def run(state):
    return state.run(state)


# ---- bounds and tolerance -----------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _expected_sizes(nodes, pairs, batch, fanout):
    """Expected (nodes, edges, sum over hops of the nodes sampled from) of one batch on an R-MAT graph.

    A node whose id has j one bits out of s appears in a pair with probability proportional to 0.24^j 0.76^(s-j),
    so its degree is about Poisson with that mean; a drawn neighbour is a node with probability proportional to its
    degree.  (Correlations between a node and its neighbours and merged duplicate pairs are left out: within
    about a tenth of what the graphs give.)"""
    s = max(1, math.ceil(math.log2(nodes)))
    j = np.arange(s + 1)
    ids = np.array([math.comb(s, int(k)) for k in j], dtype=np.float64) * (nodes / 2.0 ** s)   # nodes of each class
    lam = 2.0 * pairs * 0.24 ** j * 0.76 ** (s - j) * (2.0 ** s / nodes)
    lam = np.minimum(lam, nodes / 4.0)
    p = lam / (ids * lam).sum()
    log_fact = np.concatenate([[0.0], np.cumsum(np.log(np.arange(1, 33)))])

    def mean_drawn(k):   # E[min(degree, k)] of each class
        d = np.arange(k)
        pm = np.exp(-lam[:, None] + d[None] * np.log(lam[:, None]) - log_fact[d][None])
        return k - ((k - d)[None] * pm).sum(1)

    have = np.minimum(1.0, batch / nodes) * np.ones(s + 1)   # probability that a node of the class is in the batch
    edges = inputs = 0.0
    for k in [int(v) for v in fanout.split(",")]:
        n_in = (ids * have).sum()
        drawn = (ids * have * mean_drawn(k)).sum()
        inputs += n_in
        edges += drawn
        have = 1.0 - (1.0 - have) * np.exp(-drawn * p)
    return (ids * have).sum(), edges, inputs


def _room(case, pool):
    """Nodes, edges and nodes sampled from that the consumer's captured step has room for."""
    n, e, inputs = _expected_sizes(case["nodes"], case["pairs"], case["batch"], case["fanout"])
    return (min(pool.max_nodes, int(1.1 * n) + 1500), min(pool.max_edges, int(1.1 * e) + 1500),
            min(len(_fanout(case)) * pool.max_nodes, int(1.1 * inputs) + 1500))


def work(case):
    """Bytes: seeds and labels in and out; two CSR offsets per node sampled from; per edge its neighbour id and its
    two local ids out; per node its id out, its table entry, its row in (as it is stored) and its row out.  The path
    has no contraction and no other arithmetic to speak of."""
    if case["kind"] == "encode":
        return {"bytes": case["rows"] * (4 * case["feat"] + _slot_bytes(case["feat"])), "flops": 2 * case["rows"] * case["feat"]}
    row = case["feat"] * _SIZE[case["elt"]]
    if case["kind"] == "gather":
        return {"bytes": case["rows"] * (8 + 2 * row), "flops": 0}
    n, e, inputs = _expected_sizes(case["nodes"], case["pairs"], case["batch"], case["fanout"])
    stored = row if case["codec"] == "raw" else case["feat"] + 4
    one = 16 * case["batch"] + 16 * inputs + 12 * e + n * (8 + stored + row)
    return {"bytes": float(case["batches"] * one), "flops": 0}


def tolerance(case):
    """Rows are copied or decoded by one multiplication, codes are one rounding of one product, everything else is
    whole numbers: all of it is the same bits whatever the order of the work."""
    return "exact"
