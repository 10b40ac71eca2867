"""Sampling, dedup / relabel and counter parity of the CUDA path against the CPU checker.

Bit-exact: node ids, labels, local edge lists and both counter arrays must equal the host
replay for the same seeds, RNG seed and batch number.
"""
import numpy as np
import pytest

import legion_ibp_b200 as L
from conftest import small_graph

pytestmark = pytest.mark.gpu


def _setup(indptr, indices, train_ids, labels, batch, fanout, row_bytes=16, pipes=2):
    import torch
    dev = 0
    d_indptr = torch.from_numpy(indptr).cuda()
    d_indices = torch.from_numpy(indices).cuda()
    g = L.GraphStorage(dev, d_indptr, d_indices)
    f = L.FeatureStorage(dev, len(indptr) - 1, row_bytes, None)
    d_ids = torch.from_numpy(train_ids).cuda()
    d_lab = torch.from_numpy(labels).cuda()
    f.set_split(L.TRAINMODE, d_ids, d_lab)
    pool = L.MemoryPool(dev, batch, fanout, row_bytes, pipes)
    return g, f, pool


def _run_ops(g, f, pool, batch, it, fanout, global_batch, pipe=0, cache=None):
    pool.set_batch(it, L.TRAINMODE, pipe, global_batch)
    L.BatchGenerate(None, f, cache, pool, batch, it, 0, 0, L.TRAINMODE, False, len(fanout))
    L.FeatureCacheLookup(None, cache, pool, 1, 0)
    L.IOSubmit(None, f, pool, 2, 0)
    for h, k in enumerate(fanout):
        L.RandomSample(None, g, cache, pool, k, 0, 3 * (h + 1))
        L.FeatureCacheLookup(None, cache, pool, 3 * (h + 1) + 1, 0)
        L.IOSubmit(None, f, pool, 3 * (h + 1) + 2, 0)
    L.IOComplete(None, cache, pool, 0, L.TRAINMODE)


def _fetch(pool, pipe=0):
    nc = pool.read(L.BUF_NODE_COUNTER, pipe, 16, np.int32)
    ec = pool.read(L.BUF_EDGE_COUNTER, pipe, 16, np.int32)
    hops = int(nc[8])
    n_nodes = int(nc[9 + hops])
    n_edges = int(ec[0] + ec[1])
    return dict(node_counter=nc, edge_counter=ec,
                ids=pool.read(L.BUF_IDS, pipe, n_nodes, np.int32),
                labels=pool.read(L.BUF_LABELS, pipe, int(nc[9]), np.int32),
                agg_src=pool.read(L.BUF_AGG_SRC, pipe, n_edges, np.int32),
                agg_dst=pool.read(L.BUF_AGG_DST, pipe, n_edges, np.int32),
                src_global=pool.read(L.BUF_SRC_GLOBAL, pipe, n_edges, np.int32))


def _compare(got, ref):
    np.testing.assert_array_equal(got["node_counter"], ref["node_counter"])
    np.testing.assert_array_equal(got["edge_counter"], ref["edge_counter"])
    for k in ("ids", "labels", "src_global", "agg_dst", "agg_src"):
        np.testing.assert_array_equal(got[k], ref[k], err_msg=k)


CASES = [
    # n_nodes, n_pairs, batch, fanout, seed
    (3000, 40000, 64, [25, 10], 1),
    (3000, 40000, 200, [5, 5, 5], 2),
    (500, 20000, 50, [32, 32], 3),      # dense: most nodes above the fanout, heavy dedup
    (20000, 30000, 300, [25, 10], 4),   # sparse: many isolated and low-degree nodes
    (3000, 60000, 1, [25, 10], 5),      # single seed
    (3000, 40000, 100, [1], 6),
    (3000, 40000, 128, [15, 10, 5], 7),
]


@pytest.mark.parametrize("n_nodes,n_pairs,batch,fanout,seed", CASES)
def test_batch_matches_host_replay(oracle_mod, n_nodes, n_pairs, batch, fanout, seed):
    indptr, indices = small_graph(n_nodes, n_pairs, seed)
    rng = np.random.default_rng(seed)
    train = rng.permutation(n_nodes)[: max(batch * 3 + 7, 10)].astype(np.int32)
    labels = rng.integers(0, 47, len(train)).astype(np.int32)
    g, f, pool = _setup(indptr, indices, train, labels, batch, fanout)
    pool.set_rng(0x1234ABCD5678EF00 + seed, 64)
    n_batches = (len(train) - 1) // batch + 1
    for it in range(n_batches):  # includes the shortened tail batch
        _run_ops(g, f, pool, batch, it, fanout, global_batch=100 + it, pipe=it % 2)
        got = _fetch(pool, it % 2)
        ref = oracle_mod.run_batch(indptr, indices, train, labels, batch, it, fanout, 100 + it,
                                   0x1234ABCD5678EF00 + seed)
        _compare(got, ref)
        assert pool.device_error() == 0
    pool.close(); f.close(); g.close()


@pytest.mark.parametrize("shift", [20, 6, 0])
def test_id_map_front_and_back_regions(oracle_mod, shift):
    """The id map tries a small front region first and falls back to the worst-case-sized back region.
    With a front of 64 slots nearly every node lands in the back region, which must then be cleared
    before the next batch on the same pipe; with shift 0 the front alone is as large as the worst case."""
    n_nodes, n_pairs, batch, fanout, seed = 3000, 40000, 128, [15, 10, 5], 7
    indptr, indices = small_graph(n_nodes, n_pairs, seed)
    rng = np.random.default_rng(seed)
    train = rng.permutation(n_nodes)[: batch * 6].astype(np.int32)
    labels = rng.integers(0, 47, len(train)).astype(np.int32)
    L._check(L.lib().legion_set_tunable(b"map_front_shift", shift))
    try:
        g, f, pool = _setup(indptr, indices, train, labels, batch, fanout)
    finally:
        L._check(L.lib().legion_set_tunable(b"map_front_shift", -1))
    pool.set_rng(77, 64)
    for it in range(6):
        pipe = 0 if it < 4 else 1          # four batches in a row on one pipe, then the other
        _run_ops(g, f, pool, batch, it, fanout, global_batch=it, pipe=pipe)
        _compare(_fetch(pool, pipe), oracle_mod.run_batch(indptr, indices, train, labels, batch, it, fanout, it, 77))
        assert pool.device_error() == 0
    pool.close(); f.close(); g.close()


@pytest.mark.parametrize("max_rounds", [1, 2, 3])
def test_fallback_after_few_rounds(oracle_mod, max_rounds):
    """With the rejection rounds cut short the lane-ordered fallback settles the draws."""
    indptr, indices = small_graph(400, 12000, 11)
    rng = np.random.default_rng(0)
    train = rng.permutation(400)[:150].astype(np.int32)
    labels = np.zeros(len(train), np.int32)
    fanout = [25, 10]
    g, f, pool = _setup(indptr, indices, train, labels, 50, fanout)
    pool.set_rng(77, max_rounds)
    for it in range(3):
        _run_ops(g, f, pool, 50, it, fanout, global_batch=it)
        ref = oracle_mod.run_batch(indptr, indices, train, labels, 50, it, fanout, it, 77, max_rounds=max_rounds)
        _compare(_fetch(pool), ref)
    pool.close(); f.close(); g.close()


def test_structure_properties_large_batch(oracle_mod):
    """Size-independent properties on a batch too large to eyeball: every edge is a real CSR edge,
    no neighbour is drawn twice for one node, dst nodes are a prefix of src nodes, ids are unique."""
    n = 200000
    indptr, indices = small_graph(n, 3000000, 21)
    rng = np.random.default_rng(1)
    train = rng.permutation(n)[:8000].astype(np.int32)
    labels = rng.integers(0, 172, len(train)).astype(np.int32)
    fanout = [25, 10]
    g, f, pool = _setup(indptr, indices, train, labels, 8000, fanout)
    pool.set_rng(5, 64)
    _run_ops(g, f, pool, 8000, 0, fanout, global_batch=9)
    got = _fetch(pool)
    nc, ec = got["node_counter"], got["edge_counter"]
    ids = got["ids"]
    assert len(np.unique(ids)) == len(ids)
    np.testing.assert_array_equal(ids[:8000], train[:8000])
    assert nc[8] == 2 and nc[9] == 8000 and nc[11] == len(ids)
    e1, e2 = int(ec[10]), int(ec[11])
    assert ec[13] == 0 and ec[14] == e1
    src, dst = got["agg_src"], got["agg_dst"]
    # hop 1 samples for the seeds only, hop 2 for every node known after hop 1
    assert dst[:e1].max() < nc[9] and dst[e1:e1 + e2].max() < nc[10]
    assert src[:e1].max() < nc[10] and src.max() < nc[11]
    np.testing.assert_array_equal(ids[src], got["src_global"])
    # membership and no duplicate per (hop, dst)
    for lo, hi, k in ((0, e1, 25), (e1, e1 + e2, 10)):
        d = ids[dst[lo:hi]].astype(np.int64)
        s = got["src_global"][lo:hi].astype(np.int64)
        key = d * n + s
        # a multigraph-free CSR: (d, s) pairs of one hop must be unique
        assert len(np.unique(key)) == len(key)
        full = np.repeat(np.arange(n, dtype=np.int64), np.diff(indptr)) * n + indices
        assert np.isin(key, full).all()
        cnt = np.bincount(dst[lo:hi])
        deg = np.diff(indptr)[ids[:len(cnt)]]
        np.testing.assert_array_equal(cnt, np.minimum(deg, k))
    ref = oracle_mod.run_batch(indptr, indices, train, labels, 8000, 0, fanout, 9, 5)
    _compare(got, ref)
    pool.close(); f.close(); g.close()


def test_uniformity_chi_square(oracle_mod):
    """Each neighbour of a node of degree d is kept with probability k/d: chi-square over many batches."""
    n = 64
    train = np.arange(n, dtype=np.int32)
    labels = np.zeros(n, np.int32)
    for kk, dd in ((10, 40), (25, 30)):   # direct draw, and the leave-out branch
        indptr = np.arange(n + 1, dtype=np.int64) * dd
        indices = np.tile(np.arange(dd, dtype=np.int32), n)
        g, f, pool = _setup(indptr, indices, train, labels, n, [kk])
        pool.set_rng(2024, 64)
        counts = np.zeros(dd, np.int64)
        reps = 200
        for b in range(reps):
            _run_ops(g, f, pool, n, 0, [kk], global_batch=b)
            got = _fetch(pool)
            assert len(got["src_global"]) == n * kk
            counts += np.bincount(got["src_global"], minlength=dd)[:dd]
        expected = reps * n * kk / dd
        chi2 = float(((counts - expected) ** 2 / expected).sum())
        # dd-1 degrees of freedom; 99.99% quantile of chi2(39) ~ 78, chi2(29) ~ 64
        assert chi2 < 90, (kk, dd, chi2)
        pool.close(); f.close(); g.close()


def test_rejects_bad_arguments():
    import torch
    indptr, indices = small_graph(300, 2000, 1)
    train = np.arange(50, dtype=np.int32)
    g, f, pool = _setup(indptr, indices, train, train.copy(), 10, [5])
    with pytest.raises(L.LegionError):
        L.RandomSample(None, g, None, pool, 33, 0, 3)          # fanout above 32
    with pytest.raises(L.LegionError):
        L.RandomSample(None, g, None, pool, 5, 0, 4)           # not a sampling op id
    with pytest.raises(L.LegionError):
        L.BatchGenerate(None, f, None, pool, 11, 0, 0, 0, L.TRAINMODE, False, 1)  # above the pool's batch
    with pytest.raises(L.LegionError):
        L.MemoryPool(0, 10, [40], 16)
    pool.close(); f.close(); g.close()


def test_isolated_nodes_hubs_and_empty_topology(oracle_mod):
    """Edge cases of the topology: a graph without edges (every hop is empty), a star (one hub whose
    degree is far above the fanout, leaves of degree 1) plus isolated seeds, and ids at both ends of
    the id range."""
    # no edges at all
    n = 100
    indptr = np.zeros(n + 1, np.int64)
    indices = np.zeros(1, np.int32)
    train = np.arange(n, dtype=np.int32)[::-1].copy()
    labels = np.arange(n, dtype=np.int32)
    g, f, pool = _setup(indptr, indices, train, labels, 40, [25, 10])
    pool.set_rng(1, 64)
    for it in range(3):
        _run_ops(g, f, pool, 40, it, [25, 10], global_batch=it, pipe=it % 2)
        got = _fetch(pool, it % 2)
        ref = oracle_mod.run_batch(indptr, indices, train, labels, 40, it, [25, 10], it, 1)
        _compare(got, ref)
        assert got["edge_counter"][10] == 0 and got["edge_counter"][11] == 0 and len(got["ids"]) == min(40, 100 - 40 * it)
    pool.close(); f.close(); g.close()
    # star: node 0 is the hub of 5000 leaves; nodes 5001..5999 are isolated
    n = 6000
    deg = np.zeros(n, np.int64)
    deg[0] = 5000
    deg[1:5001] = 1
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    indices = np.concatenate([np.arange(1, 5001), np.zeros(5000)]).astype(np.int32)
    train = np.array([0, 5999, 1, 5000, 5500, 2500, 5001], np.int32)
    labels = np.arange(len(train), dtype=np.int32)
    for fanout in ([25, 10], [32, 32, 32], [1, 1]):
        g, f, pool = _setup(indptr, indices, train, labels, 7, fanout)
        pool.set_rng(9, 64)
        for gb in range(3):
            _run_ops(g, f, pool, 7, 0, fanout, global_batch=gb)
            got = _fetch(pool)
            ref = oracle_mod.run_batch(indptr, indices, train, labels, 7, 0, fanout, gb, 9)
            _compare(got, ref)
            e1 = int(got["edge_counter"][10])
            assert e1 == min(fanout[0], 5000) + 3        # the hub's picks + one edge for each of the three leaves
            assert pool.device_error() == 0
        pool.close(); f.close(); g.close()


@pytest.mark.parametrize("fanout", [[8], [9, 7], [16, 1], [17, 16], [32, 8], [2, 3, 32]])
@pytest.mark.parametrize("batch", [1, 31, 257, 1024])
@pytest.mark.parametrize("max_rounds", [1, 64])
def test_lane_groups_and_scan_tiles(oracle_mod, fanout, batch, max_rounds):
    """Fanouts at the edges of the lane groups that share an input (8, 16, 32), degrees on both sides of the fanout and
    of twice the fanout, batches around the scan's tiles of 1024 entries; with one round nearly every draw goes
    through the lane-ordered fallback."""
    indptr, indices = small_graph(2500, 30000, 31)
    rng = np.random.default_rng(batch)
    train = rng.integers(0, 2500, batch + batch // 2 + 1).astype(np.int32)   # seeds may repeat
    labels = rng.integers(0, 47, len(train)).astype(np.int32)
    g, f, pool = _setup(indptr, indices, train, labels, batch, fanout)
    pool.set_rng(9, max_rounds)
    for it in range(2):  # the second batch is the ragged tail
        _run_ops(g, f, pool, batch, it, fanout, global_batch=it)
        _compare(_fetch(pool), oracle_mod.run_batch(indptr, indices, train, labels, batch, it, fanout, it, 9, max_rounds=max_rounds))
        assert pool.device_error() == 0
    pool.close(); f.close(); g.close()


def test_large_hop_matches_host_replay(oracle_mod):
    """A hop of more 1024-entry tiles than CTAs that run at once."""
    indptr, indices = small_graph(150000, 4000000, 41)
    rng = np.random.default_rng(3)
    train = rng.permutation(150000)[:9000].astype(np.int32)
    labels = np.zeros(len(train), np.int32)
    g, f, pool = _setup(indptr, indices, train, labels, 9000, [25, 16])
    pool.set_rng(13, 64)
    for it in range(2):
        _run_ops(g, f, pool, 9000, 0, [25, 16], global_batch=it)
        _compare(_fetch(pool), oracle_mod.run_batch(indptr, indices, train, labels, 9000, 0, [25, 16], it, 13))
        assert pool.device_error() == 0
    pool.close(); f.close(); g.close()


def _replay_ops(O, indptr, indices, seeds, fanout, ops, global_batch, seed):
    """Host replay of the sampling ops in any order: every op samples all nodes known so far with the fanout and the RNG
    word of its hop; edges follow one another, new nodes are numbered in order of first appearance."""
    nc, ec = np.zeros(16, np.int32), np.zeros(16, np.int32)
    ids = list(seeds)
    local = {}
    for i, u in enumerate(ids):
        local.setdefault(int(u), i)
    O.counter_update(nc, ec, 0, len(ids), len(fanout))
    src, dst, src_global = [], [], []
    for op in ops:
        h = op // 3 - 1
        s, d = O.sample_hop(indptr, indices, np.array(ids, np.int32), fanout[h], h, global_batch, seed)
        before = len(ids)
        for u in s:
            if int(u) not in local:
                local[int(u)] = len(ids)
                ids.append(int(u))
            src.append(local[int(u)])
        src_global += list(s)
        dst += list(d)
        nc[6] += len(ids) - before
        ec[2] += len(s)
        O.counter_update(nc, ec, op, 0, 0)
    return dict(node_counter=nc, edge_counter=ec, ids=ids, agg_src=src, agg_dst=dst, src_global=src_global)


def _fetch_known(pool, pipe=0):
    """What the ops so far have left, whichever they were."""
    nc = pool.read(L.BUF_NODE_COUNTER, pipe, 16, np.int32)
    ec = pool.read(L.BUF_EDGE_COUNTER, pipe, 16, np.int32)
    n, e = int(nc[0] + nc[1]), int(ec[0] + ec[1])
    return dict(node_counter=nc, edge_counter=ec, ids=pool.read(L.BUF_IDS, pipe, n, np.int32),
                agg_src=pool.read(L.BUF_AGG_SRC, pipe, e, np.int32), agg_dst=pool.read(L.BUF_AGG_DST, pipe, e, np.int32),
                src_global=pool.read(L.BUF_SRC_GLOBAL, pipe, e, np.int32))


@pytest.mark.parametrize("fanout,ops", [([25, 10], [6]), ([25, 10], [6, 3]), ([10, 25], [6, 3]), ([25, 10], [3, 3]),
                                        ([25, 10], [3, 3, 6]), ([25, 10], [6, 6, 3]), ([5, 15, 10], [3, 9]),
                                        ([5, 15, 10], [9, 6, 3]), ([16, 2], [6, 6, 3]), ([30, 1], [6, 6, 6, 3, 6])])
@pytest.mark.parametrize("pipes", [1, 2])
def test_sampling_ops_in_any_order(oracle_mod, fanout, ops, pipes):
    """Ops that skip a hop, come in another order or more than once, as long as their nodes and edges fit the pool; the
    repeated ones have more inputs than the records hold entries for and are sampled in parts."""
    n_nodes, batch = 20000, 40
    indptr, indices = small_graph(n_nodes, 30000, 51)
    train = np.random.default_rng(2).permutation(n_nodes)[:batch * 3].astype(np.int32)
    train[5] = train[7]
    g, f, pool = _setup(indptr, indices, train, train.copy(), batch, fanout, pipes=pipes)
    pool.set_rng(21, 64)
    for it in range(3):
        pool.set_batch(it, L.TRAINMODE, it % pipes, it)
        L.BatchGenerate(None, f, None, pool, batch, it, 0, 0, L.TRAINMODE, False, len(fanout))
        for op in ops:
            L.RandomSample(None, g, None, pool, fanout[op // 3 - 1], 0, op)
        want = _replay_ops(oracle_mod, indptr, indices, train[it * batch:(it + 1) * batch], fanout, ops, it, 21)
        got = _fetch_known(pool, it % pipes)
        assert len(want["ids"]) <= pool.max_nodes and len(want["agg_src"]) <= pool.max_edges
        for k in want:
            np.testing.assert_array_equal(got[k], want[k], err_msg=k)
        assert pool.device_error() == 0
    # the pool's own order afterwards
    _run_ops(g, f, pool, batch, 0, fanout, global_batch=9)
    _compare(_fetch(pool), oracle_mod.run_batch(indptr, indices, train, train, batch, 0, fanout, 9, 21))
    pool.close(); f.close(); g.close()


def _defined(got, ref_ids, fanout, limit_nodes):
    """A batch that an error ended: counters of whole hops, indices in range, ids those of the replay."""
    nc, ec = got["node_counter"], got["edge_counter"]
    n, e = int(nc[0] + nc[1]), int(ec[0] + ec[1])
    hops = len(fanout)
    assert nc[8] == hops and nc[9] <= n <= limit_nodes and nc[9 + hops] == n and nc[6] == 0 and ec[2] == 0
    np.testing.assert_array_equal(got["ids"], ref_ids[:n])
    if e:
        assert 0 <= got["agg_src"].min() and got["agg_src"].max() < n and 0 <= got["agg_dst"].min() and got["agg_dst"].max() < n
    return n, e


@pytest.mark.parametrize("pipes", [1, 2])
def test_hop_that_does_not_fit_leaves_the_counters_of_the_hops_before(oracle_mod, pipes):
    """The first hop twice over a dense graph has more edges than the pool: error 2 in the scan.  The batch stands as after
    the first op, the ops behind it do nothing, and after the reset the pool works as before."""
    fanout, batch, n_nodes = [20, 2], 64, 20000
    indptr, indices = small_graph(n_nodes, 600000, 61)
    train = np.random.default_rng(4).permutation(n_nodes)[:batch * 2].astype(np.int32)
    g, f, pool = _setup(indptr, indices, train, train.copy(), batch, fanout, pipes=pipes)
    pool.set_rng(3, 64)
    for rep in range(2):
        pool.set_batch(0, L.TRAINMODE, 0, rep)
        L.BatchGenerate(None, f, None, pool, batch, 0, 0, 0, L.TRAINMODE, False, len(fanout))
        for op in (3, 3, 6):
            L.RandomSample(None, g, None, pool, fanout[op // 3 - 1], 0, op)
        want = _replay_ops(oracle_mod, indptr, indices, train[:batch], fanout, [3], rep, 3)
        full = _replay_ops(oracle_mod, indptr, indices, train[:batch], fanout, [3, 3], rep, 3)
        assert len(full["agg_src"]) > pool.max_edges > len(want["agg_src"])
        got = _fetch_known(pool)
        n, e = _defined(got, want["ids"], fanout, len(want["ids"]))
        assert (n, e) == (len(want["ids"]), len(want["agg_src"]))
        np.testing.assert_array_equal(got["agg_src"], want["agg_src"])
        np.testing.assert_array_equal(got["agg_dst"], want["agg_dst"])
        assert pool.device_error(reset=True) == 2
        _run_ops(g, f, pool, batch, 1, fanout, global_batch=rep)
        _compare(_fetch(pool), oracle_mod.run_batch(indptr, indices, train, train, batch, 1, fanout, rep, 3))
        assert pool.device_error() == 0
    pool.close(); f.close(); g.close()


@pytest.mark.parametrize("limit", [-1, 0])
@pytest.mark.parametrize("pipes", [1, 2])
def test_waits_of_the_scan_that_give_up(oracle_mod, limit, pipes):
    """Waits that give up at once (-1), or after one read (0: some do, some do not).  The kernels return, error 6 is
    reported, the counters are those of whole hops, no index is out of range, and the next batch is the replay's."""
    fanout, batch, n_nodes = [25, 10], 4000, 60000
    indptr, indices = small_graph(n_nodes, 700000, 62)
    train = np.random.default_rng(6).permutation(n_nodes)[:batch].astype(np.int32)
    g, f, pool = _setup(indptr, indices, train, train.copy(), batch, fanout, pipes=pipes)
    pool.set_rng(8, 64)
    errors = 0
    for rep in range(6):
        ref = oracle_mod.run_batch(indptr, indices, train, train, batch, 0, fanout, rep, 8)
        L._check(L.lib().legion_set_tunable(b"scan_wait_limit", limit))
        try:
            _run_ops(g, f, pool, batch, 0, fanout, global_batch=rep, pipe=rep % pipes)
        finally:
            L._check(L.lib().legion_set_tunable(b"scan_wait_limit", 1 << 20))
        got = _fetch_known(pool, rep % pipes)
        n, e = _defined(got, ref["ids"], fanout, len(ref["ids"]))
        assert got["edge_counter"][10:12].sum() == e
        err = pool.device_error(reset=True)
        assert err in (0, 6)
        errors += err == 6
        assert (n, e) in [(batch, 0)] if limit < 0 else (n, e) in [(batch, 0), (int(ref["node_counter"][10]), int(ref["edge_counter"][10])),
                                                                   (len(ref["ids"]), len(ref["agg_src"]))]
        if err == 0:
            _compare(_fetch(pool, rep % pipes), ref)
        _run_ops(g, f, pool, batch, 0, fanout, global_batch=rep, pipe=rep % pipes)
        _compare(_fetch(pool, rep % pipes), ref)
        assert pool.device_error() == 0
    assert errors == 6 if limit < 0 else errors > 0
    pool.close(); f.close(); g.close()


@pytest.mark.parametrize("pdl", [0, 1])
@pytest.mark.parametrize("n_nodes,n_pairs,batch,fanout,pipes", [(3000, 40000, 200, [5, 5, 5], 1), (3000, 40000, 200, [5, 5, 5], 2),
                                                                (500, 20000, 50, [32, 32], 1), (150000, 4000000, 9000, [25, 16], 1),
                                                                (150000, 4000000, 9000, [25, 16], 2)])
def test_dependent_and_ordinary_launches(oracle_mod, pdl, n_nodes, n_pairs, batch, fanout, pipes):
    """Both ways of launching the kernels of a hop, small hops and hops of more CTAs than run at once, one pipe and two."""
    indptr, indices = small_graph(n_nodes, n_pairs, 81)
    train = np.random.default_rng(5).permutation(n_nodes)[:batch].astype(np.int32)
    g, f, pool = _setup(indptr, indices, train, train.copy(), batch, fanout, pipes=pipes)
    pool.set_rng(17, 64)
    L._check(L.lib().legion_set_tunable(b"pdl", pdl))
    try:
        for it in range(3):
            _run_ops(g, f, pool, batch, 0, fanout, global_batch=it, pipe=it % pipes)
            _compare(_fetch(pool, it % pipes), oracle_mod.run_batch(indptr, indices, train, train, batch, 0, fanout, it, 17))
            assert pool.device_error() == 0
    finally:
        L._check(L.lib().legion_set_tunable(b"pdl", -1))
    pool.close(); f.close(); g.close()
