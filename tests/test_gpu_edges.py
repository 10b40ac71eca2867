"""Kernels at the sizes where their tiling can go wrong: remainders, one row, one past a full tile."""
import numpy as np
import pytest

import legion_ibp_b200 as L
from conftest import small_graph
from test_gpu_gather import Rig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 4, 5, 31, 33, 257, 4097])
@pytest.mark.parametrize("row_bytes", [4, 12, 68, 120, 2052, 2056, 2064])
def test_flat_gather_row_counts_and_widths(oracle_mod, count, row_bytes):
    """Rows outside the 16-byte path: 4-, 8- and 16-byte elements, fewer elements than lanes and more, rows per
    warp from 4 to 32.  The rows are copies, so the comparison is exact."""
    rng = np.random.default_rng(count * 31 + row_bytes)
    n = 3000
    table = rng.integers(0, 256, (n, row_bytes)).astype(np.uint8)
    ids = rng.integers(0, n, count).astype(np.int32)
    ids[:: 7] = -1 if count > 7 else ids[:: 7]
    order = rng.permutation(n).astype(np.int32)
    rig = Rig(table, ids, count, capacity=n // 2, order=order)
    got_n, feat, _ = rig.gather(0)
    assert got_n == count
    keep = ids >= 0
    np.testing.assert_array_equal(feat[keep], table[ids[keep]])
    st = rig.cache.stats()
    hit = np.isin(ids[keep], order[: n // 2]).sum()
    assert st["local_hits"] == hit and st["misses"] == keep.sum() - hit
    rig.close()


@pytest.mark.parametrize("codec", [L.CODEC_INT8, L.CODEC_E4M3])
@pytest.mark.parametrize("feat_len", [4, 64, 68, 128, 132, 256, 260, 512, 516, 768, 772, 1024, 1028])
@pytest.mark.parametrize("shift", [0, 1])
def test_encoder_row_lengths(oracle_mod, codec, feat_len, shift):
    """Row lengths around what the lanes of a row hold in registers and row counts around the rows that a warp encodes
    together; shift: source rows that start on 4 instead of 16 bytes.  Bytes equal the host
    quantiser's."""
    import torch
    rng = np.random.default_rng(feat_len + codec)
    for n in (1, 3, 4, 5, 1000):
        x = rng.standard_normal((n, feat_len)).astype(np.float32)
        x[n // 2] = 0.0
        if n > 4:
            x[1] = np.where(x[1] > 0, 3e-40, -2e-40)   # the factor of a row of denormals is not finite
            x[2, 0] = 3e38
        src = torch.zeros(n * feat_len + 1, device="cuda")
        src[shift:shift + n * feat_len] = torch.from_numpy(x).reshape(-1).cuda()
        out = torch.full((n, oracle_mod.quant_row_bytes(feat_len)), 7, dtype=torch.uint8, device="cuda")
        L.quantize_table(0, codec, src[shift:], n, feat_len, out)
        np.testing.assert_array_equal(out.cpu().numpy(), oracle_mod.quant_rows(x, codec))


@pytest.mark.parametrize("row_bytes", [16, 512, 528, 1536, 2048])
@pytest.mark.parametrize("count", [1, 3, 4, 9, 255, 1001, 40000])
def test_vector_gather_rows_per_warp(oracle_mod, row_bytes, count):
    """Short lists give a warp 4 rows, long ones up to 32; half of the rows miss.  The allocation-free call as well."""
    import torch
    rng = np.random.default_rng(count + row_bytes)
    n = 5000
    table = rng.integers(0, 256, (n, row_bytes)).astype(np.uint8)
    ids = rng.integers(0, n, count).astype(np.int32)
    order = rng.permutation(n).astype(np.int32)
    rig = Rig(table, ids, count, capacity=n // 2, order=order)
    got_n, feat, _ = rig.gather(0)
    assert got_n == count
    np.testing.assert_array_equal(feat, table[ids])
    hit = np.isin(ids, order[: n // 2]).sum()
    st = rig.cache.stats()
    assert st["local_hits"] == hit and st["misses"] == count - hit
    host = torch.from_numpy(table).pin_memory()
    out = torch.zeros((count, row_bytes), dtype=torch.uint8, device="cuda")
    for with_host in (False, True, False):
        out.zero_()
        L.gather_rows_noalloc(None, 0, torch.from_numpy(ids).cuda(), rig.cache.lut_ptr(), n // 2, 1, 0, [rig.cache.partition()[0]],
                              host if with_host else None, n, row_bytes, out)
        want = table[ids] if with_host else np.where(np.isin(ids, order[: n // 2])[:, None], table[ids], 0)
        np.testing.assert_array_equal(out.cpu().numpy(), want)
    rig.close()


@pytest.mark.parametrize("codec", [L.CODEC_INT8, L.CODEC_E4M3])
@pytest.mark.parametrize("feat_len", [4, 100, 124, 128, 132, 256, 260, 508, 512, 772])
@pytest.mark.parametrize("host_codec", [False, True])
def test_compressed_gather_row_lengths(oracle_mod, codec, feat_len, host_codec):
    """Row lengths around 128 and 256 codes (words per lane), 508 codes (rows that one 16-byte load per lane holds) and
    lists of 1 to 33 rows and more; a third of the rows is cached.  Decoding is one multiplication: bits equal the host's."""
    import torch
    rng = np.random.default_rng(feat_len)
    n = 900
    table = rng.standard_normal((n, feat_len)).astype(np.float32)
    stored = oracle_mod.quant_rows(table, codec)
    plain = oracle_mod.dequant_rows(stored, feat_len, codec)
    order = rng.permutation(n).astype(np.int32)
    cached = np.isin(np.arange(n), order[: n // 3])
    want = plain if host_codec else np.where(cached[:, None], plain, table)
    for count in (1, 33, 700):
        ids = rng.integers(0, n, count).astype(np.int32)
        d_ids = torch.from_numpy(ids).cuda()
        lab = torch.zeros(count, dtype=torch.int32, device="cuda")
        host = torch.from_numpy(stored if host_codec else table).pin_memory()
        f = L.FeatureStorage(0, n, feat_len * 4, host)
        f.set_split(L.TRAINMODE, d_ids, lab)
        cache = L.UnifiedCache(0, n, feat_len * 4, n // 3, codec=codec)
        if host_codec:
            cache.set_host_codec(codec)
        cache.fill_static(torch.from_numpy(order).cuda(), host)
        pool = L.MemoryPool(0, count, [], feat_len * 4, 1)
        pool.set_batch(0, L.TRAINMODE, 0, 0)
        L.BatchGenerate(None, f, cache, pool, count, 0, 0, 0, L.TRAINMODE, False, 0)
        L.FeatureCacheLookup(None, cache, pool, 1, 0)
        got = pool.read(L.BUF_FEATURES, 0, count * feat_len, np.float32).reshape(count, feat_len)
        np.testing.assert_array_equal(got, want[ids])
        st = cache.stats()
        assert st["local_hits"] == cached[ids].sum() and st["misses"] == count - cached[ids].sum()
        pool.close(); cache.close(); f.close()


def test_cache_that_holds_every_node_needs_no_fetch(oracle_mod):
    """A cache with room for every node skips the fetch of misses; one whose order names a node twice, and so leaves another
    out, must not, nor one that is filled again with fewer nodes."""
    import torch
    rng = np.random.default_rng(5)
    n, row_bytes, count = 700, 64, 900
    table = rng.integers(0, 256, (n, row_bytes)).astype(np.uint8)
    ids = np.concatenate([rng.permutation(n), rng.integers(0, n, count - n)]).astype(np.int32)   # every node is asked for
    order = rng.permutation(n).astype(np.int32)
    twice = order.copy()
    twice[-1] = twice[0]
    for o, held in ((order, n), (twice, n - 1), (order[: n // 2], n // 2), (order, n)):
        rig = Rig(table, ids, count, capacity=n, order=o)
        for _ in range(2):
            np.testing.assert_array_equal(rig.gather(0)[1], table[ids])
        st = rig.cache.stats()
        miss = (~np.isin(ids, o)).sum()
        assert st["misses"] == 2 * miss and st["local_hits"] == 2 * (count - miss) and (miss == 0) == (held == n)
        rig.cache.fill_static(torch.from_numpy(order[:10].copy()).cuda(), rig.h_table)
        np.testing.assert_array_equal(rig.gather(0)[1], table[ids])
        rig.close()


def test_changed_table_of_a_cache_that_holds_every_node(oracle_mod):
    """The caller takes the address of the lookup table of a full cache and marks nodes as missed: their rows come from the
    host table again, call after call, and every call empties its list of them."""
    import torch
    rng = np.random.default_rng(9)
    n, row_bytes, count = 600, 64, 600
    table = rng.integers(0, 256, (n, row_bytes)).astype(np.uint8)
    ids = rng.permutation(n).astype(np.int32)
    rig = Rig(table, ids, count, capacity=n, order=rng.permutation(n).astype(np.int32))
    np.testing.assert_array_equal(rig.gather(0)[1], table[ids])
    lut = rig.cache.lut_ptr()
    missed = np.full(n // 2, -2, np.int32)  # the first half of the nodes
    L._check(L.lib().legion_copy(L.C.c_void_p(lut), missed.ctypes.data_as(L.C.c_void_p), L.C.c_int64(missed.nbytes), L.C.c_int32(1)))
    rig.h_table[: n // 2] ^= 0x5A  # the host's rows are told from the cached ones
    want = np.where((ids < n // 2)[:, None], table[ids] ^ 0x5A, table[ids])
    for _ in range(8):  # more misses in all than the list has places
        np.testing.assert_array_equal(rig.gather(0)[1], want)
    st = rig.cache.stats()
    assert st["misses"] == 8 * (n // 2) and st["local_hits"] == count + 8 * (n // 2)
    rig.close()


@pytest.mark.parametrize("codec", [L.CODEC_INT8, L.CODEC_E4M3])
@pytest.mark.parametrize("feat_len", [4, 60, 128, 132, 516, 772, 1028, 2052])
@pytest.mark.parametrize("shift", [0, 1])
def test_encoder_rows_with_infinities_and_nan(oracle_mod, codec, feat_len, shift):
    """Rows that are not all finite, in the lanes' registers and behind them, beside rows that are: an infinity makes the
    scale infinite and every finite code 0, a NaN leaves the scale to the other values and is stored as 0 (int8) or
    0x7F (e4m3; the host may write its sign)."""
    import torch
    rng = np.random.default_rng(feat_len)
    n = 41
    x = rng.standard_normal((n, feat_len)).astype(np.float32)
    last = feat_len - 1
    x[0, 0] = np.inf
    x[3, last] = -np.inf
    x[4, last] = np.nan
    x[7, 0] = -np.nan
    x[8] = np.nan
    x[9] = np.inf
    x[12, 0], x[12, last] = np.nan, np.inf
    x[13] = 0.0
    x[13, last] = np.nan
    x[20, rng.integers(0, feat_len)] = np.inf
    x[21, rng.integers(0, feat_len)] = np.nan
    x[n - 1, last] = np.nan
    src = torch.zeros(n * feat_len + 1, device="cuda")
    src[shift:shift + n * feat_len] = torch.from_numpy(x).reshape(-1).cuda()
    out = torch.full((n, oracle_mod.quant_row_bytes(feat_len)), 7, dtype=torch.uint8, device="cuda")
    L.quantize_table(0, codec, src[shift:], n, feat_len, out)
    with np.errstate(invalid="ignore"):
        want = oracle_mod.quant_rows(x, codec)
    if codec == L.CODEC_E4M3:
        want[:, :feat_len] = np.where(want[:, :feat_len] == 0xFF, 0x7F, want[:, :feat_len])
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("batch", [300, 16383, 16384, 16385, 40000])
@pytest.mark.parametrize("share", [0.0, 0.01, 1.0])
def test_lru_lists_of_pools_that_order_them_and_that_do_not(oracle_mod, batch, share):
    """Pools on both sides of the 16,384 rows at worst from which a list of missed rows is ordered, with lists that are
    empty, short and as long as the batch: rows, hit / miss sets and counters follow the host replay."""
    rng = np.random.default_rng(batch)
    n, feat_len, sets, ways = 100000, 16, 12000, 8
    table = rng.standard_normal((n, feat_len)).astype(np.float32)
    nodes = rng.permutation(n)
    first, cold = nodes[:batch], nodes[batch:2 * batch]
    lists = [first]
    missed = int(share * batch)
    for _ in range(2):
        lists.append(rng.permutation(np.concatenate([rng.permutation(first)[:batch - missed], rng.permutation(cold)[:missed]])))
    flat = np.concatenate(lists).astype(np.int32)
    rig = Rig(table, flat, batch, lru=(sets, ways))
    ref = oracle_mod.LruCache(sets, ways)
    for it in range(3):
        ids, clock = flat[it * batch:(it + 1) * batch], rig.cache.lru_clock()
        before = rig.cache.stats()["misses"]
        cnt, feat, _ = rig.gather(it)
        assert cnt == batch
        ci = ref.lookup(ids, clock)
        np.testing.assert_array_equal(rig.pool.read(L.BUF_CACHE_INDEX, 0, cnt, np.int64), ci)
        np.testing.assert_array_equal(feat.view(np.float32).reshape(cnt, feat_len), table[ids])
        assert rig.cache.stats()["misses"] - before == (ci < 0).sum()
        ref.insert(ids, ci, clock)
    rig.close()


@pytest.mark.parametrize("pipes", [1, 2])
@pytest.mark.parametrize("kind", ["full", "part", "lru"])
def test_operators_under_stream_capture(oracle_mod, pipes, kind):
    """A caller captures a whole batch of operators, and an allocation-free gather behind it, in a graph of its own and
    replays it over other seeds: ordinary and dependent launches, with and without a fetch."""
    import torch
    n, feat_len, batch, fanout = 6000, 32, 200, [25, 10]
    indptr, indices = small_graph(n, 60000, 91)
    rng = np.random.default_rng(14)
    table = rng.standard_normal((n, feat_len)).astype(np.float32)
    h_table = torch.from_numpy(table).pin_memory()
    d_ip, d_ix = torch.from_numpy(indptr).cuda(), torch.from_numpy(indices).cuda()
    g, f = L.GraphStorage(0, d_ip, d_ix), L.FeatureStorage(0, n, feat_len * 4, h_table)
    seeds, labels = torch.zeros(batch, dtype=torch.int32, device="cuda"), torch.zeros(batch, dtype=torch.int32, device="cuda")
    f.set_split(L.TRAINMODE, seeds, labels)
    order = torch.from_numpy(rng.permutation(n).astype(np.int32)).cuda()
    if kind == "lru":
        cache = L.UnifiedCache(0, n, feat_len * 4, 0, lru=(100, 8))
        cache.set_host_table(h_table)
    else:
        cache = L.UnifiedCache(0, n, feat_len * 4, n if kind == "full" else n // 4)
        cache.fill_static(order, h_table)
    plain = L.UnifiedCache(0, n, feat_len * 4, n // 4)
    plain.fill_static(order, h_table)
    lut, part = plain.lut_ptr(), [plain.partition()[0]]
    rows = torch.zeros((batch, feat_len), device="cuda")
    pool = L.MemoryPool(0, batch, fanout, feat_len * 4, pipes)
    pool.set_rng(23, 64)
    pool.set_batch(0, L.TRAINMODE, pipes - 1, 6)
    stream = torch.cuda.Stream()

    def ops():
        L.run_batch(stream, g, f, cache, pool, 0)
        L.gather_rows_noalloc(stream, 0, seeds, lut, n // 4, 1, 0, part, h_table, n, feat_len * 4, rows)

    torch.cuda.synchronize()
    ops()   # the driver loads the kernels' code
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        ops()
    for rep in range(4):
        train = rng.permutation(n)[:batch].astype(np.int32)
        seeds.copy_(torch.from_numpy(train))
        rows.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        ref = oracle_mod.run_batch(indptr, indices, train, np.zeros(batch, np.int32), batch, 0, fanout, 6, 23)
        pipe = pipes - 1
        np.testing.assert_array_equal(pool.read(L.BUF_NODE_COUNTER, pipe, 16, np.int32), ref["node_counter"])
        np.testing.assert_array_equal(pool.read(L.BUF_EDGE_COUNTER, pipe, 16, np.int32), ref["edge_counter"])
        np.testing.assert_array_equal(pool.read(L.BUF_IDS, pipe, len(ref["ids"]), np.int32), ref["ids"])
        for which, key in ((L.BUF_AGG_SRC, "agg_src"), (L.BUF_AGG_DST, "agg_dst")):
            np.testing.assert_array_equal(pool.read(which, pipe, len(ref[key]), np.int32), ref[key])
        feat = pool.read(L.BUF_FEATURES, pipe, len(ref["ids"]) * feat_len, np.float32).reshape(-1, feat_len)
        np.testing.assert_array_equal(feat, table[ref["ids"]])
        np.testing.assert_array_equal(rows.cpu().numpy(), table[train])
        assert pool.device_error() == 0
    del graph
    pool.close(); cache.close(); plain.close(); f.close(); g.close()
