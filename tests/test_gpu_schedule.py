"""Branches of the preprocessing and the schedule at the sizes where they
change, against the oracle: vertex ranks (one CTA up to 16,384 vertices, radix
passes beyond; hubs of 32,768 and more placed by their full degrees), scans (one CTA up to 32,768
elements), degree counting over sorted and skewed input, heavy and wide rows
cut into pieces, and groups of short rows. Counts are integers: equality."""
import numpy as np
import pytest

import oracle
import tribit_b200 as tb
from tests.graphs import zip_pairs
from tests.test_gpu_rows import fans

pytestmark = pytest.mark.gpu


def check(e, n, modes=("plain",), orders=("degree", "id")):
    want, m = oracle.count(e, n)
    for order in orders:
        for mode in modes:
            with tb.Counter(order=order, dispatch=mode) as c:
                r = c.count_edges(e, n)
                assert (r.triangles, r.edges) == (want, m), (order, mode)


@pytest.mark.parametrize("n", [3, 31, 33, 1023, 1025, 16383, 16384, 16385, 32767, 32768, 32769])
def test_sizes_around_the_one_cta_kernels(n):
    check(tb.gen_er(n, 6 * n + 1, seed=n), n)


def test_degrees_past_the_exact_keys():
    # Hubs of 32,767 to 70,000 neighbours: keys of 11 leading bits, then their full degrees.
    n = 80_000
    parts = [tb.gen_er(n, 200_000, seed=5)]
    for hub, k in enumerate((32767, 32768, 33000, 40000, 65535, 65536, 70000)):
        parts.append((np.uint64(hub) << np.uint64(32)) | (np.uint64(100) + np.arange(k, dtype=np.uint64)))
    check(np.concatenate(parts), n, orders=("degree",))


def hubs_of_near_equal_degree(n, hubs, times):
    """`hubs` vertices of 32,768 and more entries, one entry less an id, the first five joined to all hubs; the rest
    of their entries name the other vertices, each about `times` times."""
    i, j = np.triu_indices(hubs, 1)
    i, j = i[i < 5], j[i < 5]
    parts = [zip_pairs(np.stack([i, j], 1))]
    joined = np.bincount(i, minlength=hubs) + np.bincount(j, minlength=hubs)
    others = hubs + np.arange(-(-(32_768 + hubs) // times), dtype=np.uint64)
    assert others[-1] < n
    for h in range(hubs):
        parts.append((np.uint64(h) << np.uint64(32)) | np.resize(others, 32_768 + hubs - 1 - h - joined[h]))
    return np.random.default_rng(n).permutation(np.concatenate(parts))


def rows_in_degree_order(e, n):
    """(neighbours, longest row) of every 32-row block under (degree, id) order, degrees counted with duplicates."""
    a, b = (e >> np.uint64(32)).astype(np.int64), (e & np.uint64(0xFFFFFFFF)).astype(np.int64)
    a, b = a[a != b], b[a != b]
    rank = np.empty(n, dtype=np.int64)
    rank[np.argsort(np.bincount(a, minlength=n) + np.bincount(b, minlength=n), kind="stable")] = np.arange(n)
    lo, hi = np.minimum(rank[a], rank[b]), np.maximum(rank[a], rank[b])
    rows = np.bincount(np.unique(lo * n + hi) // n, minlength=-(-n // 32) * 32).reshape(-1, 32)
    return rows.sum(1), rows.max(1)


@pytest.mark.parametrize("n, hubs, times", [(11_101, 45, 3), (16_001, 40, 4), (16_545, 45, 2), (90_001, 60, 1)])
@pytest.mark.parametrize("call", ["device", "host", "batch", "batch16", "budget"])
def test_hubs_of_near_equal_degree_are_ranked_by_degree(n, hubs, times, call):
    # Degrees that share their leading 11 bits, falling with the id, over a row-block
    # border: ranked by id, every hub's row would hold the wrong hubs. The features
    # give a block's neighbours and its longest row, log2(1 + x) in fp32.
    import torch
    e = hubs_of_near_equal_degree(n, hubs, times)
    with tb.Counter() as c:
        base = 0
        if call == "device":
            d = torch.from_numpy(e.view(np.int64)).cuda()
            c.prepare_device(d.data_ptr(), d.numel(), n)
        elif call == "host":
            c.count_edges(e, n)
        elif call.startswith("batch"):  # after small graphs of 32 vertices: 14 and 12 bits of degree in the keys
            base = 15 if call == "batch16" else 2
            small = [tb.gen_er(32, 100, seed=i) for i in range(base)]
            off = np.append(100 * np.arange(base + 1), 100 * base + e.size).astype(np.uint64)
            c.count_batch(np.concatenate(small + [e]), off, np.array([32] * base + [n], dtype=np.uint32))
        else:
            c.set_stream_options("rows")
            c.set_device_budget(c.device_bytes(e.size, n) * 3 // 4)
            assert c.count_edges(e, n).stream_tier == 1
        f = c.block_features().astype(np.float64)[base:]
    nnz, longest = rows_in_degree_order(e, n)
    np.testing.assert_allclose(np.exp2(f[:, 1]) - 1, nnz, rtol=1e-5, atol=1e-5)
    np.testing.assert_allclose(np.exp2(f[:, 5]) - 1, longest, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("kind", ["sorted", "reversed", "one_hub", "self_loops"])
def test_degree_counting_of_skewed_input(kind):
    n = 30_000
    e = np.sort(tb.gen_chung_lu(n, 300_000, 2.0, 3000.0, seed=17))
    if kind == "reversed":
        e = (e << np.uint64(32)) | (e >> np.uint64(32))
    elif kind == "one_hub":  # half of all entries name one vertex
        e[::2] = (np.uint64(7) << np.uint64(32)) | (e[::2] & np.uint64(0xFFFFFFFF))
    elif kind == "self_loops":
        e[1::3] = (e[1::3] >> np.uint64(32)) * np.uint64((1 << 32) + 1)
    check(e, n)


@pytest.mark.parametrize("length, stride", [
    (257, 32), (512, 32), (513, 33), (1025, 200),  # heavy: masks of up to 7,676 blocks, one and more pieces
    (900, 1000),                                   # heavy: a hash
    (1025, 1000), (2049, 500),                     # wide: masks
    (1100, 1500), (8192, 200),                     # wide: a hash, five pieces
    (8193, 200), (9000, 190),                      # wide: searched in global memory
])
def test_heavy_and_wide_rows(length, stride):
    n = 2_000_000
    # The columns' own rows are short; a second fan over the same columns
    # gives the first one long common neighbourhoods.
    e = np.concatenate([fans([(length, 64, stride), (length, 64, stride)], n),
                        np.array([(0 << 32) | 2], dtype=np.uint64)])
    check(e, n, modes=("plain", "merge", "bitmap"), orders=("id",))


def test_long_rows_in_the_hub_builder():
    # Rows of more than 2,048 neighbours in merge blocks, whose candidates a
    # CTA lists together; hubs with longer rows than the tails that meet them.
    check(tb.gen_rmat(15, 24, seed=77), 1 << 15, modes=("merge", "plain"))


@pytest.mark.parametrize("size", [2, 17, 32, 33, 34, 70])
def test_groups_of_short_rows(size):
    # Cliques: rows of 0 .. size - 1 neighbours, in groups of four up to 32.
    i, j = np.triu_indices(size, 1)
    base = (np.arange(101, dtype=np.uint64) * np.uint64(size))[:, None]
    e = (((base + i.astype(np.uint64)) << np.uint64(32)) | (base + j.astype(np.uint64))).ravel()
    check(e, 101 * size, modes=("bitmap", "merge"))


def test_batch_of_tiny_graphs():
    # Several graphs in every tile of entries and in every group of rows.
    rng = np.random.default_rng(4)
    nodes = rng.integers(1, 40, 3000).astype(np.uint32)
    sizes = rng.integers(0, 60, 3000)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    e = np.concatenate([(rng.integers(0, k, s).astype(np.uint64) << np.uint64(32)) | rng.integers(0, k, s).astype(np.uint64)
                        for k, s in zip(nodes, sizes)]).astype(np.uint64)
    want = [oracle.count(e[int(a):int(b)], int(k))[0] if b > a else 0 for a, b, k in zip(off[:-1], off[1:], nodes)]
    for mode in ("plain", "bitmap", "merge"):
        with tb.Counter(dispatch=mode) as c:
            got, r = c.count_batch(e, off, nodes)
            assert got.tolist() == want and r.triangles == sum(want)


def test_batch_in_chunks():
    # 17 million entries: four chunks of whole graphs, ranked and built one after
    # the other; graphs without entries or vertices at their borders, a graph
    # longer than a chunk, and a last chunk without entries.
    parts, nodes = [], []
    for i in range(40):
        n = 500 + 37 * i
        nodes += [n, 0, 3]
        parts += [tb.gen_er(n, 100_000 + 997 * i, seed=i), [], []]
    nodes += [40_000, 1, 0, 5] + [2_000] * 3 + [7, 0]
    parts += [tb.gen_rmat(15, 280, seed=9), [], [], []] + [tb.gen_er(2_000, 1_000_000, seed=s) for s in (1, 2, 3)] + [[], []]
    parts = [np.asarray(p, dtype=np.uint64) for p in parts]
    off = np.concatenate([[0], np.cumsum([p.size for p in parts])]).astype(np.uint64)
    assert off[-1] > 4 << 22
    want = [oracle.count(p, k)[0] if p.size else 0 for p, k in zip(parts, nodes)]
    for mode in ("plain", "merge"):
        with tb.Counter(dispatch=mode) as c:
            for _ in range(2):
                got, r = c.count_batch(np.concatenate(parts), off, nodes)
                assert got.tolist() == want and r.triangles == sum(want)


@pytest.mark.parametrize("length", [3, 4, 5, 31, 32, 33, 64, 65, 255, 256])
def test_merge_with_long_neighbour_rows(length):
    # A row of `length` blocks over neighbours whose rows are a few times longer
    # than its tail: searched in either direction.
    n = 200_000
    cols = np.uint64(40) + np.uint64(32) * np.arange(length, dtype=np.uint64)
    e = [(np.uint64(1) << np.uint64(32)) | cols]
    for i, c in enumerate(cols):  # every neighbour's row: the tail and up to 8 times as many others
        far = np.uint64(40 + 32 * length) + np.uint64(64) * np.arange((i % 9) * (length - i), dtype=np.uint64)
        e += [(c << np.uint64(32)) | cols[i + 1:], (c << np.uint64(32)) | far[far < n]]
    check(np.concatenate(e), n, modes=("merge", "bitmap"), orders=("id",))


@pytest.mark.parametrize("model", ["kernels", "queue"])
@pytest.mark.parametrize("engine", ["tcgen05", "mma_sync"])
@pytest.mark.parametrize("n", [10_000, 300_000])  # from 245,633 vertices on: the wide rows' kernel too
def test_launch_counts_are_the_launches(model, engine, n):
    # The counting launch captured into a graph: its kernel nodes and their grids.
    import ctypes

    import torch
    cu = ctypes.CDLL("libcuda.so.1")
    e = tb.gen_er(n, 3 * n, seed=n)
    d = torch.from_numpy(e.view(np.int64)).cuda()
    side = torch.cuda.Stream()
    with tb.Counter() as c:
        c.set_stream(side.cuda_stream)
        c.set_tuning(launch_model=model)
        c.set_tile_engine(engine)
        c.prepare_device(d.data_ptr(), d.numel(), n)
        c.launch_count()
        side.synchronize()
        stream, graph, num = ctypes.c_void_p(side.cuda_stream), ctypes.c_void_p(), ctypes.c_size_t()
        assert cu.cuStreamBeginCapture_v2(stream, 1) == 0
        c.launch_count()
        assert cu.cuStreamEndCapture(stream, ctypes.byref(graph)) == 0
        assert cu.cuGraphGetNodes(graph, None, ctypes.byref(num)) == 0
        nodes = (ctypes.c_void_p * num.value)()
        assert cu.cuGraphGetNodes(graph, nodes, ctypes.byref(num)) == 0
        kernels = ctas = 0
        for node in nodes:
            kind, params = ctypes.c_int(), (ctypes.c_uint32 * 32)()
            assert cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
            if kind.value != 0:  # CU_GRAPH_NODE_TYPE_KERNEL
                continue
            assert cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), params) == 0
            kernels += 1
            ctas += params[2] * params[3] * params[4]  # the grid follows the function's pointer
        assert cu.cuGraphDestroy(graph) == 0
        r = c.read_count()
        assert (r.count_kernels, r.blocks_of_threads) == (kernels, ctas)
        assert kernels == {"kernels": 4, "queue": 2}[model] + (n > 245_632)
        c.set_stream(0)
