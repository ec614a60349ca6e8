"""Graphs counted in rank ranges (tribit_count_edges past the device budget)
against the oracle.

A context's device budget (tribit_set_device_budget) below what a one-piece
count needs (tribit_device_bytes) sends the count through the streamed path:
passes of the entries through the GPU to rank them, then either the rows tier
(each range's rows built in turn into one resident oriented graph, counted
once; up to four ranges filled from one more pass of the entries each, more
from host buckets of oriented keys) or the pairs tier (host buckets, one
device count per pair of ranges). The count and the undirected edge count
must equal the oracle's for every budget, tier, range bound and dispatcher,
and the context must stay usable for one-piece counts."""
import os

import numpy as np
import pytest

import oracle
import tribit_b200 as tb
from tests.graphs import clique, comb

pytestmark = pytest.mark.gpu

ROWS, PAIRS = 1, 2
MODEL = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tribit_b200", "models",
                     "dispatch_mlp.bin")

GRAPHS = [
    ("rmat16", 1 << 16, lambda: tb.gen_rmat(16, 16, seed=16)),
    ("chung_lu", 30000, lambda: tb.gen_chung_lu(30000, 300000, 2.1, 3000.0, seed=3)),
    ("planted", 40000, lambda: tb.gen_planted(400, 100, 0.3, 2, seed=4)),
]


def _schedule(r):
    return r.row_blocks, tuple(r.row_blocks_by_variant), r.hub_edges


@pytest.mark.parametrize("name,n,make", GRAPHS, ids=[g[0] for g in GRAPHS])
def test_streamed_counts_match_oracle(name, n, make):
    e = make()
    want = oracle.count(e, n)
    with tb.Counter() as c:
        need = c.device_bytes(e.size, n)
        r = c.count_edges(e, n)
        assert (r.triangles, r.edges) == want and r.stream_ranges == 1 and r.stream_tier == 0
        one_piece = _schedule(r)
        for frac in (0.8, 0.5, 0.35):
            c.set_device_budget(int(need * frac))
            try:
                r = c.count_edges(e, n)
            except tb.TribitError as ex:  # the smallest budget may fit neither tier on a small graph
                assert ex.status == 8 and frac < 0.5, (name, frac, str(ex))
                continue
            assert (r.triangles, r.edges) == want, (name, frac, r.stream_tier, r.stream_ranges)
            assert r.stream_tier in (ROWS, PAIRS)
            if r.stream_tier == ROWS:
                # The rows tier builds the one-piece oriented graph, range by
                # range; a small budget may leave no room for the hub in-lists,
                # and the dispatcher's merge blocks then go to the bitmap sweep.
                assert r.stream_tasks == 1 and r.row_blocks == one_piece[0], (name, frac)
                mma, bitmap, merge = one_piece[1]
                assert _schedule(r) == one_piece or (r.hub_edges == 0 and frac < 0.8 and
                                                     _schedule(r)[1] == (mma, bitmap + merge, 0)), (name, frac)
        # Rows tier in a few ranges (filled from the streamed entries) and in
        # many (from host buckets): the same graph again.
        c.set_device_budget(int(need * 0.8))
        kept = int(np.count_nonzero((e >> np.uint64(32)) != (e & np.uint64(0xffffffff))))
        seen = set()
        for parts in (3, 11):
            c.set_stream_options("rows", kept // parts)
            r = c.count_edges(e, n)
            assert (r.triangles, r.edges) == want and r.stream_tier == ROWS, (name, parts)
            assert r.stream_ranges >= parts and _schedule(r) == one_piece
            seen.add(r.stream_ranges)
        assert len(seen) == 2
        # The pairs tier at the same budgets.
        seen = set()
        for frac in (0.8, 0.6, 0.45):
            c.set_device_budget(int(need * frac))
            c.set_stream_options("pairs", 0)
            r = c.count_edges(e, n)
            assert (r.triangles, r.edges) == want, (name, frac, r.stream_ranges)
            assert r.stream_tier == PAIRS and r.stream_ranges > 1 and r.stream_tasks >= r.stream_ranges
            seen.add(r.stream_ranges)
        assert len(seen) >= 2  # smaller budgets cut more ranges
        c.set_stream_options("auto", 0)
        c.set_device_budget(0)
        r = c.count_edges(e, n)
        assert (r.triangles, r.edges) == want and r.stream_ranges == 1 and r.stream_tier == 0


@pytest.mark.parametrize("tier,parts", [("rows", 3), ("rows", 8), ("pairs", 0)])
@pytest.mark.parametrize("dispatch", ["learned", "merge", "bitmap", "mma"])
def test_streamed_counts_under_every_dispatcher(dispatch, tier, parts):
    n, e = 1 << 15, tb.gen_rmat(15, 16, seed=151)
    want = oracle.count(e, n)
    with tb.Counter(dispatch=dispatch) as c:
        if dispatch == "learned":
            c.load_model(MODEL)
        c.set_device_budget(int(c.device_bytes(e.size, n) * 0.5))
        c.set_stream_options(tier, e.size // parts if parts else 0)
        r = c.count_edges(e, n)
        assert (r.triangles, r.edges) == want and r.stream_ranges > 1
        assert r.stream_tier == (ROWS if tier == "rows" else PAIRS)


@pytest.mark.parametrize("tier,parts", [("rows", 2), ("rows", 9), ("pairs", 0)])
def test_streamed_counts_from_pinned_host_memory(tier, parts):
    # Pinned host entries are copied straight from the caller's buffer.
    import torch
    n, e = 1 << 16, tb.gen_rmat(16, 16, seed=61)
    pinned = torch.empty(e.size, dtype=torch.int64, pin_memory=True)
    pinned.numpy()[:] = e.view(np.int64)
    host = pinned.numpy().view(np.uint64)
    with tb.Counter() as c:
        c.set_device_budget(int(c.device_bytes(e.size, n) * 0.6))
        c.set_stream_options(tier, e.size // parts if parts else 0)
        r = c.count_edges(host, n)
        assert (r.triangles, r.edges) == oracle.count(e, n) and r.stream_ranges > 1


def test_rows_tier_leaves_the_graph_prepared():
    # After a rows-tier count the context holds the oriented graph: launching
    # the count again gives the same result, as after a one-piece count.
    n, e = 1 << 15, tb.gen_rmat(15, 16, seed=7)
    want = oracle.count(e, n)
    with tb.Counter() as c:
        c.set_device_budget(int(c.device_bytes(e.size, n) * 0.6))
        c.set_stream_options("rows", e.size // 4)
        r = c.count_edges(e, n)
        assert r.stream_tier == ROWS and (r.triangles, r.edges) == want
        for _ in range(3):
            c.launch_count()
            assert c.read_count().triangles == want[0]


def test_streamed_duplicates_self_loops_and_dense_blocks():
    # Duplicated and reversed entries land in their lower endpoint's bucket;
    # self-loops vanish; dense cliques give rows that reach other ranges and
    # rows long enough for the CTA sort.
    sizes = [40] * 60 + [200] * 6 + [1500]
    offs = np.cumsum([0] + sizes)
    e = np.concatenate([clique(k, base=int(o)) for k, o in zip(sizes, offs)])
    rev = (e << np.uint64(32)) | (e >> np.uint64(32))
    loops = (np.arange(50, dtype=np.uint64) << np.uint64(32)) | np.arange(50, dtype=np.uint64)
    noisy = np.concatenate([e, rev[::3], e[::5], loops])
    n = int(offs[-1])
    want = sum(comb(k) for k in sizes)
    with tb.Counter() as c:
        c.set_device_budget(int(c.device_bytes(noisy.size, n) * 0.5))
        for tier, bound in (("rows", noisy.size // 6), ("pairs", 0), ("auto", 0)):
            c.set_stream_options(tier, bound)
            r = c.count_edges(noisy, n)
            assert r.triangles == want and r.edges == e.size and r.stream_ranges >= 1, tier
            assert r.stream_tier in (ROWS, PAIRS)


def test_streamed_id_range_error_and_recovery():
    n, e = 1 << 14, tb.gen_rmat(14, 16, seed=3)
    bad = e.copy()
    bad[len(bad) // 2] = (5 << 32) | (1 << 20)
    with tb.Counter() as c:
        c.set_device_budget(int(c.device_bytes(e.size, n) * 0.5))
        for tier in ("rows", "pairs"):
            c.set_stream_options(tier, e.size // 3 if tier == "rows" else 0)
            with pytest.raises(tb.TribitError) as ex:
                c.count_edges(bad, n)
            assert ex.value.status == 5
            r = c.count_edges(e, n)
            assert (r.triangles, r.edges) == oracle.count(e, n) and r.stream_ranges > 1


def test_stream_option_errors():
    n, e = 1 << 14, tb.gen_rmat(14, 16, seed=5)
    with tb.Counter() as c:
        assert tb.lib.tribit_set_stream_options(c.handle, 7, 0) == 1  # no such tier
        c.set_device_budget(int(c.device_bytes(e.size, n) * 0.5))
        # A range bound at the longest row cannot hold that row with anything else.
        c.set_stream_options("rows", 1)
        with pytest.raises(tb.TribitError) as ex:
            c.count_edges(e, n)
        assert ex.value.status == 8
        c.set_stream_options("auto", 0)
        r = c.count_edges(e, n)
        assert (r.triangles, r.edges) == oracle.count(e, n)


@pytest.mark.parametrize("pinned", [False, True])
def test_streamed_rows_tier_on_a_million_vertices(pinned):
    # Megabyte-sized uploads of the row starts and ranks through the pinned
    # staging buffers, then pieces of the entries through the same buffers
    # (pageable input): every buffer is refilled only after its last copy.
    import torch
    n, e = 1 << 20, tb.gen_rmat(20, 16, seed=20)
    host = e
    if pinned:
        t = torch.empty(e.size, dtype=torch.int64, pin_memory=True)
        t.numpy()[:] = e.view(np.int64)
        host = t.numpy().view(np.uint64)
    with tb.Counter() as c:
        want = c.count_edges(e, n)
        for parts in (2, 6):
            c.set_device_budget(int(c.device_bytes(e.size, n) * 0.6))
            c.set_stream_options("rows", e.size // parts)
            r = c.count_edges(host, n)
            assert (r.triangles, r.edges) == (want.triangles, want.edges) and r.stream_tier == ROWS, parts
            assert _schedule(r)[:2] == _schedule(want)[:2]
            c.set_device_budget(0)
            c.set_stream_options("auto", 0)


def test_one_piece_count_in_the_least_memory():
    # Rows without degree-sized slots, 4 bytes an entry less: 8 bytes staged, 4
    # of rows, 8 of scratch, 4 + 8 of CSR and bit rows, 8 of hub in-lists, and
    # less than 1 of pieces and flags.
    n, E = 60_000, 1_000_000
    e = tb.gen_chung_lu(n, E, 2.1, 3000.0, seed=6)
    want = oracle.count(e, n)
    with tb.Counter() as c:
        need = c.device_bytes(E, n)
        assert (c.device_bytes(2 * E, n) - need) / E < 41
        for budget in (need, need + 2 * E, need + 4 * E, 0):
            c.set_device_budget(budget)
            r = c.count_edges(e, n)
            assert (r.triangles, r.edges, r.stream_ranges) == (*want, 1), budget
        c.set_device_budget(need - 4096)
        r = c.count_edges(e, n)
        assert (r.triangles, r.edges) == want and r.stream_tier in (ROWS, PAIRS)


@pytest.mark.parametrize("call", ["device", "prepare", "batch"])
def test_calls_that_only_compact_rows_leave_room_for(call):
    # All but a little more than the compact layout's device memory (33 bytes an
    # entry and 8 staged, see above) is taken by another allocation, so the
    # arena with degree-sized slots (4 bytes an entry more) cannot be had.
    import torch
    n, E = 1 << 20, 50_000_000
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randint(0, n, (2, E), generator=g, device="cuda", dtype=torch.int64)
    d = (x[0] << 32) | x[1]
    host = d.cpu().numpy().view(np.uint64) if call == "batch" else None
    off, nodes = np.array([0, E], dtype=np.uint64), np.array([n], dtype=np.uint32)

    def count(c):
        if call == "batch":
            per_graph, r = c.count_batch(host, off, nodes)
            return int(per_graph[0]), r.edges
        if call == "device":
            r = c.count_edges_device(d.data_ptr(), E, n)
        else:
            m = c.prepare_device(d.data_ptr(), E, n).edges
            c.launch_count()
            r = c.read_count()
            assert r.edges == m
        return r.triangles, r.edges

    with tb.Counter() as c:
        want = count(c)
        room = c.device_bytes(0, n) + (42 if call == "batch" else 34) * E
    del x
    with tb.Counter() as c:
        c.count_edges(tb.gen_er(100, 300, seed=1), 100)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        other = torch.empty(free - room, dtype=torch.uint8, device="cuda")
        try:
            assert torch.cuda.mem_get_info()[0] < room + E
            assert count(c) == want
            left = torch.cuda.mem_get_info()[0]
            assert count(c) == want and torch.cuda.mem_get_info()[0] == left  # the arena is kept
        finally:
            del other
            torch.cuda.empty_cache()


def test_device_bytes_from_the_presort_size_on():
    # 2^27 entries and more: 8 bytes staged, 8 of rows in degree-sized slots, 16
    # of keys in the presort's two buffers, 4 + 8 of CSR and bit rows, 8 of hub
    # in-lists, and less than 1 of pieces, flags and digit counts.
    with tb.Counter() as c:
        per_entry = (c.device_bytes(1 << 28, 1 << 20) - c.device_bytes(1 << 27, 1 << 20)) / (1 << 27)
        assert 52 < per_entry < 53
