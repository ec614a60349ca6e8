"""Batched counting, CUDA-graph replay and tuning: per-graph counts exact
against the oracle, unchanged by replay and by every tuning setting."""
import numpy as np
import pytest
import torch

import oracle
import tribit_b200 as tb

pytestmark = pytest.mark.gpu


def test_gen_batch_shape_and_determinism():
    e, off, nn = tb.gen_batch(64, seed=5, min_n=64, max_n=4096)
    assert off[0] == 0 and off[-1] == e.size and nn.min() >= 64 and nn.max() <= 4096
    e2, off2, nn2 = tb.gen_batch(64, seed=5, min_n=64, max_n=4096)
    assert np.array_equal(e, e2) and np.array_equal(off, off2) and np.array_equal(nn, nn2)
    for g in range(64):
        part = e[off[g]:off[g + 1]]
        assert int((part >> np.uint64(32)).max()) < nn[g] and int((part & np.uint64(0xFFFFFFFF)).max()) < nn[g]


@pytest.mark.parametrize("model", ["kernels", "queue"])
@pytest.mark.parametrize("dispatch", ["plain", "bitmap", "merge", "mma"])
def test_batch_counts_and_graph_replay(dispatch, model):
    # Per-graph counts under both launch models: one persistent kernel per
    # variant, or the row pieces and hub pass in one queue-driven kernel.
    e, off, nn = tb.gen_batch(96, seed=7, min_n=64, max_n=8192)
    want = np.array([oracle.count(e[off[g]:off[g + 1]], int(nn[g]))[0] for g in range(96)], dtype=np.uint64)
    with tb.Counter(dispatch=dispatch) as c:
        c.set_tuning(0, 64, 64.0, launch_model=model)
        got, r = c.count_batch(e, off, nn)
        np.testing.assert_array_equal(got, want)
        assert r.triangles == int(want.sum())
        c.capture_count()
        for _ in range(3):
            c.launch_count()
            np.testing.assert_array_equal(c.batch_counts(96), want)
            assert c.read_count().triangles == int(want.sum())


def test_tuning_settings_keep_counts_exact():
    n = 1 << 15
    e = tb.gen_rmat(15, 16, seed=3)
    want = oracle.count(e, n)[0]
    d = torch.from_numpy(e.view(np.int64)).cuda()
    with tb.Counter() as c:
        c.prepare_device(d.data_ptr(), d.numel(), n)
        for model in tb.LAUNCH_MODELS:
            for ctas in (1, 4, 7):
                for width in (32, 96, 256):
                    for tile in (0.0, 64.0, 1e30):
                        c.set_tuning(ctas, width, tile, launch_model=model)
                        c.launch_count()
                        assert c.read_count().triangles == want, (model, ctas, width, tile)
        best = c.autotune(reps=1)
        assert best.count_ms > 0 and best.piece_width in (32, 64, 128)
        t = c.tuning()
        assert (t.ctas_per_sm, t.piece_width, t.launch_model) == (best.ctas_per_sm, best.piece_width,
                                                                  best.launch_model)
        c.launch_count()
        assert c.read_count().triangles == want
        c.capture_count()
        c.launch_count()
        assert c.read_count().triangles == want
    with pytest.raises(tb.TribitError):
        with tb.Counter() as c:
            c.set_tuning(4, 48, 64.0)  # not a multiple of 32


@pytest.mark.parametrize("dispatch", ["learned", "plain", "merge", "bitmap", "mma"])
def test_queue_kernel_matches_oracle(dispatch):
    # The queue launch model on graphs that reach every one of its phases:
    # hub and row pieces (RMAT), dense tiles (cliques), and heavy rows, one CTA
    # each (a dense Erdos-Renyi graph: 4,209 oriented rows span more than 256
    # bit blocks).
    import os
    from tests.graphs import clique
    cases = [(1 << 16, tb.gen_rmat(16, 16, seed=61)),
             (64 * 40, np.concatenate([clique(40, base=40 * k) for k in range(64)])),
             (16000, tb.gen_er(16000, 4_800_000, seed=9))]
    model = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tribit_b200", "models",
                         "dispatch_mlp.bin")
    with tb.Counter(dispatch=dispatch) as c:
        if dispatch == "learned":
            c.load_model(model)
        c.set_tuning(0, 64, 64.0, launch_model="queue")
        for n, e in cases:
            want = oracle.count(e, n)
            r = c.count_edges(e, n)
            assert (r.triangles, r.edges) == want, (dispatch, n)
            for _ in range(2):
                c.launch_count()
                assert c.read_count().triangles == want[0]


def _launches(call, kernel):
    """CTAs of the launches of `kernel` (a part of its name) by call(), as the profiler lists them. A session may miss
    some or all of them, so tests only say what none of those seen may be."""
    import json
    import os
    import tempfile

    from torch.profiler import ProfilerActivity, profile
    for _ in range(4):
        torch.zeros(1, device="cuda")
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            call()
            torch.cuda.synchronize()
        with tempfile.TemporaryDirectory() as d:
            prof.export_chrome_trace(os.path.join(d, "trace.json"))
            with open(os.path.join(d, "trace.json")) as f:
                events = json.load(f)["traceEvents"]
        grids = [e["args"]["grid"][0] for e in events if e.get("cat") == "kernel" and kernel in e["name"]]
        if grids:
            return grids
    return []


@pytest.mark.parametrize("before, after, E", [(0, 0, 1 << 20), (0, 0, 3_000_017), (3, 40, 9_000_017), (40, 0, 9_000_001)])
def test_batch_that_one_graph_dominates(before, after, E):
    # The large graph is copied in pieces, its degrees counted as they land: no degree pass covers it whole.
    rng = np.random.default_rng(E + before)
    nodes = [int(k) for k in rng.integers(2, 60, before)] + [50_000] + [int(k) for k in rng.integers(2, 60, after)]
    parts = [tb.gen_er(k, 100, seed=i) if k < 60 else tb.gen_er(k, E, seed=i) for i, k in enumerate(nodes)]
    off = np.concatenate([[0], np.cumsum([p.size for p in parts])]).astype(np.uint64)
    e = torch.from_numpy(np.concatenate(parts).view(np.int64)).pin_memory().numpy().view(np.uint64)
    want = [oracle.count(p, k)[0] for p, k in zip(parts, nodes)]
    with tb.Counter() as c:
        for _ in range(2):
            got, r = c.count_batch(e, off, np.asarray(nodes, dtype=np.uint32))
            assert got.tolist() == want and r.triangles == sum(want)
        # A CTA takes 4,096 entries, up to 444 CTAs a launch; pieces are of 2^20 entries and more.
        pieces = max(1, min(8, e.size >> 20))
        if pieces > 1:
            piece = -(-e.size // pieces) * 3 // 2
            assert all(g <= -(-piece // 4096) for g in
                       _launches(lambda: c.count_batch(e, off, np.asarray(nodes, dtype=np.uint32)), "k_degree"))
        e[-1 if not after else int(off[before + 1]) - 1] = (1 << 32) | 50_000  # in its last piece
        with pytest.raises(tb.TribitError) as ex:
            c.count_batch(e, off, np.asarray(nodes, dtype=np.uint32))
        assert ex.value.status == 5


def test_batch_with_a_graph_that_presorts():
    # 2^27 entries: 128 copies of a graph's, each in another order, before and after small graphs.
    base = tb.gen_rmat(15, 32, seed=3)
    rng = np.random.default_rng(2)
    big = np.concatenate([np.roll(base, int(rng.integers(base.size))) for _ in range((1 << 27) // base.size)])
    small = [tb.gen_er(500, 3_000, seed=i) for i in range(6)]
    parts, nodes = small[:3] + [big] + small[3:], [500] * 3 + [1 << 15] + [500] * 3
    assert big.size == 1 << 27
    off = np.concatenate([[0], np.cumsum([p.size for p in parts])]).astype(np.uint64)
    want = [oracle.count(base if p is big else p, k) for p, k in zip(parts, nodes)]
    e = np.concatenate(parts)
    nodes, got = np.asarray(nodes, dtype=np.uint32), []
    with tb.Counter() as c:
        # Entries that go straight to their rows take a thousand a CTA and more: only the small graphs' do.
        assert all(g < 100 for g in _launches(lambda: got.append(c.count_batch(e, off, nodes)), "k_row_fill_entries"))
        got.append(c.count_batch(e, off, nodes))
        for counts, r in got:
            assert counts.tolist() == [t for t, _ in want] and r.edges == sum(m for _, m in want)
