"""Row construction of the preprocessing (a counting sort of the oriented
entries by their lower endpoint, then a sort + dedup of each row): rows of every
sorting class -- lane groups and the warp's register sorts (up to 1,024
entries), a CTA's column bitmaps and its bitonic sorts in shared memory and in
global scratch (longer) -- with duplicated and reversed entries, against the oracle."""
import numpy as np
import pytest

import oracle
import tribit_b200 as tb
from tests.graphs import clique, comb, wheel

pytestmark = pytest.mark.gpu


def noisy(e, seed, copies=3):
    """e with every entry repeated, half of the copies reversed, shuffled."""
    rng = np.random.default_rng(seed)
    a, b = e >> np.uint64(32), e & np.uint64(0xFFFFFFFF)
    rev = (b << np.uint64(32)) | a
    parts = [e] + [np.where(rng.random(e.size) < 0.5, rev, e) for _ in range(copies - 1)]
    out = np.concatenate(parts)
    rng.shuffle(out)
    return out


@pytest.mark.parametrize("n", [1500, 5000, 20000])
def test_long_rows_in_id_order(n):
    # In id order the wheel's hub (vertex 0) owns one row of n - 1 entries
    # (x 3 with the copies): the CTA sorts, in shared memory and in scratch.
    e = noisy(wheel(n), seed=n)
    with tb.Counter(order="id") as c:
        r = c.count_edges(e, n)
        assert (r.triangles, r.edges) == (n - 1, 2 * (n - 1))


def test_clique_rows_of_every_class_in_degree_order():
    # A 1,100-clique under degree order: rows of 0..1,099 entries, x 2 with the
    # copies, so every warp class and the CTA class occur.
    k = 1100
    e = noisy(clique(k), seed=7, copies=2)
    with tb.Counter() as c:
        r = c.count_edges(e, k)
        assert (r.triangles, r.edges) == (comb(k), k * (k - 1) // 2)


@pytest.mark.parametrize("order", ["degree", "id"])
def test_random_graph_with_duplicates_matches_oracle(order):
    n = 3000
    e = noisy(tb.gen_chung_lu(n, 60_000, 2.0, 1500.0, seed=11), seed=12)
    want, m = oracle.count(e, n)
    for mode in ("plain", "merge"):
        with tb.Counter(order=order, dispatch=mode) as c:
            r = c.count_edges(e, n)
            assert (r.triangles, r.edges) == (want, m), (order, mode)


def test_self_loops_and_empty_rows():
    # Self-loops are dropped; vertices without edges leave empty rows.
    e = np.concatenate([clique(40, base=100), np.array([(5 << 32) | 5, (7 << 32) | 7], dtype=np.uint64)])
    with tb.Counter() as c:
        r = c.count_edges(e, 1000)
        assert (r.triangles, r.edges) == (comb(40), 40 * 39 // 2)


def fans(rows, n):
    """In id order, vertex 2 i owns a row of rows[i] = (length, first, stride)
    columns, and the columns of each row are joined in a path."""
    parts = []
    for i, (length, first, stride) in enumerate(rows):
        cols = first + stride * np.arange(length, dtype=np.uint64)
        assert cols[-1] < n and first > 2 * len(rows)
        parts.append((np.uint64(2 * i) << np.uint64(32)) | cols)
        parts.append((cols[:-1] << np.uint64(32)) | cols[1:])
    return np.concatenate(parts)


@pytest.mark.parametrize("name, n, rows", [
    # each class of the warp and lane-group sorts and the first CTA row, one block to many
    ("classes", 40000, [(k, 2000 + 7 * k, 1 + k % 37) for k in (1, 2, 8, 9, 16, 17, 31, 32, 33, 64, 65, 128, 129, 256,
                                                               257, 512, 513, 1023, 1024, 1025)]),
    # a column window exactly, one block past it (then bitonic), and rows of several windows
    ("windows", 3_000_000, [(1025, 32, 360), (1440, 32, 256), (1441, 32, 256), (2048, 32, 190), (2049, 64, 1000),
                            (8192, 64, 300), (8193, 96, 299)]),
    # rows of too few entries for their windows: bitonic in shared memory and in global scratch
    ("bitonic", 9_000_000, [(1100, 1000, 8000), (2047, 1000, 4000), (8192, 1001, 1000), (9000, 1002, 999)]),
])
def test_rows_of_every_length_and_span(name, n, rows):
    e = noisy(fans(rows, n), seed=len(rows), copies=1 if name == "classes" else 2)
    want, m = oracle.count(e, n)
    with tb.Counter(order="id") as c:
        r = c.count_edges(e, n)
        assert (r.triangles, r.edges) == (want, m)


def test_rows_between_long_runs_of_empty_rows():
    # 2^20 ids between one clique and the next, a long row among short ones,
    # and rows that end at and cross the emitting warps' shares.
    n = 5 << 20
    e = np.concatenate([clique(70, base=k << 20) for k in range(5)] + [fans([(3000, 1 << 19, 5), (64, 1 << 19, 64)], n)])
    want, m = oracle.count(e, n)
    for order in ("id", "degree"):
        with tb.Counter(order=order) as c:
            r = c.count_edges(noisy(e, seed=3, copies=2), n)
            assert (r.triangles, r.edges) == (want, m)


@pytest.mark.parametrize("log_n", [20, 23])
def test_presorted_fill_keeps_its_ctas_together_on_sparse_rows(log_n):
    # 2^27 entries presort their keys. With fewer than 32 entries a row the fill's
    # CTAs take them in launch order, a few tiles of 1,024 each; with more they all
    # stride through all of them.
    import torch

    from tests.test_gpu_batch import _launches
    n, E = 1 << log_n, 1 << 27
    base = tb.gen_rmat(16, 16, seed=8)
    want = oracle.count(base, 1 << 16)
    d = torch.from_numpy(base.view(np.int64)).cuda().repeat(E // base.size)
    with tb.Counter() as c:
        r = c.count_edges_device(d.data_ptr(), E, n)
        assert (r.triangles, r.edges) == want
        grids = _launches(lambda: c.count_edges_device(d.data_ptr(), E, n), "k_row_fill(")
        assert all((8 * 1024 * g >= E) == (E < 32 * n) for g in grids), grids
