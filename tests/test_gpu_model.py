"""The learned dispatcher's GPU kernels (tribit_model_*) against the CPU float64
restatement in oracle/mlp.py, and exactness of counts under learned dispatch."""
import numpy as np
import pytest

import oracle
from oracle import mlp
import tribit_b200 as tb

pytestmark = pytest.mark.gpu


def _data(rows, seed=0):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(rows, 16)).astype(np.float32) * rng.uniform(0.5, 4, size=16).astype(np.float32) + 3
    y = np.stack([x[:, 0] + 0.5 * x[:, 1], np.abs(x[:, 2]) * 0.7 - x[:, 3], x[:, 4] * x[:, 5] * 0.1], 1)
    return x, (y + 10).astype(np.float32)


def _norm(x, y):
    return np.concatenate([x.mean(0), x.std(0) + 1e-3, y.mean(0), y.std(0) + 1e-3]).astype(np.float32)


def test_gradients_match_cpu_float64():
    x, y = _data(700)
    with tb.Counter() as c:
        c.model_init(_norm(x, y), seed=3)
        p = c.model_params(effective=True)
        # BF16 weights: every weight the kernels use is representable in BF16
        w = np.concatenate([p[:1024], p[1088:5184], p[5248:5440]])
        assert np.array_equal(w, (w.view(np.uint32) & 0xFFFF0000).view(np.float32))
        g, loss = c.model_gradients(x, y)
        _, want_loss, want = mlp.forward_backward(p, _norm(x, y), x, y)
    assert abs(loss - want_loss) <= 1e-4 * abs(want_loss)
    scale = np.abs(want).max()
    assert np.abs(g - want).max() <= 1e-4 * scale, np.abs(g - want).max() / scale
    # per-block relative agreement where gradients are not tiny
    big = np.abs(want) > 1e-3 * scale
    assert np.median(np.abs(g[big] - want[big]) / np.abs(want[big])) < 1e-4


def test_predictions_match_cpu():
    x, y = _data(300, seed=1)
    with tb.Counter() as c:
        c.model_init(_norm(x, y), seed=5)
        got = c.model_predict(x)
        want = mlp.predict(c.model_params(effective=True), _norm(x, y), x)
    np.testing.assert_allclose(got, want, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("rows", [1, 7, 8, 9, 32, 33, 296 * 32, 296 * 32 + 1, 20011])
def test_passes_at_group_and_tile_edges(rows):
    # 8 rows a warp, 32-row gradient tiles, one more tile a CTA past 296 of
    # them. A 64-term fp32 sum is off by at most 64 * 2^-24 = 4e-6 of its
    # terms' magnitudes; three such layers each way stay well below 1e-4 of
    # the largest value.
    x, y = _data(max(rows, 4), seed=rows)
    norm = _norm(x, y)
    x, y = x[:rows], y[:rows]
    with tb.Counter() as c:
        c.model_init(norm, seed=11)
        p = c.model_params(effective=True)
        pred = c.model_predict(x)
        g, loss = c.model_gradients(x, y)
        again, _ = c.model_gradients(x, y)
    _, want_loss, want = mlp.forward_backward(p, norm, x, y)
    want_pred = mlp.predict(p, norm, x)
    assert np.abs(pred - want_pred).max() <= 1e-4 * np.abs(want_pred).max()
    assert abs(loss - want_loss) <= 1e-4 * want_loss
    assert np.abs(g - want).max() <= 1e-4 * np.abs(want).max()
    np.testing.assert_array_equal(g, again)  # summed in a fixed order


def test_training_reduces_loss_and_save_load_roundtrip(tmp_path):
    x, y = _data(20000, seed=2)
    with tb.Counter() as c:
        c.model_init(_norm(x, y), seed=7)
        _, loss0 = c.model_gradients(x, y)
        loss = c.model_train(x, y, epochs=25, batch=1024, lr=3e-3, seed=1)
        _, loss1 = c.model_gradients(x, y)
        assert loss1 < 0.15 * loss0, (loss0, loss1)
        assert abs(loss - loss1) < 0.5 * loss0
        path = str(tmp_path / "m.bin")
        c.save_model(path)
        pred = c.model_predict(x[:100])
    with tb.Counter() as c2:
        c2.load_model(path)
        np.testing.assert_array_equal(c2.model_predict(x[:100]), pred)


@pytest.mark.parametrize("rows", [2, 15, 16, 17, 24, 25, 511, 512, 513, 2048, 2049])
def test_passes_where_rows_a_warp_and_split_change(rows):
    # One row a warp and 8-row sums up to 512 rows, two rows a warp up to 2,048;
    # tolerances as above.
    x, y = _data(max(rows, 4), seed=rows)
    norm = _norm(x, y)
    x, y = x[:rows], y[:rows]
    with tb.Counter() as c:
        c.model_init(norm, seed=17)
        p = c.model_params()
        eff = c.model_params(effective=True)
        g, loss = c.model_gradients(x, y)
        train_loss = c.model_train(x, y, epochs=1, batch=rows, lr=1e-3, seed=1)
        got = c.model_params()
    _, want_loss, want = mlp.forward_backward(eff, norm, x, y)
    assert abs(loss - want_loss) <= 1e-4 * want_loss and abs(train_loss - want_loss) <= 1e-4 * want_loss
    assert np.abs(g - want).max() <= 1e-4 * np.abs(want).max()
    # The first Adam step moves a parameter by lr g / (|g| + 1e-8): by lr where |g| is
    # 1e-5 and more, and a parameter of up to 0.5 rounds that by 2^-25, 3e-5 of it.
    big = np.abs(want) > max(1e-2 * np.abs(want).max(), 1e-5)
    np.testing.assert_allclose((got - p)[big], -1e-3 * np.sign(want)[big], rtol=2e-3)


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_loss_of_many_rows_keeps_its_digits(seed):
    # Thousands of warps add their sums of squares: in double. What is left is the
    # result's own rounding (2^-24) and the mean of the rows' fp32 errors, whose
    # signs vary (each at most about 64 * 2^-24 of the row, over 65,521 rows).
    x, y = _data(65521, seed=seed)
    norm = _norm(x, y)
    with tb.Counter() as c:
        c.model_init(norm, seed=seed)
        p = c.model_params(effective=True)
        losses = [c.model_gradients(x, y)[1] for _ in range(5)]
    want = mlp.forward_backward(p, norm, x, y)[1]
    assert max(abs(loss - want) for loss in losses) <= 3e-7 * want, [loss / want - 1 for loss in losses]


def test_small_training_batches_are_spread_over_ctas():
    from tests.test_gpu_batch import _launches
    x, y = _data(320, seed=4)
    with tb.Counter() as c:
        c.model_init(_norm(x, y), seed=3)
        for kernel in ("k_fwd_bwd", "k_wgrad"):  # 32 rows: a row a warp of 8, 8-row sums, added by the step
            grids = _launches(lambda: c.model_train(x, y, epochs=1, batch=32), kernel)
            assert all(g == 4 for g in grids), (kernel, grids)


def _epoch_order(rows, seed):
    """Rows in the order an epoch takes them: a shuffle driven by tb_rand (csrc/gen.h)."""
    u = np.uint64

    def mix(z):
        z = z + u(0x9E3779B97F4A7C15)
        z = (z ^ (z >> u(30))) * u(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> u(27))) * u(0x94D049BB133111EB)
        return z ^ (z >> u(31))

    with np.errstate(over="ignore"):
        i = np.arange(rows, dtype=u)
        r = mix(mix(np.full(rows, seed, dtype=u)) ^ (i * u(0xD6E8FEB86659FD93)))
    order = np.arange(rows)
    for k in range(rows - 1, 0, -1):
        j = int(r[k]) % (k + 1)
        order[k], order[j] = order[j], order[k]
    return order


@pytest.mark.parametrize("rows,batch", [(18944, 9473), (19000, 10000), (25000, 16384), (9473 + 31, 9473)])
def test_training_with_a_shorter_last_batch(rows, batch):
    # The last batch's gradient takes more CTAs than the full one's (9,471 rows
    # 296, 9,473 rows 149). Two Adam steps against float64: a step moves a
    # parameter by lr (less near zero gradients), so parameters agree to a
    # hundredth of that where the gradient is above the fp32 sums' error (at
    # most 1e-4 of the largest, as above) by a factor of 100. Biases and weights
    # of the second step see bf16-rounded weights, whose rounding may go the
    # other way for a few: the median is compared, and all within one step.
    x, y = _data(rows, seed=rows)
    norm, lr = _norm(x, y), 1e-3
    with tb.Counter() as c:
        c.model_init(norm, seed=13)
        p = c.model_params().astype(np.float64)
        eff = c.model_params(effective=True)
        loss = c.model_train(x, y, epochs=1, batch=batch, lr=lr, seed=5)
        got = c.model_params()
        eff2 = c.model_params(effective=True)
    order = _epoch_order(rows, 5)
    weight = np.r_[0:1024, 1088:5184, 5248:5440]
    m, v, want_loss, big = np.zeros_like(p), np.zeros_like(p), 0.0, np.ones(p.size, dtype=bool)
    for step, part in enumerate((order[:batch], order[batch:]), 1):
        _, part_loss, g = mlp.forward_backward(eff, norm, x[part], y[part])
        want_loss += part_loss * len(part) / rows
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - lr * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
        big &= np.abs(g) > 1e-2 * np.abs(g).max()
        eff = p.astype(np.float32)
        bits = eff[weight].view(np.uint32)
        eff[weight] = ((bits + 0x7FFF + ((bits >> 16) & 1)) & np.uint32(0xFFFF0000)).view(np.float32)
    assert abs(loss - want_loss) <= 1e-3 * want_loss
    err = np.abs(got - p)
    assert big.sum() > 100 and np.median(err[big]) <= 0.01 * lr, np.median(err[big]) / lr
    assert np.quantile(err[big], 0.99) <= lr
    assert np.isfinite(eff2).all()


def test_learned_dispatch_without_model_is_an_error():
    with tb.Counter(dispatch="learned") as c:
        with pytest.raises(tb.TribitError) as ex:
            c.count_edges(tb.gen_rmat(10, 8, seed=1), 1 << 10)
        assert ex.value.status == 11


def test_learned_dispatch_counts_exactly():
    graphs = [(1 << 14, tb.gen_rmat(14, 16, seed=41)), (7115, tb.gen_chung_lu(7115, 115300, 2.0, 1000.0, seed=1)),
              (20000, tb.gen_planted(200, 100, 0.3, 2, seed=8))]
    rng = np.random.default_rng(0)
    for seed in (1, 2, 3):
        with tb.Counter(dispatch="learned") as c:
            norm = np.concatenate([np.zeros(16), np.ones(16), np.zeros(3), np.ones(3)]).astype(np.float32)
            c.model_init(norm, seed=seed)
            p = c.model_params()
            p[5440:5443] = rng.normal(size=3)  # push the argmin around
            c.set_model_params(p)
            for n, e in graphs:
                assert c.count_edges(e, n).triangles == oracle.count(e, n)[0]


def test_learned_dispatch_keeps_bit_tiles_to_blocks_that_fit_one_tile():
    # A network that rates bit tiles cheapest everywhere may still only send
    # the row blocks whose columns span 1..64 blocks to them.
    import torch
    e = tb.gen_rmat(15, 16, seed=43)
    n = 1 << 15
    d = torch.from_numpy(e.view(np.int64)).cuda()
    with tb.Counter(dispatch="learned") as c:
        norm = np.concatenate([np.zeros(16), np.ones(16), np.zeros(3), np.ones(3)]).astype(np.float32)
        c.model_init(norm, seed=1)
        p = c.model_params()
        p[5440:5443] = [-1e4, 0.0, 1e4]  # predicted: MMA cheapest, then bitmap
        c.set_model_params(p)
        r = c.prepare_device(d.data_ptr(), d.numel(), n)
        span = np.exp2(c.block_features()[:, 13]) - 1
        eligible = int(((span > 0.5) & (span <= 64.5)).sum())
        mma, bitmap, merge = r.row_blocks_by_variant
        assert 0 < mma <= eligible and merge == 0 and bitmap > 0
        c.launch_count()
        assert c.read_count().triangles == oracle.count(e, n)[0]


def test_block_features_and_times():
    import torch
    e = tb.gen_rmat(16, 16, seed=9)
    n = 1 << 16
    want = oracle.count(e, n)[0]
    d = torch.from_numpy(e.view(np.int64)).cuda()
    with tb.Counter() as c:
        c.prepare_device(d.data_ptr(), d.numel(), n)
        f = c.block_features()
        assert f.shape == ((n + 31) // 32, 16) and np.isfinite(f).all()
        for v in tb.VARIANTS:
            t, tri, ms = c.block_times(v)
            assert tri == want and ms > 0
            assert t.shape[0] == f.shape[0] and (t >= 0).all() and t.sum() > 0
        c.launch_count()
        assert c.read_count().triangles == want
