"""Sizes at which a sweep's launch meets a limit of the grid."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_range_over_many_upper_nodes(tb, cuda):
    """270,000 parents, four a block, are more blocks than a y axis has (65,535). Wide boxes have more segments
    than the gather orders and end in the level launches, narrow ones sweep."""
    N = 4_320_000
    h = tb.QueryHandler.generate(N, 1, 1.0, 100.0, False, 4, (2, 4, 2), 5, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    assert 270_000 in h.info()["meshSizes"]
    rng = np.random.default_rng(2)
    c = h.decode_points(rng.integers(0, N, 300))[0]
    for widest in (1e-5, 1e-2):
        hw = np.exp(rng.uniform(np.log(1e-6), np.log(widest), c.shape)) * 100
        Q = np.ascontiguousarray(np.concatenate([c - hw, c + hw], 1))
        before = tb.kernel_launches()
        r = h.query_batch(tb.QueryType.RANGE, Q, tb.Mode.EXACT)
        launches = tb.kernel_launches() - before
        got = r.offsets.numpy().copy(), r.ids.numpy().copy(), h.level_counts()
        assert launches == 4 or widest > 1e-5
        h.set_launch_shapes([0] * 4, [99] * 4)
        r = h.query_batch(tb.QueryType.RANGE, Q, tb.Mode.EXACT)
        h.set_launch_shapes([0] * 4, [100] * 4)
        assert np.array_equal(got[0], r.offsets.numpy()) and np.array_equal(got[1], r.ids.numpy())
        assert got[2] == h.level_counts() and got[0][-1] >= 300


def test_knn_over_many_queries(tb, cuda):
    """More queries than the bound's grid has rows for (65,535 of 256)."""
    N, nq = 2000, 65535 * 256 + 77
    X = np.random.default_rng(1).permutation(np.linspace(1.0, 100.0, N)).astype(np.float32)[:, None]
    h, _ = tb.QueryHandler.build(X, height=3, ratios=(20, 10), iters=3, seed=1)
    h.prepare_for_query(tb.LevelPolicy.L0)
    pts, ids = h.decode_points(np.arange(N))
    order = np.argsort(pts[:, 0], kind="stable")
    x, ids = pts[order, 0], ids[order]
    assert np.all(np.diff(x) > 0)
    P = np.random.default_rng(3).uniform(0.0, 101.0, nq)
    right = np.clip(np.searchsorted(x, P), 1, N - 1)
    d = np.stack([P - x[right - 1], P - x[right]], 1)
    d2 = d * d  # one dimension: the squared distance is this one rounded product
    tie = (d2[:, 0] == d2[:, 1]) & (ids[right - 1] > ids[right])
    near = np.where((d2[:, 1] < d2[:, 0]) | tie, right, right - 1)
    r = h.query_batch(tb.QueryType.POINT, P[:, None], tb.Mode.EXACT, K=1)
    assert r.total == nq and np.array_equal(r.offsets.numpy(), np.arange(nq + 1, dtype=np.uint64))
    assert np.array_equal(r.dist2.numpy(), d2.min(1))
    assert np.array_equal(r.ids.numpy(), ids[near])


def test_range_results_beyond_32_bits(tb, cuda):
    """More than 2^32 results: told at once, as the level-synchronous launches do, and the handle goes on."""
    N = 500_000
    h = tb.QueryHandler.generate(N, 3, 1.0, 100.0, False, 4, (100, 50, 20), 5, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    wide = np.repeat(np.array([[-1e3] * 3 + [1e3] * 3]), 2 ** 32 // N + 2, axis=0)
    with pytest.raises(tb.TblaeqError, match="2\\^32") as e:
        h.query_batch(tb.QueryType.RANGE, wide, tb.Mode.EXACT)
    runs = ctypes.c_uint64()
    assert tb.lib().tblaeq_last_batch_runs(h._h, ctypes.byref(runs)) == 0
    assert e.value.code == 4 and runs.value == 1
    r = h.query_batch(tb.QueryType.RANGE, wide[:2], tb.Mode.EXACT)
    assert r.total == 2 * N
