"""KNN batches the sweep cannot bound take the walk, without runs of the sweep that cannot succeed.

K above what a probe selects from, and K above the points of the clusters a probe reads where no node
holds K points (small fan-outs): the answer is the FP64 brute force's, and a warm batch takes at most the
launches of one prepared sweep beyond the walk's.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _launches(tb, h, P, K, flags=0):
    h.query_batch(tb.QueryType.POINT, P, tb.Mode.EXACT, K=K, flags=flags)
    before = tb.kernel_launches()
    r = h.query_batch(tb.QueryType.POINT, P, tb.Mode.EXACT, K=K, flags=flags)
    return tb.kernel_launches() - before, r


@pytest.mark.parametrize("N,ratios,K,beyond", [(600_000, (4, 3), 200, 0), (60_000, (4, 3), 600, 0), (60_000, (4, 3), 2048, 0),
                                               (60_000, (60, 20), 2049, 0), (1200, (4, 3), 600, 0)])
def test_walk_or_sweep_at_once(tb, oracle_mod, cuda, N, ratios, K, beyond):
    h = tb.QueryHandler.generate(N, 3, 1.0, 100.0, False, len(ratios) + 1, ratios, 9, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    pts, ids = h.decode_points(np.arange(N))
    P = np.ascontiguousarray(pts[::N // 40] + 0.25)
    b = oracle_mod.brute_query(pts, ids, oracle_mod.KNN, P, K=K)
    walk, _ = _launches(tb, h, P, K, tb.WANT_LEVELS)
    got, r = _launches(tb, h, P, K)
    assert np.array_equal(r.ids.numpy(), b.ids) and np.array_equal(r.dist2.numpy(), b.dist2)
    assert got <= walk + beyond, (got, walk)


def test_one_unbounded_query_of_a_batch(tb, oracle_mod, cuda):
    """Among queries the sweep bounds: the batch takes the walk, and the next one sweeps again."""
    N = 400_000
    h = tb.QueryHandler.generate(N, 3, 1.0, 100.0, False, 3, (4, 3), 9, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    pts, ids = h.decode_points(np.arange(N))
    P = np.ascontiguousarray(pts[:300] + 0.25)
    few = oracle_mod.brute_query(pts, ids, oracle_mod.KNN, P, K=5)
    one = oracle_mod.brute_query(pts, ids, oracle_mod.KNN, P[200:201], K=900)
    K = np.full(300, 5, np.uint32)
    K[200] = 900
    for _ in range(3):
        r = h.query_batch(tb.QueryType.POINT, P, tb.Mode.EXACT, K=K)
        offs, got = r.offsets.numpy().astype(np.int64), r.ids.numpy()
        assert np.array_equal(np.diff(offs), K)
        assert np.array_equal(got[offs[200]:offs[201]], one.ids)
        for q in (0, 199, 201, 299):
            assert np.array_equal(got[offs[q]:offs[q + 1]], few.query(q))
    launches, r = _launches(tb, h, P, 5)
    assert launches == 5 and np.array_equal(r.ids.numpy(), few.ids)
