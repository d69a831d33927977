"""KNN batches whose queries lie together or far outside the data: a few clusters are reached by nearly all of
them, and are swept in slices.

Ids and squared distances equal the FP64 brute force's for a sample of the queries, and queries at one place
answer alike; no tolerance is involved. Sizes are on either side of where slices start (512 queries) and of
a slice's and a row's words.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(tb, oracle_mod, h, pts, ids, P, K, sample):
    r = h.query_batch(tb.QueryType.POINT, P, tb.Mode.EXACT, K=K)
    offs, got, d2 = r.offsets.numpy().astype(np.int64), r.ids.numpy(), r.dist2.numpy()
    assert np.array_equal(np.diff(offs), np.full(len(P), K))
    b = oracle_mod.brute_query(pts, ids, oracle_mod.KNN, np.ascontiguousarray(P[sample]), K=K)
    for j, q in enumerate(sample):
        assert np.array_equal(got[offs[q]:offs[q + 1]], b.query(j)), q
        assert np.array_equal(d2[offs[q]:offs[q + 1]], b.dist2[b.offsets[j]:b.offsets[j + 1]]), q
    return got.reshape(len(P), K)


@pytest.fixture(scope="module", params=[(3, (50, 20)), (8, (40, 20, 10)), (12, (40, 20)), (16, (40, 30))])
def env(request, tb, cuda):
    D, ratios = request.param
    h = tb.QueryHandler.generate(60_000, D, 1.0, 100.0, False, len(ratios) + 1, ratios, 3, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    pts, ids = h.decode_points(np.arange(60_000))
    return h, pts, ids


@pytest.mark.parametrize("nq", [512, 513, 1024, 1025, 1100, 3000])
def test_queries_at_one_place_and_far_away(tb, oracle_mod, env, nq):
    h, pts, ids = env
    rng = np.random.default_rng(nq)
    ext = pts.max(0) - pts.min(0)
    sample = np.unique(np.concatenate([[0, nq // 2, nq - 1], rng.integers(0, nq, 12)]))
    for P, K in ((pts[7] + 0.003 * ext * rng.normal(0, 1, (nq, pts.shape[1])), 30), (pts[:nq] + 3.0 * ext, 5),
                 (pts[:nq] - 100.0 * ext, 60)):
        _check(tb, oracle_mod, h, pts, ids, np.ascontiguousarray(P), K, sample)
    same = _check(tb, oracle_mod, h, pts, ids, np.repeat(pts[11:12] + 0.1, nq, 0), 17, sample[:1])
    assert np.all(same == same[0])


def test_every_cluster_reached_by_every_query(tb, oracle_mod, cuda):
    """No bound (K above the points a probe reads): slices of all clusters, none lost."""
    h = tb.QueryHandler.generate(30_000, 5, 1.0, 100.0, False, 3, (10, 30), 3, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    pts, ids = h.decode_points(np.arange(30_000))
    _check(tb, oracle_mod, h, pts, ids, np.ascontiguousarray(pts[:1100] + 0.2), 400, np.array([0, 31, 1024, 1099]))
