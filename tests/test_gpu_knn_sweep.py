"""Exact KNN batches as a probe and one sweep over the clusters, at the edges of its kernels.

Results must equal the FP64 brute force's, ids and squared distances bit for bit, so no tolerance is
involved. Sizes sit at the edges of the tiles: query words of 32 and CTAs of 256 queries, padded
dimensions (odd D and each multiple of four), indexes of two and three meshes, K from 0 past the
points a probe can bound (those batches take the level-synchronous walk).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _index(tb, D, N=30000, ratios=(40, 20, 10), seed=3):
    h = tb.QueryHandler.generate(N, D, 1.0, 100.0, False, len(ratios) + 1, ratios, seed, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    pts, ids = h.decode_points(np.arange(N))
    return h, pts, ids


def _check(tb, oracle_mod, h, pts, ids, P, K):
    r = h.query_batch(tb.QueryType.POINT, P, tb.Mode.EXACT, K=K)
    offs, got, d2 = r.offsets.numpy(), r.ids.numpy(), r.dist2.numpy()
    Kq = np.broadcast_to(np.asarray(K), (len(P),))
    assert np.array_equal(np.diff(offs.astype(np.int64)), np.minimum(Kq, len(pts)))
    for k in np.unique(Kq):
        sel = np.nonzero(Kq == k)[0]
        if k == 0:
            continue
        b = oracle_mod.brute_query(pts, ids, oracle_mod.KNN, np.ascontiguousarray(P[sel]), K=int(k))
        for j, q in enumerate(sel):
            assert np.array_equal(got[offs[q]:offs[q + 1]], b.query(j)), (int(k), int(q))
            assert np.array_equal(d2[offs[q]:offs[q + 1]], b.dist2[b.offsets[j]:b.offsets[j + 1]]), (int(k), int(q))


@pytest.mark.parametrize("D", [1, 2, 3, 5, 7, 9, 13, 17, 22, 28])
def test_padded_dimensions(tb, oracle_mod, cuda, D):
    h, pts, ids = _index(tb, D)
    rng = np.random.default_rng(D)
    P = np.ascontiguousarray(pts[rng.integers(0, len(pts), 40)] + rng.normal(0, 0.7, (40, D)))
    _check(tb, oracle_mod, h, pts, ids, P, np.where(np.arange(40) % 2 == 0, 1, 13).astype(np.uint32))


@pytest.mark.parametrize("nq", [1, 31, 32, 33, 128, 129, 256, 257, 513])
def test_query_word_and_block_edges(tb, oracle_mod, cuda, nq):
    h, pts, ids = _index(tb, 6)
    rng = np.random.default_rng(nq)
    P = np.ascontiguousarray(pts[rng.integers(0, len(pts), nq)] + rng.normal(0, 0.7, (nq, 6)))
    _check(tb, oracle_mod, h, pts, ids, P, 7)


@pytest.mark.parametrize("ratios", [(25,), (400,), (50, 10), (3, 3, 3, 3)])
def test_heights_and_cluster_sizes(tb, oracle_mod, cuda, ratios):
    h, pts, ids = _index(tb, 4, N=12000, ratios=ratios)
    rng = np.random.default_rng(len(ratios))
    P = np.ascontiguousarray(pts[rng.integers(0, len(pts), 50)] + rng.normal(0, 0.5, (50, 4)))
    _check(tb, oracle_mod, h, pts, ids, P, np.where(np.arange(50) % 2 == 0, 3, 60).astype(np.uint32))


def test_extreme_queries_and_k(tb, oracle_mod, cuda):
    """K of 0, 1, more than a wave's points and more than the index; queries on a point, far outside
    and at coordinates no float square holds (those batches take the level-synchronous walk)."""
    h, pts, ids = _index(tb, 5, N=3000, ratios=(30, 10))
    P = np.ascontiguousarray(np.concatenate([pts[:4], pts[4:8] + 1e3, pts[8:12]]))
    for K in (1, 700, 2049, 5000):
        _check(tb, oracle_mod, h, pts, ids, P, K)
    _check(tb, oracle_mod, h, pts, ids, P, np.array([0, 1, 2, 3, 0, 50, 0, 9, 4, 4, 0, 0], dtype=np.uint32))
    far = P.copy()
    far[3] = 1e19
    _check(tb, oracle_mod, h, pts, ids, far, 5)
    _check(tb, oracle_mod, h, pts, ids, P, 5)


def test_equal_distances_grow_the_candidates(tb, oracle_mod, cuda):
    """Thousands of points at one distance of the query: the candidate slots grow, ties go to the
    smaller id."""
    X = np.full((6000, 4), 7.0, np.float32)
    X[3000:] += np.random.default_rng(0).uniform(5, 20, (3000, 4)).astype(np.float32)
    h, _ = tb.QueryHandler.build(X, height=3, ratios=(50, 10), iters=3, seed=1)
    h.prepare_for_query(tb.LevelPolicy.L0)
    pts, ids = h.decode_points(np.arange(6000))
    P = np.ascontiguousarray(np.repeat(np.array([[7.0, 7.0, 7.0, 7.0]]), 33, axis=0))
    _check(tb, oracle_mod, h, pts, ids, P, 12)


@pytest.mark.parametrize("D,nq", [(4, 33), (12, 128), (20, 130), (28, 257)])
@pytest.mark.parametrize("offset,scale", [(0.0, 1e-12), (3e4, 1.0), (-2e6, 1e3)])
def test_bound_products_far_from_the_origin(tb, oracle_mod, cuda, D, nq, offset, scale):
    """Two clouds far apart, both far from the origin or tiny: the bound's products must lose no cluster."""
    rng = np.random.default_rng(D + nq)
    X = rng.normal(0, scale, (6000, D)) + offset
    X[3000:] += 40 * scale
    h, _ = tb.QueryHandler.build(X.astype(np.float32), height=3, ratios=(20, 10), iters=3, seed=1)
    h.prepare_for_query(tb.LevelPolicy.L0)
    pts, ids = h.decode_points(np.arange(6000))
    P = np.ascontiguousarray(pts[rng.integers(0, 6000, nq)] + rng.normal(0, 0.3 * scale, (nq, D)))
    _check(tb, oracle_mod, h, pts, ids, P, 9)


@pytest.mark.parametrize("nq", [900, 1776, 1777, 2500])
def test_finish_of_few_and_many_candidates(tb, oracle_mod, cuda, nq):
    """Either side of the finish's forms: K from none past the candidates a CTA counts, ties included."""
    h, pts, ids = _index(tb, 4, N=8000, ratios=(40, 10))
    rng = np.random.default_rng(nq)
    P = np.ascontiguousarray(pts[rng.integers(0, len(pts), nq)] + rng.normal(0, 0.5, (nq, 4)))
    P[::7] = P[0]
    _check(tb, oracle_mod, h, pts, ids, P, rng.choice(np.array([0, 1, 31, 127, 240, 256, 512, 700], np.uint32), nq))
