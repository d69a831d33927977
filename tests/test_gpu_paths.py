"""Which path a batch takes, and the level-synchronous walk's options on the walk itself.

The sweeps' tests compare the default dispatch with the level-synchronous launches: this file asserts, by
launch counts, that the default batches of those sizes do sweep (three launches for range, four with slices, five for KNN, six
above 512 queries, two more with a scorer) and which fall back. Options that only the walk knows (refinement, point groups in
its point pass, wave 1) are tested with per-level counts asked for, which the sweeps don't serve: they
change the walk's work and none of its results.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _index(tb, D, N=30000, ratios=(40, 20, 10), seed=3):
    h = tb.QueryHandler.generate(N, D, 1.0, 100.0, False, len(ratios) + 1, ratios, seed, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    return h, h.decode_points(np.arange(N))[0]


def _boxes(pts, n, seed, lo=0.01, hi=0.3):
    rng = np.random.default_rng(seed)
    c = pts[rng.integers(0, len(pts), n)]
    hw = np.exp(rng.uniform(np.log(lo), np.log(hi), c.shape)) * (pts.max(0) - pts.min(0))
    return np.ascontiguousarray(np.concatenate([c - hw, c + hw], 1))


def _launches(tb, h, qtype, Q, K=0, flags=0):
    """Of a warm batch: the first one may grow a workspace and run again."""
    h.query_batch(qtype, Q, tb.Mode.EXACT, K=K, flags=flags)
    before = tb.kernel_launches()
    h.query_batch(qtype, Q, tb.Mode.EXACT, K=K, flags=flags)
    return tb.kernel_launches() - before


@pytest.mark.parametrize("D", [1, 2, 3, 4, 5, 7, 8, 9, 13, 16, 17, 22, 28])
def test_range_dimensions_sweep(tb, cuda, D):
    h, pts = _index(tb, D)
    Q = _boxes(pts, 70, D, 0.02, 0.6 if D > 8 else 0.2)
    assert _launches(tb, h, tb.QueryType.RANGE, Q, flags=tb.WANT_VALS) == 3
    assert _launches(tb, h, tb.QueryType.RANGE, Q, flags=tb.WANT_LEVELS) > 3


@pytest.mark.parametrize("nq,launches", [(1, 3), (1025, 3), (3000, 3), (8192, 3), (8193, 4)])  # above: a scan of the counts
def test_range_batches_sweep(tb, cuda, nq, launches):
    h, pts = _index(tb, 8, N=60000, ratios=(100, 33, 5))
    assert _launches(tb, h, tb.QueryType.RANGE, _boxes(pts, nq, nq)) == launches


@pytest.mark.parametrize("D,ratios,sweeps", [(8, (25,), True), (3, (25,), True), (8, (500,), True), (3, (512, 4), True),
                                             (3, (700, 4), False), (4, (50, 10), True), (6, (3, 3, 3, 3, 3), True),
                                             (8, (20, 3, 2, 2, 2), True), (5, (100, 65, 7), True)])
def test_range_heights_and_clusters_sweep(tb, oracle_mod, cuda, D, ratios, sweeps):
    """At dimensions whose hits leave in row order, clusters above 512 points run level by level."""
    h, pts = _index(tb, D, N=12288, ratios=ratios)  # 24 clusters of 512
    Q = _boxes(pts, 90, len(ratios))
    assert (_launches(tb, h, tb.QueryType.RANGE, Q, flags=tb.WANT_VALS) == 3) == sweeps
    r = h.query_batch(tb.QueryType.RANGE, Q, tb.Mode.EXACT)
    b = oracle_mod.brute_query(pts, h.decode_points(np.arange(12288))[1], oracle_mod.RANGE, Q)
    assert np.array_equal(r.offsets.numpy(), b.offsets)


@pytest.mark.parametrize("D,nq", [(1, 40), (5, 1), (6, 513), (8, 40), (9, 40), (28, 40)])
def test_knn_sweeps(tb, cuda, D, nq):
    h, pts = _index(tb, D)
    P = np.ascontiguousarray(pts[:nq] + 0.3)
    assert _launches(tb, h, tb.QueryType.POINT, P, 7) == 5 + (nq > 512)
    assert _launches(tb, h, tb.QueryType.POINT, P, 7, tb.WANT_LEVELS) > 7
    h.scorer_train(np.ascontiguousarray(pts[:256] + 0.3), K=10, max_samples=2000, epochs=1, seed=1)
    assert _launches(tb, h, tb.QueryType.POINT, P, 7) == 7 + (nq > 512)


def _check_walk(tb, h, P, Kq, brute):
    r = h.query_batch(tb.QueryType.POINT, P, tb.Mode.EXACT, K=Kq, flags=tb.WANT_LEVELS)
    offs, got, d2 = r.offsets.numpy(), r.ids.numpy(), r.dist2.numpy()
    for kv, b in brute.items():
        for j, q in enumerate(np.nonzero(Kq == kv)[0]):
            assert np.array_equal(got[offs[q]:offs[q + 1]], b.query(j)), q
            assert np.array_equal(d2[offs[q]:offs[q + 1]], b.dist2[b.offsets[j]:b.offsets[j + 1]]), q
    return h.knn_counters()


@pytest.fixture(scope="module", params=[5, 8, 16])
def walk(request, tb, oracle_mod, cuda):
    h, pts = _index(tb, request.param, N=100_000)
    ids = h.decode_points(np.arange(len(pts)))[1]
    rng = np.random.default_rng(1)
    P = np.ascontiguousarray(pts[rng.integers(0, len(pts), 200)] + rng.normal(0, 1.0, (200, request.param)))
    Kq = np.where(np.arange(200) % 2 == 0, 10, 60).astype(np.uint32)
    brute = {kv: oracle_mod.brute_query(pts, ids, oracle_mod.KNN, np.ascontiguousarray(P[Kq == kv]), K=kv) for kv in (10, 60)}
    return h, P, Kq, brute


def test_walk_refinement(tb, walk):
    h, P, Kq, brute = walk
    rows = {}
    try:
        for stride in (0, 3, 16):
            h.set_knn_refine(stride)
            rows[stride] = _check_walk(tb, h, P, Kq, brute)["rows"]
    finally:
        h.set_knn_refine(16)
    assert len(set(rows.values())) == 3, rows


def test_walk_point_groups(tb, walk):
    h, P, Kq, brute = walk
    rows = {}
    try:
        for on in (True, False):
            h.set_point_groups(on)
            rows[on] = _check_walk(tb, h, P, Kq, brute)["rows"]
    finally:
        h.set_point_groups(True)
    grouped = h.info()["D"] in (4, 8, 16)
    assert rows[True] < rows[False] if grouped else rows[True] == rows[False], rows


def test_walk_wave_one(tb, walk):
    h, P, Kq, brute = walk
    rows = {}
    try:
        for scale in (0.5, 4.0, 64.0):
            h.set_knn_wave1(scale)
            rows[scale] = _check_walk(tb, h, P, Kq, brute)["rows1"]
    finally:
        h.set_knn_wave1(16.0)
    assert len(set(rows.values())) == 3, rows


@pytest.mark.parametrize("D,N,ratios,nq,sweeps", [(3, 1_000_000, (2, 2, 2), 1, False), (3, 1_000_000, (2, 2, 2), 3000, False),
                                                  (3, 500_000, (4, 4), 1, False), (3, 500_000, (4, 4), 600, True),
                                                  (3, 2_000_000, (5, 5, 3, 3), 700, False), (3, 1_000_000, (100, 2, 2), 1, True)])
def test_narrow_indexes(tb, cuda, D, N, ratios, nq, sweeps):
    """Small fan-outs over many nodes: the level-synchronous launches, with the sweep's results."""
    h, pts = _index(tb, D, N, ratios)
    Q = _boxes(pts, nq, 5, 0.001, 0.01)
    assert (_launches(tb, h, tb.QueryType.RANGE, Q) <= 4) == sweeps
    r = h.query_batch(tb.QueryType.RANGE, Q, tb.Mode.EXACT)
    offs, ids = r.offsets.numpy().astype(np.int64), r.ids.numpy()
    names = h.decode_points(np.arange(N))[1]
    for q in (0, nq // 2, nq - 1):
        inside = names[((pts >= Q[q, :D]) & (pts <= Q[q, D:])).all(1)]
        assert np.array_equal(np.sort(ids[offs[q]:offs[q + 1]]), np.sort(inside))


@pytest.mark.parametrize("N,ratios,nq,K,sweeps", [(500_000, (5, 5), 40, 165, False), (500_000, (5, 5), 40, 155, True),
                                                  (2_000_000, (3, 3, 3), 1, 2, False), (2_000_000, (3, 3, 3), 8, 2, True)])
def test_knn_paths_of_small_fan_outs(tb, oracle_mod, cuda, N, ratios, nq, K, sweeps):
    h, pts = _index(tb, 4, N, ratios)
    ids = h.decode_points(np.arange(N))[1]
    P = np.ascontiguousarray(pts[::N // nq][:nq] + 0.2)
    launches = _launches(tb, h, tb.QueryType.POINT, P, K)
    assert (launches <= 10) == sweeps  # five, and five more where slots grow
    r = h.query_batch(tb.QueryType.POINT, P, tb.Mode.EXACT, K=K)
    b = oracle_mod.brute_query(pts, ids, oracle_mod.KNN, P, K=K)
    assert np.array_equal(r.ids.numpy(), b.ids) and np.array_equal(r.dist2.numpy(), b.dist2)
