"""Device memory of the sweeps: what one query asks for is not reserved for all, and a batch whose sweep
finds no memory is answered all the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _index(tb, D, N, ratios, seed=3):
    h = tb.QueryHandler.generate(N, D, 1.0, 100.0, False, len(ratios) + 1, ratios, seed, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    return h, h.decode_points(np.arange(N))[0]


def _range(tb, h, Q, flags=0):
    r = h.query_batch(tb.QueryType.RANGE, Q, tb.Mode.EXACT, flags=flags)
    return r.offsets.numpy().copy(), r.ids.numpy().copy()


def _levels(tb, h, Q):
    H = h.info()["height"]
    h.set_launch_shapes([0] * H, [99] * H)
    try:
        return _range(tb, h, Q)
    finally:
        h.set_launch_shapes([0] * H, [100] * H)


def _same(got, want):
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


def test_one_wide_box_among_a_million(tb, cuda):
    h, pts = _index(tb, 2, 400_000, (20, 20, 10))
    rng = np.random.default_rng(1)
    c = pts[rng.integers(0, len(pts), 1_000_000)]
    Q = np.ascontiguousarray(np.concatenate([c - 1e-3, c + 1e-3], 1))
    lo, hi = pts.min(0), pts.max(0)
    Q[77] = np.concatenate([lo, [hi[0], 0.5 * (lo[1] + hi[1])]])  # hundreds of segments
    want = _levels(tb, h, Q)
    held = tb.lib().tblaeq_live_device_bytes()
    for _ in range(2):
        _same(_range(tb, h, Q), want)
    assert tb.lib().tblaeq_live_device_bytes() - held < 4 << 30
    assert want[0][78] - want[0][77] > 100_000
    few = np.ascontiguousarray(Q[70:90])
    want = _levels(tb, h, few)
    for _ in range(20):  # past the batches that run level by level
        _same(_range(tb, h, few), want)


@pytest.mark.parametrize("nth", [1, 2, 3, 4])
def test_range_without_memory_for_the_sweep(tb, cuda, nth):
    h, pts = _index(tb, 8, 30_000, (40, 20, 10))
    c = pts[:50]
    Q = np.ascontiguousarray(np.concatenate([c - 20.0, c + 20.0], 1))
    want = _levels(tb, h, Q)  # every buffer but the sweep's own four
    tb.lib().tblaeq_debug_fail_alloc_after(nth)
    try:
        _same(_range(tb, h, Q), want)
    finally:
        tb.lib().tblaeq_debug_fail_alloc_after(0)
    for _ in range(20):
        _same(_range(tb, h, Q), want)


def _knn(tb, h, P, K):
    r = h.query_batch(tb.QueryType.POINT, P, tb.Mode.EXACT, K=K)
    return r.offsets.numpy().copy(), r.ids.numpy().copy(), r.dist2.numpy().copy()


def _brute(oracle_mod, pts, ids, P, K):
    b = oracle_mod.brute_query(pts, ids, oracle_mod.KNN, np.ascontiguousarray(P), K=K)
    return b.offsets, b.ids, b.dist2


def _equal(got, want):
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_ties_of_one_batch_are_not_reserved_for_the_next(tb, oracle_mod, cuda):
    """3,000 points at one distance: a second run holds them, and the next batch's first; 100,000 other queries take no more for it."""
    X = np.full((6000, 4), 7.0, np.float32)
    X[3000:] += np.random.default_rng(0).uniform(5, 20, (3000, 4)).astype(np.float32)
    h, _ = tb.QueryHandler.build(X, height=3, ratios=(50, 10), iters=3, seed=1)
    h.prepare_for_query(tb.LevelPolicy.L0)
    pts, ids = h.decode_points(np.arange(6000))
    ties = np.full((33, 4), 7.0)
    other = np.ascontiguousarray(X[np.random.default_rng(1).integers(3000, 6000, 100_000)] + 0.25)
    want = _brute(oracle_mod, pts, ids, ties, 12)
    small = _brute(oracle_mod, pts, ids, other[:50], 100)
    start = tb.lib().tblaeq_live_device_bytes()
    for runs in (2, 1):
        _equal(_knn(tb, h, ties, 12), want)
        assert h.knn_batch_info()["runs"] == runs
    got = _knn(tb, h, other, 100)
    assert tb.lib().tblaeq_live_device_bytes() - start < 4 << 30
    _equal((got[0][:51], got[1][:5000], got[2][:5000]), small)


@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("nth", [2, 4, 6])
def test_knn_without_memory_for_the_sweep(tb, oracle_mod, cuda, nth, learned):
    """A refused allocation asks for a smaller batch (which callers split), a single query takes the walk."""
    h, pts = _index(tb, 8, 30_000, (40, 20, 10))
    ids = h.decode_points(np.arange(len(pts)))[1]
    if learned:
        h.scorer_train(np.ascontiguousarray(pts[:256] + 0.3), K=10, max_samples=2000, epochs=1, seed=1)
    P = np.ascontiguousarray(pts[:200] + 0.5)
    want = _brute(oracle_mod, pts, ids, P, 10)
    _range(tb, h, np.ascontiguousarray(np.concatenate([P, P], 1)))  # the workspace shared with range batches
    one = _brute(oracle_mod, pts, ids, P[:1], 10)
    tb.lib().tblaeq_debug_fail_alloc_after(nth)  # the first is the staged K
    try:
        _equal(_knn(tb, h, P, 10), want)
    finally:
        tb.lib().tblaeq_debug_fail_alloc_after(0)
    info = h.knn_batch_info()
    assert info["traversals"] == 2 and "KNN sweep" in info["split_reason"]
    _equal(_knn(tb, h, P[:1], 10), one)
    _equal(_knn(tb, h, P, 10), want)


def test_serving_admission_counts_the_sweep(tb, cuda):
    """A lane's slots follow its memory budget: 2,000 KNN requests of K = 2,000 hold 258 MB of candidates
    alone, so 64 MiB admit fewer than 700 at once."""
    h, pts = _index(tb, 6, 60_000, (60, 20, 5))
    n = 2000
    rows = np.ascontiguousarray(np.concatenate([pts[:n] + 0.1, np.zeros((n, 6))], 1))
    with tb.Server(h, max_batch=n, memory_budget=64 << 20, learned=False, lanes=2) as srv:
        for wave in range(3):
            srv.stats(reset=True)
            srv.replay(np.zeros(n, np.int32), rows, np.full(n, 2000, np.uint32), np.zeros(n))
            assert srv.wait_idle()
            s = srv.stats()
            assert s["completed"] == n and s["failed"] == 0
            assert wave == 0 or s["max_batch"] < 700


@pytest.mark.parametrize("D", [5, 8])
def test_index_without_memory_for_the_sweep_arrays(tb, oracle_mod, cuda, D):
    """What only the sweeps read is optional: an index whose last uploads are refused prepares and answers
    by the level-synchronous launches."""
    lib, N = tb.lib(), 20_000

    def make():
        return tb.QueryHandler.generate(N, D, 1.0, 100.0, False, 4, (40, 20, 5), 3, 2.5)

    h = make()
    at = lib.tblaeq_live_device_bytes()
    h.prepare_for_query(tb.LevelPolicy.L0)
    whole = lib.tblaeq_live_device_bytes() - at
    pts, ids = h.decode_points(np.arange(N))
    P = np.ascontiguousarray(pts[:60] + 0.5)
    Q = np.ascontiguousarray(np.concatenate([P - 12.0, P + 12.0], 1))
    want, near = _levels(tb, h, Q), _brute(oracle_mod, pts, ids, P, 9)
    h.close()
    failed = served = 0
    for nth in range(1, 200):
        g = make()
        at = lib.tblaeq_live_device_bytes()
        lib.tblaeq_debug_fail_alloc_after(nth)
        try:
            g.prepare_for_query(tb.LevelPolicy.L0)
        except tb.TblaeqError as e:
            assert e.code == 4 and lib.tblaeq_live_device_bytes() == at
            failed += 1
            continue
        finally:
            lib.tblaeq_debug_fail_alloc_after(0)
        held = lib.tblaeq_live_device_bytes() - at
        if held == whole:  # every allocation was granted
            break
        assert held < whole
        _same(_range(tb, g, Q), want)
        _equal(_knn(tb, g, P, 9), near)
        served += 1
        g.close()
    assert failed >= 10 and served >= 10
