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
