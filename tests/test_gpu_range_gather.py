"""The range gather with queries of one, some and many segments, in batches on either side of its two forms
(large blocks that share a query up to 592 queries, small ones above), against the level-synchronous launches.

Equality of offsets, ids in order and coordinates; no tolerance is involved.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(tb, h, Q):
    r = h.query_batch(tb.QueryType.RANGE, Q, tb.Mode.EXACT, flags=tb.WANT_VALS)
    return r.offsets.numpy().copy(), r.ids.numpy().copy(), r.vals.numpy().copy()


@pytest.mark.parametrize("D,ratios", [(2, (20, 20, 10)), (4, (20, 40))])
@pytest.mark.parametrize("nq", [1, 3, 148, 149, 592, 593, 700])
def test_shares(tb, cuda, D, ratios, nq):
    N = 150_000
    h = tb.QueryHandler.generate(N, D, 1.0, 100.0, False, len(ratios) + 1, ratios, 11, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    pts, _ = h.decode_points(np.arange(N))
    rng = np.random.default_rng(nq)
    c = pts[rng.integers(0, N, nq)]
    ext = pts.max(0) - pts.min(0)
    Q = np.concatenate([c - 0.004 * ext, c + 0.004 * ext], 1)
    for q in range(0, nq, max(1, nq // 5)):  # a few with hundreds of segments and up to 100,000 results
        w = (0.3 + 0.1 * rng.random()) * ext
        Q[q] = np.concatenate([c[q] - w, c[q] + w])
    Q = np.ascontiguousarray(Q)
    H = len(ratios) + 1
    h.query_batch(tb.QueryType.RANGE, Q, tb.Mode.EXACT, flags=tb.WANT_VALS)
    before = tb.kernel_launches()
    got = _run(tb, h, Q)
    assert tb.kernel_launches() - before == 3
    h.set_launch_shapes([0] * H, [99] * H)
    want = _run(tb, h, Q)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
