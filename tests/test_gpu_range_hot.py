"""Range batches whose boxes lie together: the few units they meet are swept in slices.

Offsets, ids in order, coordinates and the counts per level equal the level-synchronous launches'; no tolerance
is involved. The batches are on either side of where slices start (tasks of 128 queries).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _answer(tb, h, Q):
    r = h.query_batch(tb.QueryType.RANGE, Q, tb.Mode.EXACT, flags=tb.WANT_VALS)
    return (r.offsets.numpy().copy(), r.ids.numpy().copy(), r.vals.numpy().copy()), h.level_counts(), h.group_counts()


@pytest.fixture(scope="module", params=[3, 4, 8, 12])
def env(request, tb, cuda):
    h = tb.QueryHandler.generate(300_000, request.param, 1.0, 100.0, False, 3, (10, 10), 3, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    return h, h.decode_points(np.arange(300_000))[0]


@pytest.mark.parametrize("nq,launches", [(127, 3), (512, 4), (1025, 4), (2500, 4)])
def test_boxes_at_one_place(tb, env, nq, launches):
    h, pts = env
    rng = np.random.default_rng(nq)
    ext = pts.max(0) - pts.min(0)
    spread = pts[rng.integers(0, len(pts), nq)]
    same = np.repeat(pts[7:8], nq, 0)
    near = pts[7] + 0.002 * ext * rng.normal(0, 1, spread.shape)
    mixed = np.where((np.arange(nq) % 3 == 0)[:, None], same, spread)
    for c, w in ((same, 0.05), (near, 0.03), (mixed, 0.04), (spread, 0.01)):
        Q = np.ascontiguousarray(np.concatenate([c - w * ext, c + w * ext], 1))
        h.query_batch(tb.QueryType.RANGE, Q, tb.Mode.EXACT, flags=tb.WANT_VALS)
        before = tb.kernel_launches()
        got = _answer(tb, h, Q)
        assert tb.kernel_launches() - before == launches
        h.set_launch_shapes([0] * 3, [99] * 3)
        want = _answer(tb, h, Q)
        h.set_launch_shapes([0] * 3, [100] * 3)
        assert all(np.array_equal(a, b) for a, b in zip(got[0], want[0]))
        assert got[1:] == want[1:]
