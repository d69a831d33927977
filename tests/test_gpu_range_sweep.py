"""Exact range batches as one sweep, at the edges of its kernels and against the level-synchronous launches.

The sweep must return what those launches return: ids in the same order, coordinates, offsets and the
counts per level (all compared for equality, no tolerance), at every padded dimension, unit and word
edge, index height and cluster size, and with boxes that no float holds (infinite, NaN, inverted).
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


def _answer(tb, h, Q, flags):
    r = h.query_batch(tb.QueryType.RANGE, Q, tb.Mode.EXACT, flags=flags)
    vals = r.vals.numpy().copy() if r.vals is not None else None
    return r.offsets.numpy().copy(), r.ids.numpy().copy(), vals, h.level_counts(), h.group_counts()


def _check(tb, h, Q, flags=0):
    H = h.info()["height"]
    got = _answer(tb, h, Q, flags)
    h.set_launch_shapes([0] * H, [99] * H)  # chosen shapes: the level-synchronous launches
    try:
        want = _answer(tb, h, Q, flags)
    finally:
        h.set_launch_shapes([0] * H, [100] * H)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert flags == 0 or np.array_equal(got[2], want[2])
    assert got[3] == want[3] and got[4] == want[4]
    return got


@pytest.mark.parametrize("D", [1, 2, 3, 4, 5, 7, 8, 9, 13, 16, 17, 22, 28])
def test_dimensions(tb, cuda, D):
    h, pts = _index(tb, D)
    got = _check(tb, h, _boxes(pts, 70, D, 0.02, 0.6 if D > 8 else 0.2), tb.WANT_VALS)
    assert got[0][-1] >= 70  # a box around a point holds it


@pytest.mark.parametrize("nq", [1, 31, 32, 33, 127, 1024, 1025, 3000])
def test_query_blocks(tb, cuda, nq):
    h, pts = _index(tb, 8, N=60000, ratios=(100, 33, 5))
    _check(tb, h, _boxes(pts, nq, nq))


@pytest.mark.parametrize("D,ratios", [(8, (25,)), (3, (25,)), (8, (500,)), (3, (700, 4)), (4, (50, 10)), (6, (3, 3, 3, 3, 3)),
                                      (8, (20, 3, 2, 2, 2)), (5, (100, 65, 7))])
def test_heights_and_cluster_sizes(tb, cuda, D, ratios):
    h, pts = _index(tb, D, N=12000, ratios=ratios)
    _check(tb, h, _boxes(pts, 90, len(ratios)), tb.WANT_VALS)


def test_boxes_no_float_holds(tb, cuda):
    h, pts = _index(tb, 8)
    Q = _boxes(pts, 40, 1)
    Q[0, :8], Q[0, 8:] = -np.inf, np.inf          # every point
    Q[1, 3] = np.nan
    Q[2, 8 + 5] = np.nan
    Q[3] = np.concatenate([Q[3, 8:], Q[3, :8]])   # inverted
    Q[4, :8], Q[4, 8:] = -1e300, 1e300
    Q[5, :8] = Q[5, 8:] = pts[17]                 # a point
    Q[6, :8], Q[6, 8:] = 1e30, 2e30               # far outside
    got = _check(tb, h, Q)
    n = np.diff(got[0].astype(np.int64))
    assert n[0] == n[4] == len(pts) and n[1] == n[2] == n[3] == n[6] == 0 and n[5] >= 1


def test_many_results_per_query_fall_back_and_recover(tb, cuda):
    """Queries with more segments than the gather orders run level by level, and a later small batch
    sweeps again; results grow past the first workspace on the way."""
    h, pts = _index(tb, 2, N=400000, ratios=(20, 20, 10))
    wide = np.concatenate([pts.min(0) - 1, pts.max(0) + 1])[None, :].repeat(3, 0)
    for _ in range(2):
        got = _check(tb, h, np.ascontiguousarray(wide), tb.WANT_VALS)
        assert got[0][-1] == 3 * len(pts)
    for _ in range(20):
        _check(tb, h, _boxes(pts, 5, 3, 0.01, 0.05))


def test_graph_replay_equals_direct(tb, cuda):
    import torch
    h, pts = _index(tb, 5)
    Q = torch.from_numpy(_boxes(pts, 200, 2)).cuda()
    want = _answer(tb, h, Q, 0)
    for _ in range(3):
        got = _answer(tb, h, Q, tb.USE_GRAPH)
        assert all(np.array_equal(a, b) for a, b in zip(got[:2], want[:2])) and got[3] == want[3]
