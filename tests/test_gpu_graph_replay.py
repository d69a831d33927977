"""A replayed range graph with KNN batches, and range batches of another kind, run in between.

A replay must return the range answer and its counts, through the device, the host and the asynchronous
entry, whatever ran on the handle since the capture.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(tb, cuda):
    import torch
    h = tb.QueryHandler.generate(30000, 8, 1.0, 100.0, False, 4, (40, 20, 10), 3, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    pts, _ = h.decode_points(np.arange(30000))
    rng = np.random.default_rng(1)
    c = pts[rng.integers(0, len(pts), 60)]
    hw = 0.1 * (pts.max(0) - pts.min(0))
    Q = np.ascontiguousarray(np.concatenate([c - hw, c + hw], 1))
    return h, Q, torch.from_numpy(Q).cuda(), np.ascontiguousarray(c[:7] + 0.1), Q[:3] + 1.0


def _answer(tb, h, dQ, flags):
    r = h.query_batch(tb.QueryType.RANGE, dQ, tb.Mode.EXACT, flags=flags)
    return (int(r.total), r.offsets.numpy().copy(), r.ids.numpy().copy()), h.level_counts(), h.group_counts()


def _same(got, want):
    assert got[0][0] == want[0][0]
    assert np.array_equal(got[0][1], want[0][1]) and np.array_equal(got[0][2], want[0][2])
    assert got[1:] == want[1:]


def _between(tb, h, P, Q):
    h.query_batch(tb.QueryType.POINT, P, tb.Mode.EXACT, K=3)                            # the KNN sweep
    yield
    h.query_batch(tb.QueryType.POINT, P, tb.Mode.EXACT, K=3, flags=tb.WANT_LEVELS)      # the KNN walk
    yield
    h.query_batch(tb.QueryType.RANGE, Q, tb.Mode.EXACT, flags=tb.WANT_LEVELS)           # the range levels
    yield


def test_device_entry(tb, env):
    h, Q, dQ, P, other = env
    want = _answer(tb, h, dQ, 0)
    _same(_answer(tb, h, dQ, tb.USE_GRAPH), want)
    for _ in _between(tb, h, P, other):
        _same(_answer(tb, h, dQ, tb.USE_GRAPH), want)


def test_async_entry(tb, env):
    h, Q, dQ, P, other = env
    want = _answer(tb, h, dQ, 0)
    _answer(tb, h, dQ, tb.USE_GRAPH)
    for _ in _between(tb, h, P, other):
        h.query_batch_async(tb.QueryType.RANGE, dQ, tb.Mode.EXACT, flags=tb.USE_GRAPH)
        assert h.batch_wait() == want[0][0]
        assert h.level_counts() == want[1] and h.group_counts() == want[2]


def test_host_entry(tb, env):
    h, Q, dQ, P, other = env
    want = _answer(tb, h, dQ, 0)
    offs, ids, total = np.zeros(len(Q) + 1, np.uint64), np.zeros(1 << 16, np.uint64), ctypes.c_uint64()

    def host():
        b = tb._Batch(int(tb.QueryType.RANGE), int(tb.Mode.EXACT), len(Q), Q.ctypes.data, 0, 0, tb.USE_GRAPH, None)
        assert tb.lib().tblaeq_query_batch_host(h._h, ctypes.byref(b), tb._dptr(offs, ctypes.c_uint64),
                                                tb._dptr(ids, ctypes.c_uint64), len(ids), None, ctypes.byref(total)) == 0
        n = int(total.value)
        return (n, offs, ids[:n]), h.level_counts(), h.group_counts()

    _same(host(), want)
    for _ in _between(tb, h, P, other):
        offs[:] = ids[:] = 0
        _same(host(), want)
