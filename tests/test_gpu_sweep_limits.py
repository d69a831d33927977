"""Sizes at which a sweep's launch meets a limit of the grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_range_over_many_upper_nodes(tb, cuda):
    """Fan-outs of two: 280,000 parents, four a block, are more blocks than a y axis has (65,535). Wide
    boxes have more segments than the gather orders and end in the level launches, narrow ones sweep."""
    N = 2_240_000
    h = tb.QueryHandler.generate(N, 1, 1.0, 100.0, False, 4, (2, 2, 2), 5, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    assert 280_000 in h.info()["meshSizes"]
    rng = np.random.default_rng(2)
    c = h.decode_points(rng.integers(0, N, 70))[0]
    for widest in (1e-5, 1e-2):
        hw = np.exp(rng.uniform(np.log(1e-6), np.log(widest), c.shape)) * 100
        Q = np.ascontiguousarray(np.concatenate([c - hw, c + hw], 1))
        before = tb.kernel_launches()
        r = h.query_batch(tb.QueryType.RANGE, Q, tb.Mode.EXACT)
        launches = tb.kernel_launches() - before
        got = r.offsets.numpy().copy(), r.ids.numpy().copy(), h.level_counts()
        assert launches == 3 or widest > 1e-5
        h.set_launch_shapes([0] * 4, [99] * 4)
        r = h.query_batch(tb.QueryType.RANGE, Q, tb.Mode.EXACT)
        h.set_launch_shapes([0] * 4, [100] * 4)
        assert np.array_equal(got[0], r.offsets.numpy()) and np.array_equal(got[1], r.ids.numpy())
        assert got[2] == h.level_counts() and got[0][-1] >= 70
