"""Exact KNN on data so small that float squares of its distances are denormal.

The probe bounds each query's K-th distance from float squares; what underflow takes from them must not
put the bound below the distance itself. Ids and squared distances equal the FP64 brute force's bit for
bit, so no tolerance is involved.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extent", [1e-18, 1e-20, 3e-21, 1e-23])
@pytest.mark.parametrize("D,K", [(8, 10), (3, 4), (16, 10)])
def test_denormal_squares(tb, oracle_mod, cuda, extent, D, K):
    rng = np.random.default_rng(D)
    X = rng.uniform(-extent, extent, (400, D)).astype(np.float32)
    h, _ = tb.QueryHandler.build(X, height=3, ratios=(20, 5), iters=3, seed=1)
    h.prepare_for_query(tb.LevelPolicy.L0)
    pts, ids = h.decode_points(np.arange(len(X)))
    P = np.ascontiguousarray(rng.uniform(-extent, extent, (20000, D)))
    b = oracle_mod.brute_query(pts, ids, oracle_mod.KNN, P, K=K)
    for _ in range(2):  # the second batch reuses the first one's result memory
        r = h.query_batch(tb.QueryType.POINT, P, tb.Mode.EXACT, K=K)
        assert np.array_equal(r.offsets.numpy(), b.offsets)
        assert np.array_equal(r.ids.numpy(), b.ids)
        assert np.array_equal(r.dist2.numpy(), b.dist2)
