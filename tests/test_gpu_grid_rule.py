"""The per-level plugin's choice between counting and sorting, on both sides of its rule.

Either way the level's grid must equal the reference traversal's (the oracle's restatement), in order; the
launch counts tell the path (four launches count).
"""
import numpy as np
import pytest

from conftest import oracle_from_handler

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("clusters,ratio,K,counted", [(8192, 4, 32768, True), (8193, 4, 4096, True), (8193, 4, 4098, False),
                                                      (16384, 3, 6144, True), (16384, 3, 6145, False), (16385, 3, 1, False)])
def test_counted_or_sorted(tb, oracle_mod, tmp_path, cuda, clusters, ratio, K, counted):
    h = tb.QueryHandler.generate(clusters * ratio, 4, 1.0, 100.0, False, 2, (ratio,), 7, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    o = oracle_from_handler(oracle_mod, h, tmp_path)
    pts, _ = oracle_mod.decoded_points(o)
    P = np.ascontiguousarray(pts[::clusters // 2][:2] + 0.5)
    ref = oracle_mod.ref_query(o, oracle_mod.KNN, P, K=K, sorted_ids=False)
    for q in range(len(P)):
        g = h.coarsest_grid()
        assert g.nnz == clusters
        before = tb.kernel_launches()
        g = h.run_level(0, g, tb.QueryType.POINT, point=P[q], K=K)
        assert (tb.kernel_launches() - before == 4) == counted
        assert np.array_equal(h.grid_arrays(g)[0], ref.query(q))
