"""Per-level plugin steps without a sort, at the sizes where they can go wrong.

The grid after every level must equal the reference traversal's (the oracle's restatement): same ids,
same order, for K around the children counts that decide STEP, for grids of one entry, of a block's
edge and just past the size up to which no sort is used.
"""
import numpy as np
import pytest

from conftest import oracle_from_handler

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,D,ratios", [(3000, 2, (30, 99)), (20000, 3, (10, 8)), (40000, 7, (9, 5, 3)),
                                        (49152, 4, (3,)), (49155, 4, (3,))])  # 16,384 and 16,385 clusters
def test_levels_equal_the_reference(tb, oracle_mod, tmp_path, cuda, N, D, ratios):
    h = tb.QueryHandler.generate(N, D, 1.0, 100.0, False, len(ratios) + 1, ratios, 7, 2.5)
    h.prepare_for_query(tb.LevelPolicy.L0)
    o = oracle_from_handler(oracle_mod, h, tmp_path)
    pts, _ = oracle_mod.decoded_points(o)
    rng = np.random.default_rng(1)
    P = np.ascontiguousarray(pts[rng.integers(0, N, 3)] + rng.normal(0, 0.5, (3, D)))
    P[2] = pts[5]
    hw = 0.08 * (pts.max(0) - pts.min(0))
    Q = np.ascontiguousarray(np.concatenate([P - hw, P + hw], 1))
    levels = len(ratios)
    for K in (0, 1, ratios[0], ratios[0] + 1, 10 * ratios[0], N):
        ref = oracle_mod.ref_query(o, oracle_mod.KNN, P, K=K, sorted_ids=False)
        for q in range(3):
            g, sizes = h.coarsest_grid(), []
            for l in range(levels):
                g = h.run_level(l, g, tb.QueryType.POINT, point=P[q], K=K)
                sizes.append(g.nnz)
            assert sizes == list(ref.level_sizes[q]), (K, q)
            assert np.array_equal(h.grid_arrays(g)[0], ref.query(q)), (K, q)
    ref = oracle_mod.ref_query(o, oracle_mod.RANGE, Q, sorted_ids=False)
    for q in range(3):
        g = h.coarsest_grid()
        for l in range(levels):
            g = h.run_level(l, g, tb.QueryType.RANGE, lo=Q[q, :D], hi=Q[q, D:])
            assert g.nnz == ref.level_sizes[q][l], (l, q)
        assert np.array_equal(h.grid_arrays(g)[0], ref.query(q)), q
