"""Assignment passes after the first: each point starts from the pair its last pass kept.

The centroids after one pass are known, so the second pass's labels are checked against the FP64
distances to them. Tensor-core values are off by at most 2e-5 (|x|^2 + |c|^2) (three TF32 products, FP32
sums), so a label's distance may exceed the smallest by twice that and by no more.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,k,n", [(16, 2, 129), (3, 600, 20000), (16, 1000, 30011), (8, 129, 4096)])
@pytest.mark.parametrize("offset,scale", [(0.0, 1.0), (500.0, 1.0), (0.0, 1e-12), (0.0, 1e15)])
def test_second_pass_labels(tb, cuda, D, k, n, offset, scale):
    rng = np.random.default_rng(D * k)
    X = ((rng.normal(0, 1, (n, D)) + 10 * rng.normal(0, 1, (40, D))[rng.integers(0, 40, n)] + offset) * scale).astype(np.float32)
    X[: n // 8] = X[0]  # equal points: many equal distances
    C, _, _ = tb.kmeans(X, k, iters=1, seed=4, precision=tb.KmeansPrecision.TENSOR)
    _, L, _ = tb.kmeans(X, k, iters=2, seed=4, precision=tb.KmeansPrecision.TENSOR)
    C, L, X64 = np.asarray(C, np.float64), np.asarray(L), X.astype(np.float64)
    assert L.min() >= 0 and L.max() < k
    cc = (C * C).sum(1)
    best = np.concatenate([((X64[i:i + 2000, None, :] - C[None]) ** 2).sum(2).min(1) for i in range(0, n, 2000)])
    got = ((X64 - C[L]) ** 2).sum(1)
    tol = 4e-5 * ((X64 ** 2).sum(1) + cc.max()) + 1e-29
    assert np.all(got <= best + tol)
