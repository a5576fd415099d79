"""k-means++ draws where most points are left out of a step because the new
centroid is too far from theirs: well separated groups, groups of one point,
scales at which squared distances are denormal, tiny or overflow, points at
exactly half the distance of two centroids.  Chosen points equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-21, 1e-15, 1.0, 1e16, 1e18, 8e18])
@pytest.mark.parametrize("n,d,groups,noise", [(140001, 64, 40, 0.3), (131073, 67, 2, 0.0), (65000, 130, 300, 0.05),
                                              (700, 1, 5, 0.5), (78337, 3, 9, 0.01)])
def test_groups(gpu_lib, orc, n, d, groups, noise, scale):
    import manifoldann_gb300 as M

    rng = np.random.default_rng(n + d)
    centres = rng.integers(-4, 5, (groups, d)).astype(np.float32)  # whole numbers: exact halves occur
    X = centres[rng.integers(0, groups, n)] + noise * rng.standard_normal((n, d))
    X[::7] = np.round(2 * X[::7]) / 2
    X = (X * scale).astype(np.float32)
    k = min(60, n)
    u = rng.random(k)
    _, idx = M.init_kmeans_plus_plus(X.T, k, first=5, u=u)
    assert np.array_equal(idx - 1, orc.kmeanspp(X, k, 4, u))
