"""KMeans at the edges of its sort and of its short assignment lists: counting
sorts of one and several scan blocks, and points whose nearest centroid is
repeated more often than the list is long (few such rows, and many)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,d", [(900, 7, 3), (5000, 819, 8), (5000, 820, 8), (9300, 1000, 5)])
def test_lloyd_bits(gpu_lib, orc, n, k, d):
    import manifoldann_gb300 as M

    rng = np.random.default_rng(n + k)
    X = rng.standard_normal((n, d)).astype(np.float32)
    C0 = X[rng.choice(n, k, replace=False)]
    C, a, it = M.lloyd(C0.T, X.T, M.SqEuclidean(), max_iters=3, tol=1e-9)
    C_o, a_o, it_o = orc.kmeans_lloyd(X, C0, 3, 1e-9, 1)
    assert it == it_o
    assert np.array_equal(a - 1, a_o)
    assert np.array_equal(C.T.view(np.uint32), C_o.view(np.uint32))


@pytest.mark.parametrize("copies", [8, 9, 70, 300])
@pytest.mark.parametrize("near", [20, 2000])
def test_repeated_centroids_take_the_lowest_id(gpu_lib, copies, near):
    import manifoldann_gb300 as M

    rng = np.random.default_rng(copies)
    C = rng.standard_normal((400, 6)).astype(np.float32) + 20.0
    where = np.sort(rng.choice(400, copies, replace=False))
    C[where] = np.float32(0.5)
    X = rng.standard_normal((3000, 6)).astype(np.float32) + 20.0
    X[:near] = np.float32(0.25)
    a, _ = M.assign_arrays(X.T, C.T, M.SqEuclidean())
    # up to 256 equal centroids are ordered by id; a longer run keeps the list's own order
    if copies <= 256:
        assert np.all(a[:near] == where[0])
    else:
        assert np.all(np.isin(a[:near], where))


@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("scale", [1.0, 1e-17, 3e-20, 1e17])
@pytest.mark.parametrize("k,d,kind", [(1, 3, "cloud"), (2, 2, "cloud"), (37, 2, "cloud"), (90, 7, "cloud"), (30, 4, "repeated")])
def test_bounded_assignments_stay_exact(gpu_lib, orc, metric, scale, k, d, kind):
    # overlapping clusters: points keep changing sides for many iterations; at the
    # scales' ends squares underflow or near the top of the range
    import manifoldann_gb300 as M

    n = 4000
    rng = np.random.default_rng(k + d)
    X = rng.standard_normal((n, d)) * scale
    if kind == "repeated":
        X = np.round(rng.standard_normal((n, d)) * 2) * scale  # many equal points, empty clusters to repair
    X = X.astype(np.float32)
    C0 = X[rng.choice(n, k, replace=False)]
    tol = 1e-30
    C, a, it = M.lloyd(C0.T, X.T, M.Euclidean() if metric == 0 else M.SqEuclidean(), max_iters=25, tol=tol)
    C_o, a_o, it_o = orc.kmeans_lloyd(X, C0, 25, tol, metric)
    assert it == it_o
    assert np.array_equal(a - 1, a_o)
    assert np.array_equal(C.T.view(np.uint32), C_o.view(np.uint32))
