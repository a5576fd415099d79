"""Lloyd where a point's squared distance to all but one centroid overflows: a
centroid that far away may still come near, so the point's bounds may not take
it for infinitely far."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _equal(orc, X, C0, metric, iters):
    import manifoldann_gb300 as M

    C, a, it = M.lloyd(C0.T, X.T, M.Euclidean() if metric == 0 else M.SqEuclidean(), max_iters=iters, tol=1e-30)
    C_o, a_o, it_o = orc.kmeans_lloyd(X, C0, iters, 1e-30, metric)
    assert it == it_o
    assert np.array_equal(a - 1, a_o)
    assert np.array_equal(C.T.view(np.uint32), C_o.view(np.uint32))


@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("d", [1, 4])
def test_far_centroid_comes_near(gpu_lib, orc, metric, d):
    # the point at 0 belongs to the centroid at 0; its nine fellows pull that
    # one to -1.35e19 while the other, at first out of range, moves to 1.3e19
    x = np.concatenate([[0.0], np.full(9, -1.5e19), np.full(10, 1.3e19)])
    X, C0 = np.zeros((20, d), np.float32), np.zeros((2, d), np.float32)
    X[:, 0], C0[1, 0] = x, 2.5e19
    _equal(orc, X, C0, metric, 1)
    _equal(orc, X, C0, metric, 5)


@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("seed", range(6))
def test_wide_clouds(gpu_lib, orc, metric, seed):
    rng = np.random.default_rng(seed)
    X = (rng.uniform(-2.4e19, 2.4e19, (3000, 1))).astype(np.float32)
    C0 = X[rng.choice(3000, 7, replace=False)]
    if np.abs(X.astype(np.float64) - C0[:, 0]).min(axis=1).max() ** 2 > np.finfo(np.float32).max:
        # distances that all overflow are equal to the search, which then takes the lowest id; FP64 does not
        pytest.skip("a point out of range of every centroid")
    _equal(orc, X, C0, metric, 25)
