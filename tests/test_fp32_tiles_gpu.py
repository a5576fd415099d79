"""The FP32 tile kernel where its walk, queues and thresholds can go wrong: tile
and block edges, rows whose every point is a candidate (queues run full),
equal distances across and inside tiles, and the list lengths at which the
kernel's variant changes.  Ids and distance bits equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(orc, base, q, k, metric):
    import manifoldann_gb300 as M

    m = {0: M.Euclidean(), 1: M.SqEuclidean(), 2: M.CosineDist()}[metric]
    ids, d = M.knn_arrays(M.build_index(M.BruteForceIndex, base.T, distance=m), base.T, q.T, k)
    ids_o, d_o = orc.knn_f32(base, q, k, metric)
    assert np.array_equal(ids, ids_o)
    assert np.array_equal(d.view(np.uint32), d_o.view(np.uint32))


@pytest.mark.parametrize("n,nq,d,k", [(127, 33, 16, 5), (128, 64, 17, 32), (129, 65, 4, 33), (257, 63, 31, 64),
                                      (1000, 129, 15, 65), (700, 100, 5, 128), (700, 40, 33, 129), (600, 70, 3, 256),
                                      (12801, 200, 8, 10), (9000, 1100, 12, 3)])
@pytest.mark.parametrize("metric", [0, 1, 2])
def test_edges(gpu_lib, orc, n, nq, d, k, metric):
    rng = np.random.default_rng(n + k)
    check(orc, rng.standard_normal((n, d)).astype(np.float32), rng.standard_normal((nq, d)).astype(np.float32), k,
          metric)


@pytest.mark.parametrize("k", [1, 10, 32, 48])
@pytest.mark.parametrize("metric", [0, 1])
def test_every_point_is_nearer_than_the_last(gpu_lib, orc, k, metric):
    # distances fall with the id, so every point is admitted and every queue runs full in every tile
    n, d = 1500, 8
    base = np.zeros((n, d), np.float32)
    base[:, 0] = np.arange(n, 0, -1, dtype=np.float32) * np.float32(0.37)
    q = np.zeros((70, d), np.float32)
    q[:, 1] = np.arange(70, dtype=np.float32)
    check(orc, base, q, k, metric)


@pytest.mark.parametrize("metric", [0, 1])
def test_equal_distances_take_the_lowest_ids(gpu_lib, orc, metric):
    rng = np.random.default_rng(5)
    base = np.repeat(rng.integers(0, 3, (9, 6)).astype(np.float32), 120, axis=0)  # runs of duplicates across tiles
    base = base[rng.permutation(len(base))]
    q = rng.integers(0, 3, (100, 6)).astype(np.float32)
    for k in (7, 31, 60):
        check(orc, base, q, k, metric)


@pytest.mark.parametrize("scale", [1e-30, 1e-21, 3e18, 2e19])
def test_thresholds_at_the_ends_of_the_range(gpu_lib, orc, scale):
    # squares that underflow, and that overflow to infinity
    rng = np.random.default_rng(6)
    base = (rng.standard_normal((900, 6)) * scale).astype(np.float32)
    q = (rng.standard_normal((80, 6)) * scale).astype(np.float32)
    check(orc, base, q, 12, 0)
    check(orc, base, q, 12, 1)


def test_not_a_number_sorts_last(gpu_lib, orc):
    rng = np.random.default_rng(7)
    base = rng.standard_normal((700, 5)).astype(np.float32)
    base[rng.choice(700, 650, replace=False), 2] = np.nan
    check(orc, base, rng.standard_normal((90, 5)).astype(np.float32), 64, 0)


@pytest.mark.parametrize("k", [5, 32, 42, 64, 100])
def test_rows_of_nothing_but_nan_take_the_lowest_ids(gpu_lib, orc, k):
    # a zero query has a NaN cosine to every point: more equal candidates than a queue holds
    rng = np.random.default_rng(8)
    q = rng.standard_normal((70, 9)).astype(np.float32)
    q[::3] = 0.0
    check(orc, rng.standard_normal((700, 9)).astype(np.float32), q, k, 2)
