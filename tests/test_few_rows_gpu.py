"""Searches of a handful of rows, whose kernel merges and writes its results
itself: block counts around one, list lengths with and without that path,
graphs of tiny sets (the row itself dropped), results past the staging of
small host calls, repeated calls.  Equal to the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nq,d,k", [(1, 1, 3, 1), (5, 4, 7, 5), (255, 1, 64, 10), (256, 2, 2048, 32), (257, 3, 2048, 33),
                                      (300, 4, 2047, 64), (300, 4, 2049, 12), (66000, 1, 16, 32), (70001, 4, 5, 31),
                                      (900, 5, 64, 10), (40, 3, 9, 40)])
@pytest.mark.parametrize("metric", [0, 1, 2])
def test_few_rows(gpu_lib, orc, n, nq, d, k, metric):
    import manifoldann_gb300 as M

    m = {0: M.Euclidean(), 1: M.SqEuclidean(), 2: M.CosineDist()}[metric]
    rng = np.random.default_rng(n + nq)
    base = rng.standard_normal((n, d)).astype(np.float32)
    if n > 200:
        base[100:180] = base[99]  # a run of equal distances
    q = rng.standard_normal((nq, d)).astype(np.float32)
    index = M.build_index(M.BruteForceIndex, base.T, distance=m)
    ids_o, d_o = orc.knn_f32(base, q, min(k, n), metric)
    handle = M.DeviceDataset(base.T)
    for data in (base.T, handle, handle):
        ids, dd = M.knn_arrays(index, data, q.T, k)
        assert np.array_equal(ids, ids_o)
        assert np.array_equal(dd.view(np.uint32), d_o.view(np.uint32))


@pytest.mark.parametrize("n,k", [(2, 1), (3, 2), (4, 3), (4, 1), (33, 32), (33, 5), (40, 31)])
def test_graphs_of_tiny_sets(gpu_lib, orc, n, k):
    import manifoldann_gb300 as M

    X = np.random.default_rng(n).integers(0, 3, (n, 2)).astype(np.float32)
    index = M.build_index(M.BruteForceIndex, X.T, distance=M.SqEuclidean())
    ids, d = M.knn_graph_arrays(index, X.T, k)
    ids_o, d_o = orc.knn_graph_f32(X, k, 1)
    assert np.array_equal(ids, ids_o)
    assert np.array_equal(d.view(np.uint32), d_o.view(np.uint32))


@pytest.mark.parametrize("nq", [819, 820, 8192])
def test_results_around_the_staging_of_small_calls(gpu_lib, orc, nq):
    import manifoldann_gb300 as M

    rng = np.random.default_rng(nq)
    base, q = rng.standard_normal((500, 4)).astype(np.float32), rng.standard_normal((nq, 4)).astype(np.float32)
    index = M.build_index(M.BruteForceIndex, base.T, distance=M.SqEuclidean())
    ids, d = M.knn_arrays(index, M.DeviceDataset(base.T), q.T, 10)
    ids_o, d_o = orc.knn_f32(base, q, 10, 1)
    assert np.array_equal(ids, ids_o) and np.array_equal(d.view(np.uint32), d_o.view(np.uint32))
