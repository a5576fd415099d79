"""A handful of rows of four-wide widths, whose points come in through shared
memory a slice at a time: widths around a slice, point counts off a warp's 32
and a block's 256, one to four rows, short and long lists.  Equal to the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,nq,k", [(31, 4, 1, 3), (257, 36, 4, 33), (300, 28, 3, 64), (8197, 2048, 4, 10), (70001, 260, 1, 32), (280037, 60, 3, 7), (466033, 36, 2, 1),
                                      (262144, 64, 1, 20), (1048577, 16, 4, 5), (4200001, 4, 1, 9)])
@pytest.mark.parametrize("metric", [0, 1, 2])
def test_sliced(gpu_lib, orc, n, d, nq, k, metric):
    import manifoldann_gb300 as M

    m = {0: M.Euclidean(), 1: M.SqEuclidean(), 2: M.CosineDist()}[metric]
    rng = np.random.default_rng(n)
    base = rng.standard_normal((n, d)).astype(np.float32)
    base[-20:-3] = base[-1]  # equal distances at the end
    q = rng.standard_normal((nq, d)).astype(np.float32)
    q[0] = base[-1] + 0.01 * q[0]
    ids, dd = M.knn_arrays(M.build_index(M.BruteForceIndex, base.T, distance=m), base.T, q.T, k)
    ids_o, d_o = orc.knn_f32(base, q, k, metric)
    assert np.array_equal(ids, ids_o)
    assert np.array_equal(dd.view(np.uint32), d_o.view(np.uint32))
