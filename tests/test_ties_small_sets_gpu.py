"""FP64 order of near-ties in sets that a row's list holds whole: no point lies
beyond the list, so a cluster that runs to its end is ordered like any other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("n,k", [(2, 1), (5, 3), (8, 8), (31, 4), (32, 24), (33, 1), (40, 9), (64, 24)])
def test_shells(gpu_lib, orc, precision, metric, n, k):
    import torch

    from manifoldann_gb300 import _lib

    rng = np.random.default_rng(n)
    d, nq = 16, 50
    X = rng.standard_normal((n, d))
    X = (X / np.linalg.norm(X, axis=1, keepdims=True)).astype(np.float32)
    Q = (1e-9 * rng.standard_normal((nq, d))).astype(np.float32)  # every point at 1 within FP32 rounding
    x, q = torch.from_numpy(X).cuda(), torch.from_numpy(Q).cuda()
    ids = torch.empty((nq, k), dtype=torch.int32, device="cuda")
    dist = torch.empty((nq, k), dtype=torch.float32, device="cuda")
    p = _lib.params(metric, k, precision, 0, _lib.FLAG_FP64_TIES)
    _lib.check(gpu_lib.mann_knn_device(p, x.data_ptr(), n, q.data_ptr(), nq, d, ids.data_ptr(), dist.data_ptr(), None,
                                       None))
    torch.cuda.synchronize()
    want, _ = orc.knn_f64(X, Q, k, metric)
    assert np.array_equal(ids.cpu().numpy(), want)


@pytest.mark.parametrize("k", [2, 8, 9, 33])
def test_assignment_to_few_centroids(gpu_lib, orc, k):
    import manifoldann_gb300 as M

    rng = np.random.default_rng(k)
    C = rng.standard_normal((k, 16))
    C = (C / np.linalg.norm(C, axis=1, keepdims=True)).astype(np.float32)
    X = (1e-9 * rng.standard_normal((500, 16))).astype(np.float32)
    a, _ = M.assign_arrays(X.T, C.T, M.SqEuclidean())
    want, _ = orc.kmeans_assign_f64(X, C, 1)
    assert np.array_equal(a, want)
