"""FP64 order of near-ties where a cluster of equal points runs past the lists
of the FP32 form, for results of one entry up to nearly the longest list, in
sets smaller and larger than the lists."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 31, 33, 60, 224, 225, 250])
@pytest.mark.parametrize("n,copies", [(1000, 40), (1000, 255), (1000, 300), (300, 70), (257, 257)])
@pytest.mark.parametrize("metric", [0, 1])
def test_repeated_points(gpu_lib, orc, k, n, copies, metric):
    import torch

    from manifoldann_gb300 import _lib

    rng = np.random.default_rng(k + n + copies)
    X = rng.standard_normal((n, 6)).astype(np.float32) + 9.0
    X[np.sort(rng.choice(n, copies, replace=False))] = np.float32(0.5)
    Q = rng.standard_normal((40, 6)).astype(np.float32)
    x, q = torch.from_numpy(X).cuda(), torch.from_numpy(Q).cuda()
    ids = torch.empty((40, k), dtype=torch.int32, device="cuda")
    dist = torch.empty((40, k), dtype=torch.float32, device="cuda")
    p = _lib.params(metric, k, _lib.PREC_FP32, 0, _lib.FLAG_FP64_TIES)
    _lib.check(gpu_lib.mann_knn_device(p, x.data_ptr(), n, q.data_ptr(), 40, 6, ids.data_ptr(), dist.data_ptr(), None,
                                       None))
    torch.cuda.synchronize()
    want, _ = orc.knn_f64(X, Q, k, metric)
    every, all_d = orc.knn_f32(X, Q, n, metric)
    dw = np.take_along_axis(np.take_along_axis(all_d, np.argsort(every, axis=1), axis=1), want, axis=1)
    # equal points keep their order by id, in lists of at most 256 entries too
    assert np.array_equal(ids.cpu().numpy(), want)
    assert np.array_equal(dist.cpu().numpy().view(np.uint32), dw.view(np.uint32))


@pytest.mark.parametrize("k,shell", [(20, 60), (40, 80), (64, 100), (100, 150), (200, 250)])
@pytest.mark.parametrize("metric", [0, 1])
def test_near_ties_past_long_lists(gpu_lib, orc, k, shell, metric):
    import torch

    from manifoldann_gb300 import _lib

    rng = np.random.default_rng(k)
    n, d, nq = 900, 16, 40
    X = rng.standard_normal((n, d))
    X = X / np.linalg.norm(X, axis=1, keepdims=True)
    far = np.sort(rng.choice(n, n - shell, replace=False))
    X[far] *= rng.uniform(2.0, 3.0, (n - shell, 1))  # `shell` points at 1 within FP32 rounding
    X = X.astype(np.float32)
    Q = (1e-9 * rng.standard_normal((nq, d))).astype(np.float32)
    x, q = torch.from_numpy(X).cuda(), torch.from_numpy(Q).cuda()
    ids = torch.empty((nq, k), dtype=torch.int32, device="cuda")
    dist = torch.empty((nq, k), dtype=torch.float32, device="cuda")
    rep = _lib.KnnReport()
    p = _lib.params(metric, k, _lib.PREC_FP32, 0, _lib.FLAG_FP64_TIES)
    _lib.check(gpu_lib.mann_knn_device(p, x.data_ptr(), n, q.data_ptr(), nq, d, ids.data_ptr(), dist.data_ptr(), rep,
                                       None))
    torch.cuda.synchronize()
    want, _ = orc.knn_f64(X, Q, k, metric)
    assert np.array_equal(ids.cpu().numpy(), want)
    assert rep.rows_unresolved == 0
