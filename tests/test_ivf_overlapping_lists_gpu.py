"""Inverted lists that share points (every point in several lists): a point that
several probed lists hold is one result, as in the oracle's exact search of the
probed points."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,nprobe", [(3, 2), (40, 5), (700, 9), (60, 40), (9000, 3)])
@pytest.mark.parametrize("k", [1, 10, 31, 32, 33])
@pytest.mark.parametrize("copies", [2, 4])
def test_points_in_several_lists(gpu_lib, orc, nq, nprobe, k, copies):
    import torch

    from manifoldann_gb300 import _lib

    rng = np.random.default_rng(nq + k)
    n, d, nlist = 3000, 12, 40
    X, Q = rng.standard_normal((n, d)).astype(np.float32), rng.standard_normal((nq, d)).astype(np.float32)
    X[100:130] = X[100]  # equal distances of different points
    owners = np.argsort(rng.random((n, nlist)), axis=1)[:, :copies]
    lists = [np.flatnonzero((owners == c).any(axis=1)).astype(np.int32) for c in range(nlist)]
    lists[7] = lists[3].copy()  # one list twice
    offs = np.concatenate([[0], np.cumsum([len(v) for v in lists])]).astype(np.int64)
    probes = np.argsort(rng.random((nq, nlist)), axis=1)[:, :nprobe].astype(np.int32)
    probes[0, :2] = (3, 7)
    probes[0, 2:] = -1
    x, q, ids, off, pr = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
                          for a in (X, Q, np.concatenate(lists), offs, probes)]
    oi = torch.empty((nq, k), dtype=torch.int32, device="cuda")
    od = torch.empty((nq, k), dtype=torch.float32, device="cuda")
    _lib.check(gpu_lib.mann_ivf_scan_device(_lib.params(1, k), pr.data_ptr(), nprobe, x.data_ptr(), n, d, nlist,
                                            off.data_ptr(), ids.data_ptr(), q.data_ptr(), nq, oi.data_ptr(),
                                            od.data_ptr(), None))
    torch.cuda.synchronize()
    oi, od = oi.cpu().numpy(), od.cpu().numpy()
    for r in range(0, nq, max(1, nq // 40)):
        own = np.unique(np.concatenate([lists[c] for c in probes[r] if c >= 0]))
        m = min(k, len(own))
        want, dw = orc.knn_f32(X[own], Q[r:r + 1], m, orc.SQEUCLIDEAN)
        assert np.array_equal(oi[r, :m], own[want[0]])
        assert np.array_equal(od[r, :m].view(np.uint32), dw[0].view(np.uint32))
        assert np.all(oi[r, m:] == -1)
