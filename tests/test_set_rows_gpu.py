"""Many-set tensor-core graphs whose rows need the exact scan of their own set
(runs of equal points leave no certificate): sets around a warp's 64 points,
a block's pass and a chunk, empty sets among many, widths with and without
four-wide loads.  Ids and distance bits equal the oracle's."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[40, 64, 65, 511, 512, 513], [4095, 4096, 4097, 8300], [45] * 1100 + [700]])
@pytest.mark.parametrize("d", [3, 16, 30, 36])
@pytest.mark.parametrize("metric", [0, 1])
def test_rows_of_sets(gpu_lib, orc, sizes, d, metric):
    import torch

    from manifoldann_gb300 import _lib

    rng = np.random.default_rng(d + len(sizes))
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    X = rng.standard_normal((offs[-1], d)).astype(np.float32)
    for a, b in zip(offs[:-1], offs[1:]):
        X[a + 2:a + 40] = X[a + 2]  # more equal points than a list holds
    k = 7
    x = torch.from_numpy(X).cuda()
    ids = torch.empty((len(X), k), dtype=torch.int32, device="cuda")
    dist = torch.empty((len(X), k), dtype=torch.float32, device="cuda")
    rep = _lib.KnnReport()
    _lib.check(gpu_lib.mann_knn_graph_batched_device(_lib.params(metric, k, _lib.PREC_BF16), x.data_ptr(),
                                                     offs.ctypes.data, len(sizes), d, 0, ids.data_ptr(),
                                                     dist.data_ptr(), C.byref(rep), None))
    torch.cuda.synchronize()
    assert rep.rows_fallback > 0
    ids, dist = ids.cpu().numpy(), dist.cpu().numpy()
    for c in sorted({0, 1, 2, 3, len(sizes) // 2, len(sizes) - 1}):
        a, b = offs[c], offs[c + 1]
        ids_o, d_o = orc.knn_graph_f32(X[a:b], k, metric)
        assert np.array_equal(ids[a:b], ids_o)
        assert np.array_equal(dist[a:b].view(np.uint32), d_o.view(np.uint32))


@pytest.mark.parametrize("sizes", [[41, 45, 60, 700], [43, 41] * 600])
@pytest.mark.parametrize("k", [1, 31, 32, 40])
@pytest.mark.parametrize("include_self", [0, 1])
def test_results_of_sets(gpu_lib, orc, sizes, k, include_self):
    """Results of lists up to 32 entries and past them, sets hardly larger than k, ids counted from their set."""
    import torch

    from manifoldann_gb300 import _lib

    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    X = np.random.default_rng(k).standard_normal((offs[-1], 5)).astype(np.float32)
    x = torch.from_numpy(X).cuda()
    ids = torch.empty((len(X), k), dtype=torch.int32, device="cuda")
    dist = torch.empty((len(X), k), dtype=torch.float32, device="cuda")
    _lib.check(gpu_lib.mann_knn_graph_batched_device(_lib.params(1, k), x.data_ptr(), offs.ctypes.data, len(sizes), 5,
                                                     include_self, ids.data_ptr(), dist.data_ptr(), None, None))
    torch.cuda.synchronize()
    ids, dist = ids.cpu().numpy(), dist.cpu().numpy()
    for c in sorted({0, 1, 2, 3, len(sizes) // 2, len(sizes) - 1}):
        a, b = offs[c], offs[c + 1]
        want = orc.knn_f32(X[a:b], X[a:b], k, 1) if include_self else orc.knn_graph_f32(X[a:b], k, 1)
        assert np.array_equal(ids[a:b], want[0])
        assert np.array_equal(dist[a:b].view(np.uint32), want[1].view(np.uint32))
