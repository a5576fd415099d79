"""Searches of few queries, whose probed lists are scanned in parts: one long
list, as many lists as a query's merge takes, lists shorter than a part, short
and long results.  With every list probed the answer is the oracle's exact one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nlist", [(9001, 1), (2049, 3), (300, 9), (20000, 50), (6000, 128)])
@pytest.mark.parametrize("nq,k", [(1, 1), (2, 20), (17, 32), (40, 33), (3, 64)])
@pytest.mark.parametrize("d", [5, 64])
def test_all_lists(gpu_lib, orc, n, nlist, nq, k, d):
    import torch

    import manifoldann_gb300 as M
    from manifoldann_gb300 import _lib

    rng = np.random.default_rng(n + nq + d)
    X, Q = rng.standard_normal((n, d)).astype(np.float32), rng.standard_normal((nq, d)).astype(np.float32)
    X[n // 2:n // 2 + 40] = X[n // 2]  # equal distances
    owner = rng.integers(0, nlist, n) ** 2 // max(nlist, 1)  # uneven, some empty
    ids = np.argsort(owner, kind="stable").astype(np.int32)
    offs = np.searchsorted(owner[ids], np.arange(nlist + 1)).astype(np.int64)
    probes = np.tile(np.arange(nlist, dtype=np.int32), (nq, 1))
    dev = [torch.from_numpy(a).cuda() for a in (X, Q, ids, offs, probes)]
    x, q, lids, loff, pr = dev
    oi = torch.empty((nq, k), dtype=torch.int32, device="cuda")
    od = torch.empty((nq, k), dtype=torch.float32, device="cuda")
    _lib.check(gpu_lib.mann_ivf_scan_device(_lib.params(1, k), pr.data_ptr(), nlist, x.data_ptr(), n, d, nlist,
                                            loff.data_ptr(), lids.data_ptr(), q.data_ptr(), nq, oi.data_ptr(),
                                            od.data_ptr(), None))
    torch.cuda.synchronize()
    ids_o, d_o = orc.knn_f32(X, Q, k, 1)
    assert np.array_equal(oi.cpu().numpy(), ids_o)
    assert np.array_equal(od.cpu().numpy().view(np.uint32), d_o.view(np.uint32))
