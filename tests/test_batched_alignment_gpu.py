"""Batched FP32 graphs of points that start at any float of a larger buffer:
rows whose width is a multiple of four lie on no 16-byte boundary there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric,k", [(0, 6), (1, 40)])
@pytest.mark.parametrize("lead", [1, 2, 3, 4])
def test_points_inside_a_buffer(gpu_lib, orc, metric, k, lead):
    import torch

    from manifoldann_gb300 import _lib

    rng = np.random.default_rng(lead)
    sizes, d = [150, 300, 70], 12
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n = int(offs[-1])
    pts = rng.standard_normal((n, d)).astype(np.float32)
    buf = torch.zeros(n * d + 8, device="cuda")
    x = buf[lead:lead + n * d]
    x.copy_(torch.from_numpy(pts.reshape(-1)))
    ids = torch.empty((n, k), dtype=torch.int32, device="cuda")
    dist = torch.empty((n, k), dtype=torch.float32, device="cuda")
    p = _lib.params(metric, k, _lib.PREC_FP32)
    for _ in range(2):  # measured candidates and capture, then the replay
        ids.fill_(-7)
        _lib.check(gpu_lib.mann_knn_graph_batched_device(p, x.data_ptr(), offs.ctypes.data, len(sizes), d, 0,
                                                         ids.data_ptr(), dist.data_ptr(), None,
                                                         torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        for c, m in enumerate(sizes):
            want, dw = orc.knn_graph_f32(pts[offs[c]:offs[c + 1]], k, metric)
            assert np.array_equal(ids.cpu().numpy()[offs[c]:offs[c + 1]], want)
            assert np.array_equal(dist.cpu().numpy()[offs[c]:offs[c + 1]].view(np.uint32), dw.view(np.uint32))
