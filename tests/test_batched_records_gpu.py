"""Batched graphs after a call of the other form that failed: the device copies
of an FP32 plan and of its set offsets are used again only when they are still
the ones that the plan was uploaded with."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(lib, pts, sizes, k, precision, include_self=0):
    from manifoldann_gb300 import _lib

    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n, d = pts.shape
    ids, dist = np.full((n, k), -7, np.int32), np.full((n, k), 7.0, np.float32)
    st = lib.mann_knn_graph_batched(_lib.params(_lib.METRIC_SQEUCLIDEAN, k, precision), pts.ctypes.data,
                                    offs.ctypes.data, len(sizes), d, include_self, ids.ctypes.data, dist.ctypes.data,
                                    None)
    return st, ids, dist


@pytest.mark.parametrize("precision", [1, 4])
@pytest.mark.parametrize("failure", ["refused", "launch"])
def test_fp32_plan_after_a_failed_tensor_core_call(gpu_lib, orc, precision, failure):
    from manifoldann_gb300 import _lib

    rng = np.random.default_rng(3)
    pts = rng.standard_normal((900, 16)).astype(np.float32)
    a, b = [300, 250, 350], [40, 460, 400]
    k = 7
    st, _, _ = _call(gpu_lib, pts, a, k, 0)
    assert st == _lib.MANN_OK
    if failure == "refused":  # more neighbours than the tensor-core forms keep
        st, _, _ = _call(gpu_lib, pts, b, 30, precision)
        assert st == _lib.MANN_EINVAL_ARG
    else:
        try:
            _lib.check(gpu_lib.mann_debug_inject(_lib.INJECT_LAUNCH, 1))
            st, _, _ = _call(gpu_lib, pts, b, k, precision)
            assert st == _lib.MANN_ECUDA
        finally:
            gpu_lib.mann_debug_inject(_lib.INJECT_LAUNCH, 0)
    st, ids, dist = _call(gpu_lib, pts, a, k, 0)
    assert st == _lib.MANN_OK
    o = 0
    for n in a:
        want, dw = orc.knn_graph_f32(pts[o:o + n], k, orc.SQEUCLIDEAN)
        assert np.array_equal(ids[o:o + n], want)
        assert np.array_equal(dist[o:o + n].view(np.uint32), dw.view(np.uint32))
        o += n
