"""A launch that fails while k-means++ draws its centroids fails that call, at
any of its steps and in every form of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# points out of reach are left out from 2^23 coordinates on (two launches a step)
@pytest.mark.parametrize("n,d", [(3000, 8), (131073, 64)])
@pytest.mark.parametrize("nth", [1, 2, 7])
def test_injected_launch_error(gpu_lib, n, d, nth):
    from manifoldann_gb300 import _lib

    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, d)).astype(np.float32)
    k, u = 9, rng.random(9)

    def call():
        idx = np.full(k, -7, np.int64)
        return gpu_lib.mann_kmeanspp(X.ctypes.data, n, d, k, 5, u.ctypes.data, idx.ctypes.data), idx

    st, idx0 = call()
    assert st == _lib.MANN_OK
    try:
        _lib.check(gpu_lib.mann_debug_inject(_lib.INJECT_LAUNCH, nth))
        for _ in range(nth):  # each failure ends the call that meets it
            st, _ = call()
            assert st == _lib.MANN_ECUDA
            assert b"injected" in gpu_lib.mann_last_error()
        st, idx1 = call()
    finally:
        gpu_lib.mann_debug_inject(_lib.INJECT_LAUNCH, 0)
    assert st == _lib.MANN_OK and np.array_equal(idx0, idx1)
