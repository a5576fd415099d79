"""The register form of the local PCA where its lane groups can go wrong: the
neighbour counts at which the group width changes, dimensions at which its
register width changes, gaps in the neighbour rows, missing centres and a
number of centres that leaves a warp partly empty.  Each centre's fit equals
the fit of that centre alone in a full-width row (bit for bit), and the
oracle's eigenvalues."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2, 7, 8, 9, 15, 16, 17, 31])
@pytest.mark.parametrize("d,dim", [(3, 2), (8, None), (9, 2), (16, None), (20, 3), (32, None)])
def test_groups(gpu_lib, k, d, dim):
    import manifoldann_gb300 as M
    from oracle import pca as opca

    rng = np.random.default_rng(100 * k + d)
    n, m = 300, 37
    X = (rng.standard_normal((n, d)) * np.linspace(3.0, 0.2, d)).astype(np.float32)
    nb = np.stack([rng.choice(n, k, replace=False) + 1 for _ in range(m)])
    nb[rng.random((m, k)) < 0.15] = 0  # gaps
    nb[5] = 0  # no neighbours at all
    centres = rng.integers(1, n + 1, m)
    method = M.PCAMethod(intrinsic_dim=dim, min_variance_ratio=0.9)
    dims, eig, basis = M.fit_geometries(method, X.T, nb, centers=centres)
    wide = np.zeros((m, 32), nb.dtype)  # the same neighbours in 32-wide rows, gaps kept
    wide[:, :k] = nb
    dw, ew, bw = M.fit_geometries(method, X.T, wide, centers=centres)
    r = min(d, k)
    assert np.array_equal(dims, np.minimum(dw, r))
    assert np.array_equal(eig.view(np.uint32), ew[:, :r].view(np.uint32))
    assert np.array_equal(basis.view(np.uint32), bw[:, :r].view(np.uint32))
    for i in range(m):
        own = nb[i][nb[i] > 0] - 1
        if len(own) >= 2:
            _, vals, _ = opca.fit_pca(X[centres[i] - 1], X[own], intrinsic_dim=dim, min_variance_ratio=0.9)
            got = eig[i, :dims[i]]
            mm = min(len(got), len(vals))
            # one-sided Jacobi in FP32: errors of a few (d + k) u of the largest eigenvalue
            assert np.allclose(got[:mm], vals[:mm], rtol=0, atol=8 * (d + k) * 2.0**-24 * float(vals[0]))
