"""The inverted-list scan at the edges of its passes and of its selection: list
lengths around one and two passes, empty lists, list lengths of one lane,
results longer than a list, equal distances, more queries per list than a
chunk, dimensions around a stage.  Equal to the oracle's exact search of the
probed points (ties at the k-th place to the lower id)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 10, 31, 32, 33, 64])
@pytest.mark.parametrize("d,nq,kind", [(8, 40, "plain"), (128, 7, "plain"), (130, 70, "plain"), (33, 20, "equal"),
                                       (16, 9, "falling")])
def test_scan(gpu_lib, orc, k, d, nq, kind):
    import manifoldann_gb300 as M

    sizes = [0, 1, 5, 31, 32, 33, 255, 256, 257, 511, 513, 900]
    n, nlist = sum(sizes), len(sizes)
    rng = np.random.default_rng(k * 1000 + d)
    X = rng.standard_normal((n, d)).astype(np.float32)
    if kind == "equal":
        X = rng.integers(0, 2, (n, d)).astype(np.float32)
        X[:, 3:] = 0.0
    elif kind == "falling":  # every point of a list is nearer than the one before it
        X[:] = 0.0
        X[:, 0] = np.arange(n, 0, -1)
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    ids = np.arange(n, dtype=np.int32) if kind == "falling" else np.concatenate(
        [np.sort(p) for p in np.split(rng.permutation(n), offs[1:-1])]).astype(np.int32)
    C = rng.standard_normal((nlist, d)).astype(np.float32)
    Q = np.zeros((nq, d), np.float32) if kind == "falling" else rng.standard_normal((nq, d)).astype(np.float32)
    index = M.IVFFlatIndex(np.asfortranarray(C.T), (C**2).sum(1), offs, ids, d, 4, M.SqEuclidean(), M.Euclidean())
    for nprobe in (4, nlist):
        got, dist = index.search_arrays(X.T, Q.T, k, nprobe=nprobe)
        probes, _ = orc.knn_f32(C, Q, nprobe, orc.EUCLIDEAN)
        for r in range(nq):
            own = np.sort(np.concatenate([ids[offs[c]:offs[c + 1]] for c in probes[r]]))
            m = min(k, len(own))
            assert np.all(got[r, m:] == -1)
            if m:
                want, dw = orc.knn_f32(X[own], Q[r:r + 1], m, orc.SQEUCLIDEAN)
                assert np.array_equal(got[r, :m], own[want[0]])
                assert np.array_equal(dist[r, :m].view(np.uint32), dw[0].view(np.uint32))
