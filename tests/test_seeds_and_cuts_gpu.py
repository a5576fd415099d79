"""The tensor-core form where its seed pass and its segmented pass's CTA ranges
can go wrong: sizes around the least sample, the densest sample and the
remainders of its stride, lists for every seed rank, and many-set layouts with
fewer items than CTAs, tiny sets and sets with no sampled point.  Ids and
distance bits equal the oracle's."""
import numpy as np
import pytest

from manifoldann_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nq,k", [(2047, 5000, 1), (2048, 5000, 10), (2049, 4900, 20), (4099, 2500, 4),
                                    (16389, 700, 24), (40003, 300, 2)])
@pytest.mark.parametrize("precision", ["bf16", "fp16"])
def test_single_set(gpu_lib, orc, n, nq, k, precision):
    import manifoldann_gb300 as M

    X = synthetic.anisotropic_clusters(n + nq, 40, seed=n, clusters=64)
    base, q = X[:n], X[n:]
    ids, d = M.knn_arrays(M.build_index(M.BruteForceIndex, base.T, distance=M.SqEuclidean()), base.T, q.T, k,
                          precision=precision)
    rows = np.random.default_rng(k).choice(nq, 200, replace=False)
    ids_o, d_o = orc.knn_f32(base, q[rows], k, 1)
    assert np.array_equal(ids[rows], ids_o)
    assert np.array_equal(d[rows].view(np.uint32), d_o.view(np.uint32))


@pytest.mark.parametrize("sizes", [[20], [16, 17, 127, 128, 129, 255, 256, 257], [20] * 300, [9000] + [18] * 40 + [2600]])
@pytest.mark.parametrize("k", [3, 15])
def test_many_sets(gpu_lib, orc, sizes, k):
    import manifoldann_gb300 as M

    clouds = synthetic.manifold_clouds(len(sizes), 10, 11, 12, seed=4)
    rng = np.random.default_rng(len(sizes))
    clouds = [(c[rng.integers(0, len(c), m)] + 0.3 * rng.standard_normal((m, 12))).astype(np.float32)
              for c, m in zip(clouds, sizes)]
    for _ in range(2):  # the second call runs the tuned list depth
        ids, d, offs = M.knn_graph_batched_arrays([c.T for c in clouds], k, distance=M.SqEuclidean(), precision="bf16")
    for c in range(0, len(sizes), max(1, len(sizes) // 12)):
        ids_o, d_o = orc.knn_graph_f32(clouds[c], k, 1)
        assert np.array_equal(ids[offs[c]:offs[c + 1]], ids_o)
        assert np.array_equal(d[offs[c]:offs[c + 1]].view(np.uint32), d_o.view(np.uint32))
