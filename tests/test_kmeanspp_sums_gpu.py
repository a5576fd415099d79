"""k-means++ draws at the edges of its blocked sums: block and slice remainders,
and distances whose ordered FP64 sums round (ranges past 53 bits), so that the
integer sums do not apply.  Chosen points equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(orc, X, k, seed):
    import manifoldann_gb300 as M

    rng = np.random.default_rng(seed)
    u = rng.random(k)
    first = int(rng.integers(len(X)))
    _, idx = M.init_kmeans_plus_plus(X.T, k, first=first + 1, u=u)
    assert np.array_equal(idx - 1, orc.kmeanspp(X, k, first, u))


@pytest.mark.parametrize("n,d", [(2, 1), (127, 3), (1023, 64), (1024, 65), (1025, 4), (5000, 130), (9217, 7), (140000, 5)])
def test_block_edges(gpu_lib, orc, n, d):
    X = np.random.default_rng(n).standard_normal((n, d)).astype(np.float32)
    check(orc, X, min(n, 30), n)


@pytest.mark.parametrize("span", [3, 8, 18])
def test_ranges_past_exact_sums(gpu_lib, orc, span):
    rng = np.random.default_rng(span)
    X = (rng.standard_normal((4500, 6)) * 10.0 ** rng.uniform(-span, span, (4500, 1))).astype(np.float32)
    X[100:160] = X[100]  # zero distances among them
    check(orc, X, 40, span)


def test_infinite_distances(gpu_lib, orc):
    X = np.random.default_rng(1).standard_normal((1500, 4)).astype(np.float32)
    X[7] = 3e38
    check(orc, X, 5, 3)
