"""Probe training step by step: the trained parameters and losses against the
same batches driven one at a time through the gradient call, with AdamW in
numpy.  Batch counts below and above the point where steps replay a graph, a
ragged last batch, layer widths with padding, with and without the prior."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MASK = (1 << 64) - 1


def shuffled(n, state):
    """The library's seeded Fisher-Yates order; returns (order, next state)."""
    perm = np.arange(n)
    for i in range(n - 1, 0, -1):
        state = (state + 0x9E3779B97F4A7C15) & MASK
        z = state
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & MASK
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & MASK
        j = (z ^ (z >> 31)) % (i + 1)
        perm[i], perm[j] = perm[j], perm[i]
    return perm, state


@pytest.mark.parametrize("prior", [False, True])
@pytest.mark.parametrize("nq,batch,epochs", [(300, 128, 2), (1100, 128, 2), (640, 128, 4)])
def test_training_equals_its_gradient_steps(gpu_lib, nq, batch, epochs, prior):
    import manifoldann_gb300 as M

    din, h, nout, lr, wd = 20, 96, 200, 1e-3, 1e-2
    rng = np.random.default_rng(nq)
    X = rng.standard_normal((nq, din)).astype(np.float32)
    C = rng.standard_normal((nout, din)).astype(np.float32)
    labels = rng.integers(-1, nout, (nq, 3)).astype(np.int32)

    def make(params=None):
        return M.ProbeModel(din, nout, (h, h), use_prior=prior, centroids=C, batch=batch, lr=lr, weight_decay=wd,
                            seed=5, params=params)

    model = make()
    w = model.params().astype(np.float64)
    loss = model.train(X, labels, epochs)
    decay = np.zeros(w.size, bool)
    at = 0
    for rows, cols in ((h, din), (h, h), (nout, h)):
        decay[at:at + rows * cols] = True
        at += rows * cols + rows
    m, v = np.zeros_like(w), np.zeros_like(w)
    state, step = 5 ^ 0xC0FFEE, 0
    for e in range(epochs):
        order, state = shuffled(nq, state)
        losses = []
        for s in range(0, nq, batch):
            rows = order[s:s + batch]
            lo, g = make(w.astype(np.float32)).grad(X[rows], labels[rows])
            losses.append(lo)
            step += 1
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g.astype(np.float64) ** 2
            w = np.where(decay, w * (1 - lr * wd), w)
            w = w - lr * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
        assert np.isclose(loss[e], np.mean(losses), rtol=2e-3)
    # an update is about lr per step; rounding may flip BF16 copies, a wrong
    # batch, count or correction would move most weights by the whole update
    diff = np.abs(model.params() - w)
    assert diff.mean() < 0.02 * step * lr
