"""The cost model's kernels at the edges of their shapes: rows around the
chunk of 256 staged at a time and around a CTA's 8, feature counts around the
groups of 4 weight rows, mini-batches with a short last one."""
import numpy as np
import pytest

import mlp_ref

pytestmark = pytest.mark.gpu


def _data(n, n_in, seed):
    rng = np.random.default_rng(seed)
    return (rng.normal(size=(n, n_in)).astype(np.float32), rng.normal(size=n).astype(np.float32))


@pytest.mark.parametrize("n_in", [1, 3, 4, 5, 38, 64])
def test_gradient_and_prediction(gat, n_in):
    from graphautotune_b200 import costmodel

    for n in (1, 7, 8, 9, 255, 256, 257, 600):
        m = costmodel.MLP(n_in, seed=n)
        X, T = _data(n, n_in, n)
        grad, loss = m.gradient(X, T)
        want_loss, want = mlp_ref.loss_and_grad(m.params(), X, T, n_in)
        # fp32 sums in order: at most a rounding (2^-24) per term of every
        # sum on the way, against the size of the terms
        u = (n_in + 64 + 64 + 64 + n + 16) * 2.0 ** -24
        size = np.abs(want).max() * np.sqrt(n) + 1e-30
        assert np.abs(grad - want).max() <= 8 * u * size, (n, n_in)
        assert abs(loss - want_loss) <= 8 * u * max(want_loss, 1e-3)
        y = mlp_ref.forward(m.params(), X, n_in)[0]
        assert np.abs(m.predict(X) - y).max() <= 8 * u * max(np.abs(y).max(), 1.0)


@pytest.mark.parametrize("n,batch", [(1, 1), (9, 4), (257, 256), (300, 300), (600, 1000)])
def test_training_steps(gat, n, batch):
    """The first Adam step moves every parameter by lr against its gradient's
    sign; the same training twice gives the same parameters."""
    from graphautotune_b200 import costmodel

    n_in, lr = 38, 1e-3
    X, T = _data(n, n_in, n)
    m = costmodel.MLP(n_in, seed=1)
    p0 = m.params()
    _, g = mlp_ref.loss_and_grad(p0, X, T, n_in)
    m.train(X, T, epochs=1, batch=max(batch, n), lr=lr, seed=5)
    sure = np.abs(g) > 1e-3 * np.abs(g).max()
    assert np.allclose((m.params() - p0)[sure], -lr * np.sign(g[sure]), rtol=0, atol=1e-2 * lr)
    runs = []
    for _ in range(2):
        m.set_params(p0)
        m.train(X, T, epochs=3, batch=batch, lr=lr, seed=7)
        runs.append(m.params())
    assert np.array_equal(runs[0], runs[1])
    assert not np.array_equal(runs[0], p0)
