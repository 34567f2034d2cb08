"""The network's tiled kernels at the edges of their tiles and of a training
batch's split over the cluster, against the FP64 restatement.

Tolerances are those of the other network tests: FP32 sums of at most a few
thousand terms against FP64 (1e-4 forward, 2e-3 gradients), 2e-5 a step for
parameters whose gradient stands clear of FP32 noise."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(0, 1.5, (n, 16)).astype(np.float32)
    y = np.stack([np.sin(x[:, 0]) + 0.3 * x[:, 3], 0.5 * x[:, 1] - 0.2 * x[:, 7]], 1).astype(np.float32)
    return x, y


@pytest.mark.parametrize("n", [1, 4, 63, 64, 65, 128, 64 * 296 + 1, 1 << 19])
def test_forward_and_gradient(n):
    import vine_b200 as v
    from oracle import mlp_ref
    x, y = _data(n, 23)
    m = v.MLP(seed=4)
    want, _ = mlp_ref.forward(m.params, x)
    np.testing.assert_allclose(m.forward(x), want, rtol=1e-4, atol=1e-4)
    loss, grad = m.loss_grad(x, y)
    wl, wg = mlp_ref.loss_grad(m.params, x, y)
    assert abs(loss - wl) <= 1e-4 * max(1.0, abs(wl))
    np.testing.assert_allclose(grad, wg, rtol=2e-3, atol=2e-5 * np.abs(wg).max())


@pytest.mark.parametrize("n,batch", [(3, 1), (40, 31), (70, 32), (513, 512), (1030, 515), (2049, 2048),
                                     (4200, 2049), (900, 4000)])
def test_training_steps(n, batch):
    """All rows alike: every shuffle gives the same batches, the last one
    shorter, so an epoch is ceil(n / batch) known Adam steps.  2049 and more
    rows a batch take one launch a step."""
    import vine_b200 as v
    from oracle import mlp_ref
    x, y = _data(1, 5)
    m = v.MLP(seed=7)
    p = m.params.astype(np.float64)
    mm, vv = np.zeros_like(p), np.zeros_like(p)
    _, g0 = mlp_ref.loss_grad(p, x, y)
    steps = -(-n // batch)
    for k in range(steps):
        _, g = mlp_ref.loss_grad(p, x, y)
        p, mm, vv = mlp_ref.adam_step(p, mm, vv, g, k + 1, 1e-3)
    loss = m.train(np.repeat(x, n, 0), np.repeat(y, n, 0), epochs=1, batch=batch, lr=1e-3, seed=1)
    ok = np.abs(g0) > 1e-4 * np.abs(g0).max()
    np.testing.assert_allclose(m.params[ok], p[ok], rtol=0, atol=2e-5 * steps)
    wl, _ = mlp_ref.loss_grad(p, x, y)
    assert abs(loss - wl) <= 2e-3 * max(1.0, abs(wl))
