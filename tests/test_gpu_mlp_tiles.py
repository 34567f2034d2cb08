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


def _mt19937_64(seed):
    """std::mt19937_64 (the C++ standard's linear_congruential-seeded 64-bit
    Mersenne twister with its published parameters)."""
    mask = (1 << 64) - 1
    x = [seed & mask]
    for i in range(1, 312):
        x.append((6364136223846793005 * (x[-1] ^ (x[-1] >> 62)) + i) & mask)
    i = 312
    while True:
        if i == 312:
            for k in range(312):
                y = (x[k] & 0xFFFFFFFF80000000) | (x[(k + 1) % 312] & 0x7FFFFFFF)
                x[k] = x[(k + 156) % 312] ^ (y >> 1) ^ (0xB5026F5AA96619E9 if y & 1 else 0)
            i = 0
        y = x[i]
        y ^= (y >> 29) & 0x5555555555555555
        y ^= (y << 17) & 0x71D67FFFEDA60000
        y ^= (y << 37) & 0xFFF7EEE000000000
        yield y ^ (y >> 43)
        i += 1


@pytest.mark.parametrize("n,batch,epochs", [(513, 513, 1), (2048, 2048, 1), (100, 32, 1), (700, 129, 2),
                                            (1030, 515, 1), (1500, 600, 1), (2049, 1024, 1), (4200, 2100, 1)])
def test_training_reads_the_rows_of_each_batch(n, batch, epochs):
    """Rows that all differ, in the order of the seeded shuffle (Fisher-Yates):
    a batch that reads other rows than its own, one row twice or a neighbour's,
    takes other steps.  A parameter is compared where its gradient stands clear of
    FP32 noise in every step; a step moves it by up to 1e-3."""
    import vine_b200 as v
    from oracle import mlp_ref
    x, y = _data(n, 31)
    m = v.MLP(seed=9)
    p = m.params.astype(np.float64)
    mm, vv, k = np.zeros_like(p), np.zeros_like(p), 0
    rng, order, clear = _mt19937_64(77), np.arange(n), np.ones(p.shape, bool)
    for _ in range(epochs):
        for i in range(n - 1, 0, -1):
            j = next(rng) % (i + 1)
            order[i], order[j] = order[j], order[i]
        for b in range(0, n, batch):
            rows = order[b:b + batch]
            _, g = mlp_ref.loss_grad(p, x[rows], y[rows])
            clear &= np.abs(g) > 1e-3 * np.abs(g).max()
            k += 1
            p, mm, vv = mlp_ref.adam_step(p, mm, vv, g, k, 1e-3)
    m.train(x, y, epochs=epochs, batch=batch, lr=1e-3, seed=77)
    assert clear.mean() > 0.2
    np.testing.assert_allclose(m.params[clear], p[clear], rtol=0, atol=2e-5 * k)
