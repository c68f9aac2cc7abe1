"""The training pass where its tiles end: the smallest batch, batches that wrap
around the data, more tiles than blocks, and the fixed order of its sums."""
import numpy as np
import pytest

import mlp_oracle
import wasl_b200

pytestmark = pytest.mark.gpu


def samples(seed, n, F):
    rng = np.random.Generator(np.random.PCG64(seed))
    return ((2.0 * rng.standard_normal((n, F))).astype(np.float32),
            (rng.uniform(size=n) < 0.25).astype(np.uint8))


@pytest.mark.parametrize("F", [16, 32, 48])
@pytest.mark.parametrize("n", [64, 192, 9536])
def test_gradient_over_any_number_of_tiles(F, n):
    """n = 64: two tiles; 9536: more tiles (298) than blocks (296)."""
    x, y = samples(F + n, n, F)
    with wasl_b200.Mlp(F, seed=F) as net:
        w = net.weights()
        g, loss = net.gradient(x, y, positive_weight=3.0)
        again, _ = net.gradient(x, y, positive_weight=3.0)
    loss_o, g_o = mlp_oracle.loss_and_gradient(w, x, y, 3.0)
    assert abs(loss - loss_o) <= 1e-5 * abs(loss_o)
    assert np.linalg.norm(g - g_o) <= 1e-3 * np.linalg.norm(g_o)
    assert np.array_equal(g, again)


@pytest.mark.parametrize("F", [16, 32, 48])
def test_batches_wrap_around_the_data(F):
    """100 samples, batches of 192: each step's gradient is that of the wrapped
    samples, and Adam's update (FP32, lr 1e-3) follows from it; training twice
    from the same weights gives the same bits."""
    x, y = samples(F, 100, F)
    with wasl_b200.Mlp(F, seed=1) as net, wasl_b200.Mlp(F, seed=1) as twin:
        w = net.weights().astype(np.float64)
        for n in (net, twin):
            n.set_data(x, y)
        m1, m2 = np.zeros_like(w), np.zeros_like(w)
        for step in range(1, 4):
            at = (192 * (step - 1) + np.arange(192)) % 100
            g, loss_g = net.gradient(x[at], y[at], positive_weight=2.0)
            g = g.astype(np.float64)
            loss = net.train(1, batch=192, learning_rate=1e-3, positive_weight=2.0)
            assert abs(loss - loss_g) <= 1e-6 * abs(loss_g)
            m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
            # FP32: each update is within a few rounding steps of lr = 1e-3,
            # and 1 - beta2^step loses up to 2^-24 / 1e-3 of itself.
            w = w - 1e-3 * (m1 / (1 - 0.9 ** step)) / (np.sqrt(m2 / (1 - 0.999 ** step)) + 1e-8)
            assert np.max(np.abs(net.weights() - w)) <= step * (1e-3 * 1e-4 + 2e-7)
        twin.train(3, batch=192, learning_rate=1e-3, positive_weight=2.0)
        assert np.array_equal(net.weights(), twin.weights())
