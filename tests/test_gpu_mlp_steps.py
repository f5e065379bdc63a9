"""The MLP's gradient and training kernel (one cluster, tiles of 16 samples,
chunks of 256) vs the FP64 oracle, at batch sizes around tiles and chunks."""
import numpy as np
import pytest

from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


def model(seed):
    from ptwalker_gb300 import learned
    rng = np.random.default_rng(seed)
    m = learned.MLP(seed=seed)
    p, _ = m.params()
    p = p + rng.normal(0, 0.05, p.shape).astype(np.float32)
    norm = np.concatenate([rng.normal(0, 1, 8), rng.uniform(0.5, 2, 8), [0.3, 1.7]]).astype(np.float32)
    m.set_params(p, norm)
    return m, p, norm, rng


# FP32 sums of B terms in order against FP64: relative error up to about
# B * 2^-24 of the sum of magnitudes (2e-5 at B = 300); the bounds leave a
# factor of 50 for cancellation, as the gradient test at B = 333 does.
@pytest.mark.parametrize("B", [1, 15, 16, 17, 240, 255, 256, 257, 511, 4111])
def test_gradient_and_forward(gpu, B):
    m, p, norm, rng = model(B)
    x = rng.normal(0, 1.5, (B, 8)).astype(np.float32)
    t = rng.normal(0, 2, B).astype(np.float32)
    loss, g = m.grad(x, t)
    loss64, g64, y64 = omlp.forward_backward(p, norm, x, t)
    assert abs(loss - loss64) <= 1e-5 * max(1.0, loss64)
    np.testing.assert_allclose(g, g64, rtol=1e-3, atol=1e-5 * np.abs(g64).max())
    np.testing.assert_allclose(m.forward(x), y64 * norm[17] + norm[16], rtol=1e-4, atol=1e-4)
    loss2, g2 = m.grad(x, t)
    assert loss2 == loss and np.array_equal(g, g2)  # a fixed order of additions
    m.close()


@pytest.mark.parametrize("N,batch", [(1, 1), (40, 16), (300, 256), (513, 100), (257, 1000)])
def test_training_steps(gpu, N, batch):
    """The loss of the first epochs: every step's gradient, Adam update and
    order of samples enters the next one."""
    from ptwalker_gb300 import learned
    rng = np.random.default_rng(N)
    x = rng.normal(0, 1, (N, 8)).astype(np.float32)
    t = (x[:, 0] - 0.5 * x[:, 1] ** 2).astype(np.float32)
    m = learned.MLP(seed=7)
    p = m.params()[0].astype(np.float64)
    epochs, lr = 3, 1e-3
    curve = m.train(x, t, epochs=epochs, batch=batch, lr=lr, seed=11)
    norm = m.params()[1].astype(np.float64)
    m.close()
    mask, rs, perm = (1 << 64) - 1, (11 * 0x9E3779B97F4A7C15 + 1) & ((1 << 64) - 1), list(range(N))
    mom, var, step = np.zeros_like(p), np.zeros_like(p), 0
    batch = min(batch, N)
    for ep in range(epochs):
        for i in range(N - 1, 0, -1):
            rs = (rs * 6364136223846793005 + 1442695040888963407) & mask
            j = (rs >> 33) % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        losses = []
        for b0 in range(0, N, batch):
            idx = perm[b0:b0 + batch]
            loss, g, _ = omlp.forward_backward(p, norm, x[idx], t[idx])
            losses.append(loss)
            step += 1
            mom = 0.9 * mom + 0.1 * g
            var = 0.999 * var + 0.001 * g * g
            p = p - lr * (mom / (1 - 0.9 ** step)) / (np.sqrt(var / (1 - 0.999 ** step)) + 1e-8)
        # a gradient of rounding size may step the other way (2 lr) in FP32:
        # some of 4,801 weights by 1e-3 each, well inside 1% of the loss
        assert abs(curve[ep] - np.mean(losses)) <= 1e-2 * np.mean(losses) + 1e-6
