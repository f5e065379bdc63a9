"""A sample whose error is infinite enters only the gradients of the units that were
active on it, at the sums' chunk edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,bad", [(16, 3), (256, 255), (300, 256), (300, 0)])
def test_infinite_error_stays_with_active_units(gpu, B, bad):
    from ptwalker_gb300 import learned
    rng = np.random.default_rng(B + bad)
    m = learned.MLP(seed=2)
    p, _ = m.params()
    norm = np.concatenate([np.zeros(8), np.ones(8), [0.0, 1.0]]).astype(np.float32)
    m.set_params(p, norm)
    x = rng.normal(0, 1, (B, 8)).astype(np.float32)
    t = rng.normal(0, 1, B).astype(np.float32)
    keep = np.arange(B) != bad
    _, rest = m.grad(x[keep], t[keep])
    t[bad] = np.inf
    _, g = m.grad(x, t)
    m.close()
    p = p.astype(np.float64)
    w1, b1, w2, b2 = p[:512].reshape(8, 64), p[512:576], p[576:4672].reshape(64, 64), p[4672:4736]
    a1 = np.maximum(x[bad].astype(np.float64) @ w1 + b1, 0)
    z2 = a1 @ w2 + b2
    hit = (a1 > 0)[:, None] & (z2 > 0)[None, :]
    got = g[576:4672].reshape(64, 64)
    assert hit.any() and not hit.all()
    assert np.array_equal(np.isfinite(got), ~hit)
    # the others are the sums over the rest, divided by B: FP32 sums of up to 300
    # terms in order, as in the gradient tests
    want = rest[576:4672].reshape(64, 64).astype(np.float64) * (B - 1) / B
    np.testing.assert_allclose(got[~hit], want[~hit], rtol=1e-3, atol=1e-5 * np.abs(want).max())
