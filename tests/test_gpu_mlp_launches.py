"""Training where the device has no room for a cluster of 16 blocks, and where copies
from pageable memory read it late: gradients and parameters bit for bit as elsewhere."""
import pytest

import failing_lib

pytestmark = pytest.mark.gpu

# The epochs of a launch double (1, 2, 4, ...): 2^k - 1 of them leave no shorter
# launch at the end, so that a plan copied too late would still hold sample indices
# where the launch before it reads them.
TRAIN = """
    import hashlib
    from ptwalker_gb300 import learned
    fake({what}, True)
    h = hashlib.sha256()
    rng = np.random.default_rng(5)
    for N, batch, epochs in ((1, 1, 3), (300, 256, 7), (777, 300, 15), (2000, 64, 31)):
        x = rng.normal(0, 1, (N, 8)).astype(np.float32)
        t = (x[:, 0] - 0.5 * x[:, 1] ** 2).astype(np.float32)
        m = learned.MLP(seed=7)
        loss, g = m.grad(x, t)
        curve = m.train(x, t, epochs=epochs, batch=batch, lr=1e-3, seed=11)
        h.update(g.tobytes() + curve.tobytes() + m.params()[0].tobytes())
        m.close()
    print(h.hexdigest())
"""


@pytest.fixture(scope="module")
def failing(gpu, tmp_path_factory):
    return failing_lib.build("mlp.cu", tmp_path_factory.mktemp("lib"))


@pytest.mark.parametrize("what", [failing_lib.NO_CLUSTERS, failing_lib.LATE_COPIES])
def test_training(failing, what):
    want = failing_lib.run(None, TRAIN.format(what=what))
    assert failing_lib.run(failing, TRAIN.format(what=what)) == want
