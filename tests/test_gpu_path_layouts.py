"""DeepWalk on extended columns and node2vec with p = q = 1 (its first draw is the
move) vs the oracle replay, at the walker counts where the launch changes, on a
directed multigraph with dead ends and sparse names."""
import numpy as np
import pytest

import oracle
from oracle.replay import START_UNIFORM

pytestmark = pytest.mark.gpu


def walkers(x):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return x if isinstance(x, int) else sms * x[0] + x[1]


@pytest.fixture(scope="module")
def small(gpu):
    rng = np.random.default_rng(6)
    names = np.sort(rng.choice(1 << 20, size=3000, replace=False)).astype(np.uint32)
    src = names[(rng.random(60000) ** 3 * 2950).astype(np.int64)]  # the last 50 names have no out-edge
    dst = names[(rng.random(60000) ** 2 * 3000).astype(np.int64)]
    G = gpu.Graph.from_edges(src, dst)
    yield G, oracle.canonical_from_edges(src, dst)
    G.close()


def named(canon, idx):
    return np.where(idx < 0, -1, canon.names[np.maximum(idx, 0)].astype(np.int64)).astype(np.int32)


@pytest.mark.parametrize("W", [1, 33, (1024, 0), (1024, 1), (2048, 37)])
@pytest.mark.parametrize("L", [1, 2, 33])
@pytest.mark.parametrize("hints", [0, 1])
def test_extended_columns(gpu, small, W, L, hints):
    G, canon = small
    W, first, tune = walkers(W), (5 << 32) + 3, G.tune
    try:
        G.tune = gpu.Tune(ext_columns=2, cache_hints=hints)
        got = gpu.deepwalk(G, W, L, 17, "uniform", first_walker=first)
    finally:
        G.tune = tune
    want = oracle.replay_paths(canon, first, first + W, L, 17, START_UNIFORM, threads=8)
    assert np.array_equal(got, named(canon, want))


@pytest.mark.parametrize("W", [1, 33, (512, 0), (512, 1), (1024, 0), (1024, 1), (2048, 37)])
@pytest.mark.parametrize("p,q", [(1.0, 1.0), (2.0, 0.5)])
def test_node2vec(gpu, small, W, p, q):
    G, canon = small
    W, L, first = walkers(W), 21, (1 << 33) + 9
    got, st = gpu.node2vec(G, W, L, p, q, 8, "uniform", first_walker=first, stats=True)
    want, trials = oracle.replay_node2vec(canon, first, first + W, L, 8, p, q, START_UNIFORM, threads=8)
    assert np.array_equal(got, named(canon, want))
    assert st.trials == trials and st.moves == int((got[:, 1:] >= 0).sum())
    if p == q == 1.0:
        assert st.checks == st.probes == 0
