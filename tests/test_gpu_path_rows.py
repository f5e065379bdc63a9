"""DeepWalk paths of graphs with their first launch parameters (plain columns,
row table, paths written 32 positions at a time or from registers) vs the oracle
replay, at the sizes where kernel or launch change, on a directed multigraph with
dead ends and sparse names, into outputs at any 4-byte address."""
import numpy as np
import pytest

import oracle
from oracle.replay import START_PER_VERTEX, START_SOURCES, START_UNIFORM

pytestmark = pytest.mark.gpu

MODES = {"per_vertex": START_PER_VERTEX, "uniform": START_UNIFORM, "sources": START_SOURCES}


def lanes():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count * 1024


@pytest.fixture(scope="module")
def small(gpu):
    rng = np.random.default_rng(5)
    names = np.sort(rng.choice(1 << 20, size=3000, replace=False)).astype(np.uint32)
    src = names[(rng.random(60000) ** 3 * 2950).astype(np.int64)]  # the last 50 names have no out-edge
    dst = names[(rng.random(60000) ** 2 * 3000).astype(np.int64)]
    G = gpu.Graph.from_edges(src, dst)
    yield G, oracle.canonical_from_edges(src, dst)
    G.close()


def named(canon, idx):
    return np.where(idx < 0, -1, canon.names[np.maximum(idx, 0)].astype(np.int64)).astype(np.int32)


@pytest.mark.parametrize("W", [1, 31, 33, 4096, "lanes", "lanes+1", "2*lanes+37"])
@pytest.mark.parametrize("L,shift", [(1, 0), (2, 3), (5, 1), (31, 0), (32, 2), (33, 0), (80, 1), (64, 0)])
def test_deepwalk(gpu, small, W, L, shift):
    import torch
    G, canon = small
    W = eval(W, {"lanes": lanes()}) if isinstance(W, str) else W
    first = (3 << 32) + 11
    buf = torch.full((W * L + 4,), -7, dtype=torch.int32, device="cuda")
    gpu.deepwalk(G, W, L, 13, "uniform", out=buf[shift:shift + W * L], first_walker=first)
    got = buf.cpu().numpy()
    want = named(canon, oracle.replay_paths(canon, first, first + W, L, 13, START_UNIFORM, threads=8))
    assert np.array_equal(got[shift:shift + W * L].reshape(W, L), want)
    assert (got[:shift] == -7).all() and (got[shift + W * L:] == -7).all()


@pytest.mark.parametrize("W", [500, "lanes+500"])
@pytest.mark.parametrize("start", ["per_vertex", "sources"])
def test_deepwalk_starts_and_host_output(gpu, small, W, start):
    G, canon = small
    W = eval(W, {"lanes": lanes()}) if isinstance(W, str) else W
    src = [int(canon.names[i]) for i in (0, 7, 2999)] if start == "sources" else None  # the last one is a dead end
    got = gpu.deepwalk(G, W, 9, 4, start, sources=src)
    want = oracle.replay_paths(canon, 0, W, 9, 4, MODES[start], src, threads=8)
    assert np.array_equal(got, named(canon, want))
