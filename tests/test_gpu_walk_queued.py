"""Walks of graphs with their first launch parameters (one walker per lane, a
second one queued behind it, rows from the row table) vs the oracle replay, at
the sizes where kernel, layout or launch change."""
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
    """A directed multigraph with dead ends, self-loops and sparse names."""
    rng = np.random.default_rng(3)
    names = np.sort(rng.choice(1 << 20, size=3000, replace=False)).astype(np.uint32)
    src = names[(rng.random(40000) ** 3 * 2500).astype(np.int64)]  # the last 500 names have no out-edge
    dst = names[rng.integers(0, 3000, 40000)]
    G = gpu.Graph.from_edges(src, dst)
    yield G, oracle.canonical_from_edges(src, dst)
    G.close()


def check(gpu, G, canon, W, start, sp, max_moves=0, n_sources=1, first=0):
    src = None
    if start == "sources":
        src = canon.names[np.linspace(0, canon.n - 1, n_sources).astype(np.int64)].tolist()
    got, st = gpu.pagerank(G, W, sp, 9, start, src, max_moves, first_walker=first, stats=True)
    idx, moves = oracle.replay_counts(canon, first, first + W, sp, 9, MODES[start], src, max_moves, threads=8)
    want = np.zeros(G.id_bound, np.uint32)
    want[canon.names] = idx
    assert np.array_equal(got, want) and st.moves == moves
    got, st = gpu.rwr(G, W, sp, 9, start, src, max_moves, first_walker=first, stats=True)
    want, moves = oracle.replay_pairs(canon, first, first + W, sp, 9, MODES[start], src, max_moves)
    assert np.array_equal(got, canon.names[want]) and st.moves == int(np.sum(moves))


@pytest.mark.parametrize("W", [1, 31, 33, 24575, 24576, "lanes-1", "lanes", "lanes+1", "2*lanes+37"])
@pytest.mark.parametrize("start,n_sources", [("per_vertex", 0), ("uniform", 0), ("sources", 1), ("sources", 3)])
def test_launch_sizes(gpu, small, W, start, n_sources):
    W = eval(W, {"lanes": lanes()}) if isinstance(W, str) else W
    check(gpu, *small, W, start, 0.15, n_sources=n_sources, first=(5 << 32) + 3 if n_sources else 0)


@pytest.mark.parametrize("W", [1000, "lanes+4099"])
@pytest.mark.parametrize("sp,max_moves", [(1.0, 0), (0.001, 7), (0.5, 1)])
def test_terminations(gpu, small, W, sp, max_moves):
    W = eval(W, {"lanes": lanes()}) if isinstance(W, str) else W
    check(gpu, *small, W, "uniform", sp, max_moves)


@pytest.mark.parametrize("degrees", [
    np.full(700, 3),                 # one run
    np.arange(1, 2200),              # every vertex a run, past the single-id buckets
    np.repeat(np.arange(1, 40), 97),
    np.arange(0, 8193),              # one run more than the table holds: row records from memory
    np.arange(0, 8192),              # exactly full
], ids=["one", "distinct", "blocks", "too_many", "full"])
def test_row_tables(gpu, degrees):
    rng = np.random.default_rng(len(degrees))
    n = len(degrees)
    degrees = rng.permutation(degrees)
    row_ptr = np.concatenate([[0], np.cumsum(degrees)]).astype(np.uint64)
    col = rng.integers(0, n, int(row_ptr[-1])).astype(np.uint32)
    col[:n] = rng.permutation(n)  # every vertex is some vertex's neighbour
    with gpu.Graph.from_csr(row_ptr, col) as G:
        src = np.repeat(np.arange(n, dtype=np.uint32), degrees)
        canon = oracle.canonical_from_edges(src, col)
        check(gpu, G, canon, lanes() + 1000, "per_vertex", 0.3)
