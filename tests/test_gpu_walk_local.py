"""Count and endpoint walks of graphs that are walked from shared memory (up to 160
KB of row records and columns) vs the oracle replay, at sizes that are no multiples
of a copy's 16 bytes and on both sides of the line."""
import numpy as np
import pytest

import oracle
from oracle.replay import START_PER_VERTEX, START_UNIFORM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("names,edges", [(1, 1), (2, 3), (3, 5), (50, 1001), (777, 30002), (500, 39960), (500, 39961),
                                         (500, 41000)])
@pytest.mark.parametrize("W", [1, 255, 257, 30000])
def test_walks(gpu, names, edges, W):
    rng = np.random.default_rng(names + edges)
    table = np.sort(rng.choice(1 << 20, size=names, replace=False)).astype(np.uint32)
    src, dst = (table[(rng.random(edges) ** 2 * names).astype(np.int64)] for _ in range(2))
    canon = oracle.canonical_from_edges(src, dst)
    first = (9 << 32) + 77
    with gpu.Graph.from_edges(src, dst) as G:
        counts = gpu.pagerank(G, W, 0.2, 31, "uniform", first_walker=first)
        pairs = gpu.rwr(G, W, 0.3, 32, "per_vertex", first_walker=first, max_moves=5)
        bound = G.id_bound
    want, _ = oracle.replay_counts(canon, first, first + W, 0.2, 31, START_UNIFORM, threads=4)
    by_name = np.zeros(bound, dtype=np.uint32)
    by_name[canon.names] = want
    assert np.array_equal(counts, by_name)
    want, _ = oracle.replay_pairs(canon, first, first + W, 0.3, 32, START_PER_VERTEX, max_moves=5)
    assert np.array_equal(pairs, canon.names[want])
