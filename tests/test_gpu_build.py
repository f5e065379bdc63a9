"""CSR build and export vs the oracle where the build changes its ways: names from a
table over their range or by sorting the endpoints (a range of 4 names per entry is
the line), exports at the edges of a tile, one hub beside single edges, and
generators that drop self-loops and duplicates."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def check(G, canon):
    names, row_ptr, col = G.export_csr()
    assert np.array_equal(names, canon.names)
    assert np.array_equal(row_ptr, canon.row_ptr)
    assert np.array_equal(col, canon.col)
    assert G.max_degree == int(np.diff(canon.row_ptr.astype(np.int64)).max())


@pytest.mark.parametrize("und", [False, True])
@pytest.mark.parametrize("m", [1, 2, 5, 127, 128, 255, 256, 257, 513, 5001])
@pytest.mark.parametrize("bound", ["dense", "line", "line+1", 1 << 31, (1 << 32) - 1, 1 << 32])
def test_name_ranges(gpu, und, m, bound):
    rng = np.random.default_rng(m)
    line = 4 * m * (2 if und else 1)
    bound = {"dense": max(2, m // 8), "line": line, "line+1": line + 1}.get(bound, bound)
    src, dst = (rng.integers(0, bound, m, dtype=np.uint64).astype(np.uint32) for _ in range(2))
    dst[m // 2] = src[m // 2]  # a self-loop
    src[0] = bound - 1
    with gpu.Graph.from_edges(src, dst, as_undirected=und) as G:
        check(G, oracle.canonical_from_edges(src, dst, und))


@pytest.mark.parametrize("hub,leaves", [(300, 0), (256, 256), (10000, 777), (3, 100000)])
def test_hub_and_leaves(gpu, hub, leaves):
    src = np.concatenate([np.full(hub, 7, np.uint32), np.arange(100, 100 + leaves, dtype=np.uint32)])
    dst = np.concatenate([np.arange(hub, dtype=np.uint32) % 91, np.full(leaves, 7, np.uint32)])
    with gpu.Graph.from_edges(src, dst) as G:
        check(G, oracle.canonical_from_edges(src, dst))


@pytest.mark.parametrize("n,mean_degree", [(5, 2.0), (1000, 0.5), (3001, 8.0)])
def test_clean_generators_are_simple_and_symmetric(gpu, n, mean_degree):
    with gpu.Graph.chung_lu(n, mean_degree=mean_degree, seed=3) as G:
        names, row_ptr, col = G.export_csr()
    rows = np.repeat(np.arange(len(names), dtype=np.uint32), np.diff(row_ptr.astype(np.int64)))
    assert np.array_equal(names, np.arange(len(names), dtype=np.uint32))
    keys = rows.astype(np.uint64) << np.uint64(32) | col
    assert (np.diff(keys.astype(np.int64)) > 0).all() and (rows != col).all()
    assert np.array_equal(np.sort(col.astype(np.uint64) << np.uint64(32) | rows), keys)
    assert set(col.tolist()) == set(range(len(names)))
