"""Full lists of batches whose tables have as many pieces (2 KB) as one block sums
up, fewer and more, vs the oracle replay of single queries."""
import numpy as np
import pytest

import oracle
from oracle.replay import START_SOURCES

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G16(gpu):
    G = gpu.Graph.rmat(16, 16, 0.57, 0.19, 0.19, seed=1, clean=True)
    yield G
    G.close()


# a dense table of the graph's 46,879 vertices has 12 chunks of 8 pieces
@pytest.mark.parametrize("nq", [1, 42, 43, 86, 341, 342])
def test_full_lists(gpu, G16, s16_canon, nq):
    rng = np.random.default_rng(nq)
    sources = rng.integers(0, G16.n, nq)
    budgets = np.where(np.arange(nq) % 50 == 7, 30, 20000)  # some hash tables between the dense ones
    res = gpu.ppr_batch(G16, sources, budgets, sp=0.2, seed=6)
    for i in sorted({0, nq // 2, min(7, nq - 1), min(8, nq - 1), nq - 1}):
        w0 = i << 32
        want, _ = oracle.replay_counts(s16_canon, w0, w0 + int(budgets[i]), 0.2, 6, START_SOURCES, [int(sources[i])])
        nz = np.nonzero(want)[0]
        names, counts = res.query(i)
        assert np.array_equal(names, nz.astype(np.uint32)) and np.array_equal(counts, want[nz])
