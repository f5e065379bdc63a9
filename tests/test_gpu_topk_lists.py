"""Top-k lists where their sorting changes (tables that keep up to 4,096 entries are
sorted by a block each) vs the full lists of the same walks, and servers whose many
results and scattered tables are taken and cleared together vs the batch call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def star(gpu):
    """A hub with 6,000 leaves: a walk of one move ends at each about equally often,
    so thousands of counts tie."""
    leaves = np.arange(1, 6001, dtype=np.uint32)
    G = gpu.Graph.from_edges(np.zeros(6000, np.uint32), leaves, as_undirected=True)
    yield G
    G.close()


def expect(full, i, k):
    names, counts = full.query(i)
    order = np.lexsort((names, -counts.astype(np.int64)))[:k]
    return names[order], counts[order]


@pytest.mark.parametrize("nq", [1, 3, 1025, 2100])
@pytest.mark.parametrize("k", [1, 2, 1000, 4095, 4096, 4097, 1 << 20])
def test_lists(gpu, star, nq, k):
    rng = np.random.default_rng(nq + k)
    # the first query keeps nearly all leaves, then small ones and a few between
    budgets = rng.integers(1, 60, nq)
    budgets[:3] = [5500, 1, 40000][:min(3, nq)]
    sources = np.where(np.arange(nq) % 2 == 0, 0, 17)
    full = gpu.ppr_batch(star, sources, budgets, sp=0.4, seed=5)
    top = gpu.ppr_batch(star, sources, budgets, sp=0.4, seed=5, top_k=k)
    for i in list(range(min(nq, 6))) + [nq - 1, nq // 2]:
        names, counts = top.query(i)
        want_names, want_counts = expect(full, i, k)
        assert np.array_equal(names, want_names) and np.array_equal(counts, want_counts), i


@pytest.mark.parametrize("top_k", [0, 5])
def test_server_takes_many(gpu, star, top_k):
    rng = np.random.default_rng(top_k)
    budgets = rng.integers(1, 3000, 1200)
    budgets[::100] = 20000
    sources = rng.integers(0, 6001, 1200)
    want = gpu.ppr_batch(star, sources, budgets, sp=0.3, seed=9, top_k=top_k)
    # an arena of a few dozen tables: they are handed out in pieces and reused
    with gpu.Server(star, sp=0.3, seed=9, top_k=top_k, table_bytes=4 << 20, tick_walkers=1 << 14) as srv:
        for q in range(1200):
            srv.submit(int(sources[q]), int(budgets[q]), q)
        while srv.n_pending or srv.n_active or not srv.stats()["completed"]:
            srv.step(take=False)
        res = srv.results(copy=top_k == 0)
        assert srv.results() == []
        assert sorted(r["query_id"] for r in res) == list(range(1200))
        for r in res:
            names, counts = want.query(r["query_id"])
            assert r["source"] == sources[r["query_id"]] and r["budget"] == budgets[r["query_id"]]
            assert np.array_equal(r["names"], names) and np.array_equal(r["counts"], counts)
            assert r["names"].flags.writeable == (top_k == 0)
