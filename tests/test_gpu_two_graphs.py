"""Graphs with row tables of different sizes, used in turn and from two threads:
the kernels' shared memory limits belong to the functions that they share."""
import threading

import numpy as np
import pytest

import oracle
from oracle.replay import START_SOURCES

pytestmark = pytest.mark.gpu

DISTINCT = 4000  # distinct degrees: a row table of 56 KB


@pytest.fixture(scope="module")
def big(gpu):
    deg = np.arange(1, DISTINCT + 1)
    s = np.repeat(deg - 1, deg).astype(np.uint32)
    d = np.random.default_rng(1).integers(0, DISTINCT, s.size).astype(np.uint32)
    G = gpu.Graph.from_edges(s, d)
    yield G, oracle.canonical_from_edges(s, d)
    G.close()


def replay(canon, src, qid, budget, sp, seed):
    c, _ = oracle.replay_counts(canon, qid << 32, (qid << 32) + budget, sp, seed, START_SOURCES, [src])
    return c


@pytest.mark.parametrize("use_graph", [True, False])
def test_server_beside_a_smaller_graph(gpu, big, use_graph):
    G, canon = big
    queries = {k: (int(canon.names[37 * k]), 3000 + 500 * k) for k in range(6)}
    got = {}
    with gpu.Graph.rmat(10, 16, 0.57, 0.19, 0.19, seed=1, clean=True) as small, \
            gpu.Server(G, sp=0.2, seed=4, tick_walkers=8192, use_graph=use_graph) as srv:
        for k, (src, budget) in queries.items():
            srv.submit(src, budget, k)
        while len(got) < len(queries):
            gpu.ppr_batch(small, [0, 1], [500, 500], sp=0.2, seed=1).close()
            with gpu.Server(small, sp=0.2) as other:
                other.submit(0, 100, 0)
                other.drain()
            for r in srv.step():
                got[r["query_id"]] = r
    for k, (src, budget) in queries.items():
        want = replay(canon, src, k, budget, 0.2, 4)
        nz = np.nonzero(want)[0]
        assert np.array_equal(got[k]["names"], canon.names[nz])
        assert np.array_equal(got[k]["counts"], want[nz])


def test_two_threads(gpu, big):
    """One handle per thread, walks of more than one wave."""
    W = 400_000
    errors = []

    def batch(G):
        r = gpu.ppr_batch(G, [0, 1], [3000, 3000], sp=0.2, seed=1)
        out = np.concatenate(r.query(1))
        r.close()
        return out

    with gpu.Graph.rmat(16, 16, 0.57, 0.19, 0.19, seed=1, clean=True) as other:
        graphs = [big[0], other]
        calls = [lambda G: gpu.pagerank(G, W, 0.5, 3), lambda G: gpu.deepwalk(G, W, 4, 3), batch]
        want = [[f(G) for f in calls] for G in graphs]
        start = threading.Barrier(2)

        def loop(i):
            try:
                start.wait()
                for k in range(200):
                    c = k % len(calls)
                    if not np.array_equal(calls[c](graphs[i]), want[i][c]):
                        raise AssertionError("call %d of graph %d differs" % (c, i))
            except Exception as e:
                errors.append(e)

        threads = [threading.Thread(target=loop, args=(i,)) for i in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not errors, errors
