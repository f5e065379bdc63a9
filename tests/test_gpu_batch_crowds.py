"""Batched and served walks where the walkers of a query meet (tiny components,
stars, chains, vertices of low degree) and at the sizes of descriptors and
tables, with and without the row table, vs the oracle replay of each query
alone."""
import numpy as np
import pytest

import oracle
from oracle.replay import START_SOURCES

pytestmark = pytest.mark.gpu


def crowd_edges(distinct):
    """R-MAT plus small components; `distinct` vertices of degree 1, 2, ... more
    (names are sparse)."""
    s, d = oracle.rmat_clean_edges(10, 8, 0.57, 0.19, 0.19, 3)
    s, d = s.astype(np.int64) * 3, d.astype(np.int64) * 3
    extra = [(5000, 5001), (5001, 5000)]                                     # a pair
    extra += [(6000, 6000)]                                                  # a self-loop alone
    extra += [e for k in range(1, 40) for e in ((7000, 7000 + k), (7000 + k, 7000))]  # a star
    extra += [e for k in range(50) for e in ((8000 + k, 8001 + k), (8001 + k, 8000 + k))]  # a chain
    extra += [(9000, 9001)]                                                  # ends at once
    e = np.array(extra)
    s, d = np.concatenate([s, e[:, 0]]), np.concatenate([d, e[:, 1]])
    if distinct:
        deg = np.arange(1, distinct + 1)
        s = np.concatenate([s, np.repeat(10000 + deg, deg)])
        d = np.concatenate([d, 10000 + 1 + np.random.default_rng(1).integers(0, distinct, int(deg.sum()))])
    return s.astype(np.uint32), d.astype(np.uint32)


@pytest.fixture(scope="module", params=[0, 8300], ids=["row_table", "row_records"])
def crowd(gpu, request):
    s, d = crowd_edges(request.param)
    G = gpu.Graph.from_edges(s, d)
    yield G, oracle.canonical_from_edges(s, d)
    G.close()


SOURCES = [5000, 5001, 6000, 7000, 7003, 8000, 8025, 9000, 9001, 0, 3, 30]
BUDGETS = [1, 31, 32, 33, 255, 256, 257, 5000, 60000]


def want(canon, src, qid, budget, sp, app):
    w0 = qid << 32
    if app == "visits":
        return oracle.replay_counts(canon, w0, w0 + budget, sp, 6, START_SOURCES, [src], threads=4)[0]
    pairs, _ = oracle.replay_pairs(canon, w0, w0 + budget, sp, 6, START_SOURCES, [src])
    return np.bincount(pairs[:, 1], minlength=canon.n)


@pytest.mark.parametrize("app", ["visits", "endpoint"])
@pytest.mark.parametrize("ratio", [1, 64])  # hash tables for small budgets, dense arrays for nearly all
def test_batch(gpu, crowd, app, ratio):
    G, canon = crowd
    src = np.repeat(SOURCES, len(BUDGETS))
    bud = np.tile(BUDGETS, len(SOURCES))
    saved = gpu.get_batch_tune(G)
    gpu.set_batch_tune(G, gpu.BatchTune(dense_ratio=ratio))
    try:
        r = gpu.ppr_batch(G, src, bud, sp=0.2, seed=6, app=app)
    finally:
        gpu.set_batch_tune(G, saved)
    for i in range(len(src)):
        w = want(canon, int(src[i]), i, int(bud[i]), 0.2, app)
        nz = np.nonzero(w)[0]
        names, counts = r.query(i)
        assert np.array_equal(names, canon.names[nz]) and np.array_equal(counts, w[nz]), (src[i], bud[i])
    r.close()


def test_server(gpu, crowd):
    G, canon = crowd
    with gpu.Server(G, sp=0.2, seed=6, tick_walkers=1 << 14, table_bytes=1 << 28) as srv:
        for i, (s, b) in enumerate(zip(SOURCES, BUDGETS + BUDGETS)):
            srv.submit(s, b, i)
        res = {x["query_id"]: x for x in srv.drain()}
    for i, (s, b) in enumerate(zip(SOURCES, BUDGETS + BUDGETS)):
        w = want(canon, s, i, b, 0.2, "visits")
        nz = np.nonzero(w)[0]
        assert np.array_equal(res[i]["names"], canon.names[nz]) and np.array_equal(res[i]["counts"], w[nz])
