"""Launch parameters of walks beyond one wave (below it they do not matter) vs the
oracle replay: the column layouts, kernels and block sizes of k_walk and its
variants with more walkers than 1,024 per SM, and the same launches at the line."""
import numpy as np
import pytest

import oracle
from oracle.replay import START_UNIFORM

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small(gpu):
    rng = np.random.default_rng(8)
    names = np.sort(rng.choice(1 << 20, size=3000, replace=False)).astype(np.uint32)
    src = names[(rng.random(60000) ** 3 * 2950).astype(np.int64)]  # the last 50 names have no out-edge
    dst = names[(rng.random(60000) ** 2 * 3000).astype(np.int64)]
    G = gpu.Graph.from_edges(src, dst)
    yield G, oracle.canonical_from_edges(src, dst)
    G.close()


TUNES = [
    dict(block=768, ilp=2, chunk=64, hot_k=8192, ext_columns=3),
    dict(block=512, ilp=4, chunk=64, hot_k=512, ext_columns=1),
    dict(block=256, ilp=1, chunk=5, hot_k=0, cache_hints=0, ext_columns=1),
    dict(block=512, ilp=4, chunk=64, hot_k=0, min_blocks=2),
    dict(block=1024, ilp=2, chunk=256, hot_k=8192),
    dict(block=128, ilp=2, chunk=33, hot_k=300, blocks_per_sm=2),
    dict(block=256, ilp=2, chunk=64, hot_k=50, ext_columns=1, warp_agg=1),
    dict(block=128, ilp=2, chunk=5, hot_k=64, gather_slots=8, ext_columns=1),
]


@pytest.mark.parametrize("tune", TUNES)
@pytest.mark.parametrize("waves,more", [(1, 0), (1, 1), (2, 1111)])
def test_counts_and_pairs(gpu, small, tune, waves, more):
    import torch
    G, canon = small
    W = waves * torch.cuda.get_device_properties(0).multi_processor_count * 1024 + more
    saved, first = G.tune, (7 << 32) + 5
    try:
        G.tune = gpu.Tune(**tune)
        counts = gpu.pagerank(G, W, 0.3, 23, "uniform", first_walker=first)
        pairs = gpu.rwr(G, W, 0.4, 24, "uniform", first_walker=first)
    finally:
        G.tune = saved
    want, _ = oracle.replay_counts(canon, first, first + W, 0.3, 23, START_UNIFORM, threads=8)
    by_name = np.zeros(G.id_bound, dtype=np.uint32)
    by_name[canon.names] = want
    assert np.array_equal(counts, by_name)
    want, _ = oracle.replay_pairs(canon, first, first + W, 0.4, 24, START_UNIFORM)
    assert np.array_equal(pairs, canon.names[want])
