"""Count and endpoint walks from one source, between calls from several, under launches
that read the source from a list and launches that take it as an argument."""
import numpy as np
import pytest

import oracle
from oracle.replay import START_SOURCES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walkers", [3000, 200_000])
def test_one_and_several(gpu, walkers):
    s, d = oracle.rmat_clean_edges(11, 8, 0.57, 0.19, 0.19, 5)
    s, d = s.astype(np.uint32) * 3 + 1, d.astype(np.uint32) * 3 + 1
    canon = oracle.canonical_from_edges(s, d)
    tunes = [gpu.Tune(), gpu.Tune(block=768, chunk=64, hot_k=8192, ext_columns=1),
             gpu.Tune(block=1024, hot_k=8192), gpu.Tune(chunk=64, hot_k=2048, warp_agg=1, ext_columns=1),
             gpu.Tune(chunk=64, gather_slots=8)]
    with gpu.Graph.from_edges(s, d) as G:
        for sources in (canon.names[[5]], canon.names[[900, 3]], canon.names[[41]]):
            want, _ = oracle.replay_counts(canon, 0, walkers, 0.4, 7, START_SOURCES, sources)
            pairs, _ = oracle.replay_pairs(canon, 0, walkers, 0.4, 7, START_SOURCES, sources)
            for t in tunes:
                G.tune = t
                got = gpu.pagerank(G, walkers, 0.4, 7, "sources", sources)
                assert np.array_equal(got[canon.names], want), t
                got = gpu.rwr(G, walkers, 0.4, 7, "sources", sources)
                assert np.array_equal(got, canon.names[pairs]), t
