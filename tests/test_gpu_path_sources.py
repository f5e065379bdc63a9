"""DeepWalk from one source and from several under every path launch (untouched and
tuned, each column layout and walkers per lane), to the host and to the device."""
import numpy as np
import pytest

import oracle
from oracle.replay import START_SOURCES

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph(gpu):
    s, d = oracle.rmat_clean_edges(11, 8, 0.57, 0.19, 0.19, 5)
    s, d = s.astype(np.uint32) * 3 + 1, d.astype(np.uint32) * 3 + 1
    with gpu.Graph.from_edges(s, d) as G:
        yield G, oracle.canonical_from_edges(s, d)


@pytest.mark.parametrize("W,L", [(1, 2), (33, 32), (4500, 64), (200_000, 5)])
@pytest.mark.parametrize("sources", [[17], [100, 5, 900]], ids=["one", "several"])
def test_deepwalk_from_sources(gpu, graph, sources, W, L):
    import torch
    G, canon = graph
    names = canon.names[sources]
    want = oracle.replay_paths(canon, 7, 7 + W, L, 3, START_SOURCES, names)
    want = np.where(want < 0, -1, canon.names[np.maximum(want, 0)].astype(np.int32))
    tunes = [gpu.Tune()] + [gpu.Tune(paths_ilp=i, paths_named=n, ext_columns=e, cache_hints=h)
                            for i in (1, 2, 4) for n, e, h in ((0, 0, 1), (1, 0, 0), (0, 2, 1))]
    for t in tunes:
        G.tune = t
        got = gpu.deepwalk(G, W, L, 3, "sources", sources=names, first_walker=7)
        assert np.array_equal(got, want), t
        out = torch.empty((W, L), dtype=torch.int32, device="cuda")
        gpu.deepwalk(G, W, L, 3, "sources", sources=names, first_walker=7, out=out)
        assert np.array_equal(out.cpu().numpy(), want), t
    G.tune = gpu.Tune()
