"""node2vec with p = q = 1 reads the CSR only and builds nothing beside it; other
parameters build the extended columns and the edge filter, as they read them."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("host", [False, True], ids=["device", "host"])
def test_first_draw_walks_build_nothing(gpu, host):
    import torch
    s, d = oracle.rmat_clean_edges(12, 16, 0.57, 0.19, 0.19, 1)
    canon = oracle.canonical_from_edges(s, d)
    W, L = 5000, 9
    with gpu.Graph.rmat(12, 16, 0.57, 0.19, 0.19, seed=1, clean=True) as G:
        def paths(p, q):
            if host:
                return gpu.node2vec(G, W, L, p, q, 8, "uniform")
            out = torch.empty((W, L), dtype=torch.int32, device="cuda")
            gpu.node2vec(G, W, L, p, q, 8, "uniform", out=out)
            return out.cpu().numpy()

        for p, q in ((1.0, 1.0), (2.0, 0.5), (1.0, 1.0)):
            before = G.device_bytes
            got = paths(p, q)
            want, _ = oracle.replay_node2vec(canon, 0, W, L, 8, p, q, 1)
            assert np.array_equal(got, want)
            assert (G.device_bytes > before) == (p != 1.0)
