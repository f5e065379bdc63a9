"""Launch parameters with which the walk kernel does not fit on an SM are refused
whatever the number of walkers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walkers", [31, 24_133, 155_648, 400_000])
@pytest.mark.parametrize("call", ["pagerank", "rwr"])
def test_unfit_launch(gpu, call, walkers):
    f = getattr(gpu, call)
    with gpu.Graph.rmat(10, 16, 0.57, 0.19, 0.19, seed=1, clean=True) as G:
        want = f(G, walkers, 0.5, 3)
        for ext in (0, 1):
            G.tune = gpu.Tune(block=1024, ilp=4, ext_columns=ext)
            with pytest.raises(gpu.PTWError, match="does not fit on an SM"):
                f(G, walkers, 0.5, 3)
            G.tune = gpu.Tune(block=512, ilp=4, ext_columns=ext)
            assert np.array_equal(f(G, walkers, 0.5, 3), want)
