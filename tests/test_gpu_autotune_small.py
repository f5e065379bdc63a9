"""The launch that the autotuner picks on a graph of less than one wave of vertices
serves later calls of several waves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# The sweep keeps the library's own launch unless another is faster beyond the
# spread of its timings; 1.5 leaves room for a busy machine (a launch picked at
# random took 1.2 to 23 times as long, or did not fit on an SM).
@pytest.mark.parametrize("scale", [10, 14])
def test_tuned_walk_of_several_waves(gpu, scale):
    W = 2_000_000
    with gpu.Graph.rmat(scale, 16, 0.57, 0.19, 0.19, seed=1, clean=True) as G:
        def took():
            runs = [gpu.pagerank(G, W, 0.15, 3, stats=True) for _ in range(5)]
            return min(st.kernel_ms for _, st in runs), runs[0][0]

        own, want = took()
        for _ in range(3):
            G.tune = gpu.Tune()
            G.autotune(0.15)
            ms, got = took()
            assert np.array_equal(got, want)
            assert ms <= 1.5 * own, G.tune
