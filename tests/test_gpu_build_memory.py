"""What a graph's construction and its export leave mapped: the graph's own arrays, and
at most 1 GB of the pool that their buffers came from (or what the pool held before)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rmat(gpu):
    return gpu.Graph.rmat(23, 24, 0.57, 0.19, 0.19, seed=1, clean=True)  # 1.6 GB of edges


def chung_lu(gpu):
    return gpu.Graph.chung_lu(40_000_000, 2.5, 8.0, seed=1)  # 1.3 GB of edges, 0.6 GB of weights


def csr(gpu):
    n, per = 1 << 20, 200
    row_ptr = np.arange(n + 1, dtype=np.uint64) * per
    col = np.tile(np.arange(n, dtype=np.uint32), per)  # 0.8 GB, 1.7 GB of edges
    return gpu.Graph.from_csr(row_ptr, col)


def edges(gpu):
    m = 150_000_000  # 1.2 GB
    s = np.arange(m, dtype=np.uint32) & 0xFFFFF
    return gpu.Graph.from_edges(s, s[::-1])


def refused_csr(gpu):
    n, per = 1 << 20, 200
    row_ptr = np.arange(n + 1, dtype=np.uint64) * per
    col = np.full(n * per, n, dtype=np.uint32)  # columns out of range
    with pytest.raises(gpu.PTWError):
        gpu.Graph.from_csr(row_ptr, col)


@pytest.mark.parametrize("make", [rmat, chung_lu, csr, edges, refused_csr], ids=lambda f: f.__name__)
def test_memory_left_mapped(gpu, make):
    import torch
    gpu.Graph.rmat(4, 4, 0.57, 0.19, 0.19, seed=1, clean=True).close()  # the context and the pool exist
    gpu.trim_memory()
    free0 = torch.cuda.mem_get_info()[0]
    G = make(gpu)
    held = free0 - torch.cuda.mem_get_info()[0] - (G.device_bytes if G else 0)
    if G:
        G.close()
    gpu.trim_memory()
    # 1 GB, the rounding of nine arrays and of the pool to their granularities
    assert held <= (1 << 30) + (128 << 20)


def test_memory_left_mapped_by_export(gpu):
    import torch
    with rmat(gpu) as G:  # 1.4 GB of columns
        gpu.trim_memory()
        free0 = torch.cuda.mem_get_info()[0]
        names, row_ptr, col = G.export_csr()
        held = free0 - torch.cuda.mem_get_info()[0]
        assert col.nbytes > 1 << 30 and int(row_ptr[-1]) == G.m
    gpu.trim_memory()
    assert held <= (1 << 30) + (128 << 20)
