// Compiled in front of one source of the library (-include) by failing_lib.py:
// CUDA calls that a test can make fail or delay on the host.
#pragma once
#include <cuda_runtime.h>

#include <cstring>
#include <vector>

namespace fake {
static int no_pool = 0, no_clusters = 0, late_copies = 0;

// Memory from a pool: out of memory on demand.
inline cudaError_t malloc_from_pool(void **p, size_t bytes, cudaMemPool_t pool, cudaStream_t st)
{
    return no_pool ? cudaErrorMemoryAllocation : cudaMallocFromPoolAsync(p, bytes, pool, st);
}

// A partition of the device without 16 SMs for one cluster.
template <typename T> cudaError_t max_clusters(int *n, T fn, const cudaLaunchConfig_t *cfg)
{
    if (no_clusters) {
        *n = 0;
        return cudaSuccess;
    }
    return cudaOccupancyMaxActiveClusters(n, fn, cfg);
}
template <typename... F, typename... A>
cudaError_t launch(const cudaLaunchConfig_t *cfg, void (*fn)(F...), A &&...args)
{
    for (unsigned i = 0; no_clusters && i < cfg->numAttrs; ++i)
        if (cfg->attrs[i].id == cudaLaunchAttributeClusterDimension && cfg->attrs[i].val.clusterDim.x > 8)
            return cudaErrorInvalidClusterSize;
    return cudaLaunchKernelEx(cfg, fn, static_cast<A &&>(args)...);
}

// A copy from pageable memory that reads it when the stream gets there, as the
// runtime may do where the device can read all host memory.
struct Late {
    const void *from;
    void *pinned;
    size_t bytes;
};
inline void CUDART_CB read_late(void *x)
{
    Late *l = static_cast<Late *>(x);
    std::memcpy(l->pinned, l->from, l->bytes);
    delete l;
}
inline cudaError_t copy(void *to, const void *from, size_t bytes, cudaMemcpyKind kind, cudaStream_t st)
{
    if (!late_copies || kind != cudaMemcpyHostToDevice) return cudaMemcpyAsync(to, from, bytes, kind, st);
    static std::vector<void *> kept;  // (until the process ends)
    void *pinned = nullptr;
    cudaError_t e = cudaMallocHost(&pinned, bytes);
    if (e != cudaSuccess) return e;
    kept.push_back(pinned);
    e = cudaLaunchHostFunc(st, read_late, new Late{from, pinned, bytes});
    return e == cudaSuccess ? cudaMemcpyAsync(to, pinned, bytes, kind, st) : e;
}
}  // namespace fake

extern "C" inline __attribute__((used, visibility("default"))) void ptw_test_fake(int what, int on)
{
    (what == 0 ? fake::no_pool : what == 1 ? fake::no_clusters : fake::late_copies) = on;
}

#define cudaMallocFromPoolAsync fake::malloc_from_pool
#define cudaOccupancyMaxActiveClusters fake::max_clusters
#define cudaLaunchKernelEx fake::launch
#define cudaMemcpyAsync fake::copy
