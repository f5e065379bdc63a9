// Device graph construction: canonical CSR + degree-sorted relabelling.
//
// Replaces the reference loader's CSR build and NUMA/cache partitioner
// (src/core/graph.hpp:277-785).  The reference compacts names in first
// appearance order, splits hubs (degree >= --db) from low-degree vertices,
// runs a max-cut split and L2-sized chunks and relabels randomly; all of that
// exists to keep CPU partitions cache-resident.  On one GB300 the whole CSR
// sits in HBM, so the only relabelling kept is by descending degree: the rows,
// counters and column blocks of hub vertices land at the low end of every
// array, where the 129 MB L2 keeps them.
//
// Pipeline (all on the graph's stream):
//   edges -> names = ascending distinct endpoints, index of every name ->
//   packed u64 keys (src index << b | dst index) [without self-loops] -> radix
//   sort -> [unique] -> row bounds, degrees -> stable sort by degree (desc) ->
//   internal CSR.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "ptw_internal.cuh"

namespace ptw {
namespace {

constexpr int kThreads = 256;

inline unsigned grid_for(uint64_t n, int threads = kThreads)
{
    uint64_t b = (n + threads - 1) / threads;
    return (unsigned)std::min<uint64_t>(std::max<uint64_t>(b, 1), 1u << 20);
}

// Largest of 2m names; one atomic per block.
__global__ void __launch_bounds__(kThreads) k_max2(const uint32_t *a, const uint32_t *b, uint64_t m, unsigned *out)
{
    __shared__ unsigned s_mx[kThreads / 32];
    unsigned mx = 0;
    const uint64_t t = blockIdx.x * (uint64_t)kThreads + threadIdx.x, stride = (uint64_t)gridDim.x * kThreads;
    const uint4 *a4 = reinterpret_cast<const uint4 *>(a), *b4 = reinterpret_cast<const uint4 *>(b);
    for (uint64_t i = t; i < m / 4; i += stride) {
        const uint4 x = a4[i], y = b4[i];
        mx = max(mx, max(max(max(x.x, x.y), max(x.z, x.w)), max(max(y.x, y.y), max(y.z, y.w))));
    }
    for (uint64_t i = (m & ~3ull) + t; i < m; i += stride) mx = max(mx, max(a[i], b[i]));
    mx = __reduce_max_sync(0xffffffffu, mx);
    if ((threadIdx.x & 31) == 0) s_mx[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x < kThreads / 32) {
        mx = __reduce_max_sync((1u << (kThreads / 32)) - 1, s_mx[threadIdx.x]);
        if (threadIdx.x == 0) atomicMax(out, mx);
    }
}

// seen[x] = 1 for both names of every edge (of every edge that is not a
// self-loop), *n_out += edges.  A name already seen is only read: hubs stay in L1.
__global__ void __launch_bounds__(kThreads) k_mark_names(const uint32_t *src, const uint32_t *dst, uint64_t m,
                                                         bool drop_loops, uint32_t *seen, unsigned long long *n_out)
{
    __shared__ unsigned long long s_n;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    unsigned n = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)kThreads + threadIdx.x; i < m; i += (uint64_t)gridDim.x * kThreads) {
        const uint32_t u = src[i], v = dst[i];
        if (drop_loops && u == v) continue;
        ++n;
        if (!seen[u]) seen[u] = 1;
        if (!seen[v]) seen[v] = 1;
    }
    if (n) atomicAdd(&s_n, (unsigned long long)n);
    __syncthreads();
    if (threadIdx.x == 0 && s_n) atomicAdd(n_out, s_n);
}

// names[index_of[x]] = x of every name seen (index_of: exclusive sums of the
// marks, [bound + 1]); *n_out = their number.
__global__ void k_collect_names(const uint32_t *index_of, uint64_t bound, uint32_t *names, unsigned long long *n_out)
{
    for (uint64_t x = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; x < bound; x += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t i = index_of[x], j = index_of[x + 1];
        if (i != j) names[i] = (uint32_t)x;
        if (x + 1 == bound) *n_out = j;
    }
}

__device__ __forceinline__ uint32_t lower_bound_u32(const uint32_t *a, uint32_t n, uint32_t x)
{
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        uint32_t mid = lo + ((hi - lo) >> 1);
        if (a[mid] < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// keys[i] = (index of src[i]) << bits | index of dst[i], and the reverse in
// keys[m + i] (both).  A dropped self-loop becomes the last key of all: no kept
// edge of a graph without loops equals it.  index_of null: indices by search of
// the n names.
__global__ void k_make_keys(const uint32_t *src, const uint32_t *dst, uint64_t m, int bits, bool both, bool drop_loops,
                            const uint32_t *index_of, const uint32_t *names, uint32_t n, unsigned long long *keys)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t u = src[i], v = dst[i];
        unsigned long long k = ~0ull >> (64 - 2 * bits), r = k;
        if (!(drop_loops && u == v)) {
            const unsigned long long a = index_of ? index_of[u] : lower_bound_u32(names, n, u);
            const unsigned long long b = index_of ? index_of[v] : lower_bound_u32(names, n, v);
            k = a << bits | b;
            r = b << bits | a;
        }
        keys[i] = k;
        if (both) keys[m + i] = r;
    }
}

// Row bounds from the sorted keys, without atomics (a hub of
// degree d would otherwise serialise d atomics on one counter): the first
// entry of a run of v records first[v], the last records end[v].
__global__ void k_row_bounds(const unsigned long long *keys, uint64_t m, int bits, uint32_t *first, uint32_t *end)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = (uint32_t)(keys[i] >> bits);
        if (i == 0 || (uint32_t)(keys[i - 1] >> bits) != v) first[v] = (uint32_t)i;
        if (i + 1 == m || (uint32_t)(keys[i + 1] >> bits) != v) end[v] = (uint32_t)(i + 1);
    }
}

// deg[v] = end[v] - first[v] in place (both 0 for a vertex without out-edges).
__global__ void k_degrees(uint32_t *end_deg, const uint32_t *first, uint32_t n, uint32_t *iota)
{
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        end_deg[v] -= first[v];
        iota[v] = v;
    }
}

// Everything of internal vertex i = rank by degree, order[i] its canonical index,
// off the exclusive sums of deg.  shift[index]: internal minus canonical place of
// a row.  run: {0: runs of equal degree (also beyond max_runs), largest degree},
// then {id, first column, degree} of each run's first vertex, unordered.
__global__ void k_relabel(const uint32_t *order, const uint32_t *deg, const uint32_t *off, const uint32_t *first,
                          const uint32_t *names, bool compact, uint32_t n, uint32_t *idx2int, uint32_t *int2name,
                          uint2 *adj, uint32_t *shift, uint32_t max_runs, uint4 *run)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t idx = order[i], d = deg[i], o = off[i];
        idx2int[idx] = i;
        int2name[i] = compact ? idx : names[idx];
        adj[i] = make_uint2(o, d);
        shift[idx] = o - first[idx];
        if (i == 0) run[0].y = d;
        if (i != 0 && deg[i - 1] == d) continue;
        const uint32_t p = atomicAdd(&run[0].x, 1u);
        if (p < max_runs) run[1 + p] = make_uint4(i, o, d, 0u);
    }
}

__global__ void k_iota(uint32_t *x, uint32_t n)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        x[i] = i;
}

// Canonical edges into internal rows.
__global__ void k_fill_col(const unsigned long long *keys, uint64_t m, int bits, const uint32_t *shift,
                           const uint32_t *idx2int, uint32_t *col)
{
    const uint32_t mask = (uint32_t)((1ull << bits) - 1);
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
        const unsigned long long k = keys[e];
        col[shift[k >> bits] + (uint32_t)e] = idx2int[(uint32_t)k & mask];
    }
}

// Canonical export: kExportTile consecutive columns per warp.  A row per warp left
// it to one warp to copy a hub and 27 lanes of most others idle (16 M entries, 3 M
// rows: 695 -> 124 us).  Rows lie in the order of their columns; those of a tile are found
// from its two ends, by division where all have one degree.
constexpr uint32_t kExportTile = 256;

__device__ __forceinline__ uint32_t row_with(const uint2 *adj, uint32_t lo, uint32_t hi, uint32_t e)
{
    while (hi - lo > 1) {  // adj[lo].x <= e < adj[hi].x (hi may be n)
        const uint32_t mid = lo + (hi - lo) / 2;
        if (adj[mid].x <= e) lo = mid;
        else hi = mid;
    }
    return lo;
}

__global__ void k_export(const uint2 *adj, const uint32_t *col, const uint32_t *int2idx, const uint32_t *canon_off,
                         uint32_t n_rows, uint64_t m, uint32_t *out_col)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t t = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; t * kExportTile < m; t += warps) {
        const uint64_t e0 = t * kExportTile, e1 = e0 + kExportTile < m ? e0 + kExportTile : m;
        uint32_t row = 0;
        if (lane < 2) row = row_with(adj, 0, n_rows, (uint32_t)(lane ? e1 - 1 : e0));
        const uint32_t lo = __shfl_sync(0xffffffffu, row, 0), hi = __shfl_sync(0xffffffffu, row, 1);
        const uint2 first = adj[lo];
        const bool even = first.y == adj[hi].y;
        for (uint64_t e = e0 + lane; e < e1; e += 32) {
            const uint32_t r = even ? lo + ((uint32_t)e - first.x) / first.y : row_with(adj, lo, hi + 1, (uint32_t)e);
            const uint32_t start = even ? first.x + (r - lo) * first.y : adj[r].x;
            out_col[canon_off[int2idx[r]] + ((uint32_t)e - start)] = int2idx[col[e]];
        }
    }
}

// Degrees by canonical index, [n + 1] with a 0 at the end.
__global__ void k_deg_by_index(const uint2 *adj, const uint32_t *idx2int, uint32_t n, uint32_t *deg)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x)
        deg[i] = i < n ? adj[idx2int[i]].y : 0u;
}

// Row offsets as the caller takes them.
__global__ void k_widen(const uint32_t *x, uint64_t n, unsigned long long *y)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        y[i] = x[i];
}

__global__ void k_rmat(uint32_t scale, uint64_t m, uint32_t ta, uint32_t tab, uint32_t tabc,
                       uint32_t k0, uint32_t k1, uint32_t *src, uint32_t *dst)
{
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m;
         e += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t u = 0, v = 0;
        uint4 w = make_uint4(0, 0, 0, 0);
        for (uint32_t l = 0; l < scale; ++l) {
            if ((l & 3u) == 0)
                w = philox(make_uint4((uint32_t)e, (uint32_t)(e >> 32), l >> 2, PTW_TAG_RMAT), k0, k1);
            const uint32_t x = (l & 3u) == 0 ? w.x : (l & 3u) == 1 ? w.y : (l & 3u) == 2 ? w.z : w.w;
            const uint32_t rb = x >= tab;
            const uint32_t cb = (x >= ta && x < tab) || x >= tabc;
            u = (u << 1) | rb;
            v = (v << 1) | cb;
        }
        src[e] = u;
        dst[e] = v;
    }
}

// Chung-Lu: vertex i has weight (i + 1)^(-expo), expo = 1 / (gamma - 1);
// both endpoints of an edge are drawn proportionally to weight by inverse
// CDF (binary search over the inclusive prefix sums).
__global__ void k_cl_weights(uint32_t n, double expo, double *w)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        w[i] = pow((double)i + 1.0, -expo);
}

__device__ __forceinline__ uint32_t cdf_pick(const double *cdf, uint32_t n, double x)
{
    uint32_t lo = 0, hi = n - 1;  // first i with cdf[i] > x
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (cdf[mid] > x) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

__global__ void k_cl_edges(uint64_t m, const double *cdf, uint32_t n, uint32_t k0, uint32_t k1, uint32_t *src,
                           uint32_t *dst)
{
    const double total = cdf[n - 1];
    const double inv53 = 1.0 / 9007199254740992.0;  // 2^-53
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m;
         e += (uint64_t)gridDim.x * blockDim.x) {
        const uint4 r = philox(make_uint4((uint32_t)e, (uint32_t)(e >> 32), 0u, PTW_TAG_CHUNGLU), k0, k1);
        const double u1 = (double)(((uint64_t)(r.x >> 5) << 26) | (r.y >> 6)) * inv53;
        const double u2 = (double)(((uint64_t)(r.z >> 5) << 26) | (r.w >> 6)) * inv53;
        src[e] = cdf_pick(cdf, n, u1 * total);
        dst[e] = cdf_pick(cdf, n, u2 * total);
    }
}

// CSR -> (src, dst) names, one thread per entry.  The row of entry e is the
// largest r with row_ptr[r] <= e (row_ptr is validated non-decreasing with
// row_ptr[0] = 0 and row_ptr[n] = m on the host, so the search invariant
// row_ptr[lo] <= e < row_ptr[hi] holds from lo = 0, hi = n).  A column index
// >= n raises *bad and writes name 0 so the arrays stay defined.
__global__ void k_csr_to_edges(const uint64_t *row_ptr, const uint32_t *col, const uint32_t *names,
                               uint32_t n, uint64_t m, uint32_t *src, uint32_t *dst, unsigned *bad)
{
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m;
         e += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = n;
        while (hi - lo > 1) {
            const uint32_t mid = lo + (hi - lo) / 2;
            if (row_ptr[mid] <= e) lo = mid;
            else hi = mid;
        }
        const uint32_t c = col[e];
        if (c >= n) {
            atomicOr(bad, 1u);
            src[e] = dst[e] = 0;
            continue;
        }
        src[e] = names ? names[lo] : lo;
        dst[e] = names ? names[c] : c;
    }
}

// Raises *bad when two neighbours of a sorted array are equal.
__global__ void k_adjacent_equal(const uint32_t *x, uint32_t n, unsigned *bad)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i + 1 < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        if (x[i] == x[i + 1]) atomicOr(bad, 2u);
}

// Frees every pointer on scope exit (stream-ordered).
struct AsyncBufs {
    cudaStream_t st;
    std::vector<void *> ptrs;
    explicit AsyncBufs(cudaStream_t s) : st(s) {}
    template <typename T> cudaError_t alloc(T **p, uint64_t count)
    {
        void *q = nullptr;
        cudaError_t e = pooled_alloc_async(&q, std::max<uint64_t>(count, 1) * sizeof(T), st);
        if (e == cudaSuccess) ptrs.push_back(q);
        *p = (T *)q;
        return e;
    }
    void release(void *p)
    {
        for (auto &q : ptrs)
            if (q == p) {
                cudaFreeAsync(q, st);
                q = nullptr;
            }
    }
    ~AsyncBufs()
    {
        for (void *q : ptrs)
            if (q) cudaFreeAsync(q, st);
    }
};

template <typename F> cudaError_t cub_call(F f, cudaStream_t st)
{
    size_t bytes = 0;
    cudaError_t e = f(nullptr, bytes);
    if (e != cudaSuccess) return e;
    void *tmp = nullptr;
    e = pooled_alloc_async(&tmp, std::max<size_t>(bytes, 16), st);
    if (e != cudaSuccess) return e;
    e = f(tmp, bytes);
    cudaFreeAsync(tmp, st);
    return e;
}

int bits_for(uint64_t bound)
{
    int b = 1;
    while (b < 32 && (1ull << b) < bound) ++b;
    return b;
}

}  // namespace

int graph_init_handle(ptw_graph *g)
{
    PTW_CUDA(cudaGetDevice(&g->device));
    PTW_CUDA(cudaDeviceGetAttribute(&g->num_sms, cudaDevAttrMultiProcessorCount, g->device));
    PTW_CUDA(cudaStreamCreateWithFlags(&g->own_stream, cudaStreamNonBlocking));
    g->stream = g->own_stream;
    for (auto &e : g->ev) PTW_CUDA(cudaEventCreate(&e));
    g->tune = default_tune();
    return PTW_OK;
}

void graph_release(ptw_graph *g)
{
    if (!g) return;
    if (g->stream) cudaStreamSynchronize(g->stream);
    for (void *p : g->arrays) cudaFree(p);  // dg.adj .. dg.names, dg.rows, sc.counts, sc.ctrl
    cudaFree(g->dg.col_named);
    cudaFree(g->dg.col_ext);
    cudaFree(g->dg.vtx_ext);
    cudaFree(g->dg.edge_filter);
    cudaFree(g->sc.sources);
    cudaFree(g->sc.by_name);
    cudaFree(g->sc.out_stage);
    for (auto &e : g->ev)
        if (e) cudaEventDestroy(e);
    if (g->copy_stream) cudaStreamSynchronize(g->copy_stream);
    for (ptw::AsyncSlot &a : g->async) {
        cudaFree(a.by_name);
        cudaFreeHost(a.h_moves);
        for (cudaEvent_t e : {a.ev_start, a.ev_walk, a.ev_copy})
            if (e) cudaEventDestroy(e);
    }
    if (g->copy_stream) cudaStreamDestroy(g->copy_stream);
    if (g->own_stream) cudaStreamSynchronize(g->own_stream);
    if (g->own_stream) cudaStreamDestroy(g->own_stream);
    delete[] g->h_names;
    delete[] g->h_idx2int;
}

int rmat_generate_device(uint32_t scale, uint64_t m, uint32_t ta, uint32_t tab, uint32_t tabc,
                         uint64_t seed, uint32_t *d_src, uint32_t *d_dst, cudaStream_t st)
{
    k_rmat<<<grid_for(m), kThreads, 0, st>>>(scale, m, ta, tab, tabc, (uint32_t)seed,
                                             (uint32_t)(seed >> 32), d_src, d_dst);
    PTW_CUDA(cudaGetLastError());
    return PTW_OK;
}

int chung_lu_generate_device(uint32_t n, double gamma, uint64_t m, uint64_t seed, uint32_t *d_src,
                             uint32_t *d_dst, cudaStream_t st)
{
    AsyncBufs tmp(st);
    double *w = nullptr, *cdf = nullptr;
    PTW_CUDA(tmp.alloc(&w, n));
    PTW_CUDA(tmp.alloc(&cdf, n));
    k_cl_weights<<<grid_for(n), kThreads, 0, st>>>(n, 1.0 / (gamma - 1.0), w);
    PTW_CUDA(cub_call([&](void *t, size_t &b) {
        return cub::DeviceScan::InclusiveSum(t, b, w, cdf, (int64_t)n, st);
    }, st));
    k_cl_edges<<<grid_for(m), kThreads, 0, st>>>(m, cdf, n, (uint32_t)seed, (uint32_t)(seed >> 32), d_src, d_dst);
    PTW_CUDA(cudaGetLastError());
    PTW_CUDA(cudaStreamSynchronize(st));
    return PTW_OK;
}

int csr_to_device_edges(const uint64_t *h_row_ptr, const uint32_t *h_col, const uint32_t *h_names,
                        uint32_t n, uint32_t **d_src, uint32_t **d_dst, cudaStream_t st)
{
    *d_src = *d_dst = nullptr;
    const uint64_t m = h_row_ptr[n];
    AsyncBufs tmp(st);
    uint64_t *row = nullptr;
    uint32_t *col = nullptr, *names = nullptr, *src = nullptr, *dst = nullptr;
    unsigned *bad = nullptr;
    PTW_CUDA(tmp.alloc(&row, (uint64_t)n + 1));
    PTW_CUDA(tmp.alloc(&col, m));
    PTW_CUDA(tmp.alloc(&bad, 1));
    PTW_CUDA(cudaMemsetAsync(bad, 0, sizeof(unsigned), st));
    PTW_CUDA(cudaMemcpyAsync(row, h_row_ptr, ((uint64_t)n + 1) * 8, cudaMemcpyHostToDevice, st));
    PTW_CUDA(cudaMemcpyAsync(col, h_col, m * 4, cudaMemcpyHostToDevice, st));
    if (h_names) {
        uint32_t *sorted = nullptr;
        PTW_CUDA(tmp.alloc(&names, n));
        PTW_CUDA(tmp.alloc(&sorted, n));
        PTW_CUDA(cudaMemcpyAsync(names, h_names, (uint64_t)n * 4, cudaMemcpyHostToDevice, st));
        PTW_CUDA(cub_call([&](void *t, size_t &b) {
            return cub::DeviceRadixSort::SortKeys(t, b, names, sorted, (int64_t)n, 0, 32, st);
        }, st));
        k_adjacent_equal<<<grid_for(n), kThreads, 0, st>>>(sorted, n, bad);
        tmp.release(sorted);
    }
    // The edge arrays are handed to the caller, so they are not in tmp.
    PTW_CUDA(pooled_alloc_async((void **)&src, std::max<uint64_t>(m, 1) * 4, st));
    cudaError_t e = pooled_alloc_async((void **)&dst, std::max<uint64_t>(m, 1) * 4, st);
    if (e != cudaSuccess) {
        cudaFreeAsync(src, st);
        return cuda_fail(e, "CSR edge buffers");
    }
    k_csr_to_edges<<<grid_for(m), kThreads, 0, st>>>(row, col, names, n, m, src, dst, bad);
    unsigned h_bad = 0;
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h_bad, bad, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess || h_bad) {
        cudaFreeAsync(src, st);
        cudaFreeAsync(dst, st);
        if (e != cudaSuccess) return cuda_fail(e, "CSR expansion");
        return fail(PTW_EINVAL, (h_bad & 1) ? "CSR column index >= n" : "CSR vertex names are not distinct");
    }
    *d_src = src;
    *d_dst = dst;
    return PTW_OK;
}

namespace {

// Host image of the row table from the runs of equal degree (k_relabel); empty
// when there are more than kMaxRowRuns of them.
std::vector<uint32_t> row_table_image(const std::vector<uint4> &found, uint32_t n)
{
    const uint32_t runs = found[0].x;
    if (runs > kMaxRowRuns) return {};
    std::vector<uint4> run(found.begin() + 1, found.begin() + 1 + runs);
    std::sort(run.begin(), run.end(), [](const uint4 &x, const uint4 &y) { return x.x < y.x; });
    std::vector<uint32_t> img(row_words(runs, n), 0u);
    for (uint32_t k = 0; k < runs; ++k) {
        img[k] = run[k].x;
        img[row_pairs_at(runs) + 2 * k] = run[k].y - run[k].x * run[k].z;
        img[row_pairs_at(runs) + 2 * k + 1] = run[k].z;
    }
    img[runs] = img[runs + 1] = ~0u;
    img[row_pairs_at(runs) + 2 * runs] = img[row_pairs_at(runs) + 2 * runs - 2];
    img[row_pairs_at(runs) + 2 * runs + 1] = img[row_pairs_at(runs) + 2 * runs - 1];
    uint16_t *bucket = reinterpret_cast<uint16_t *>(img.data() + row_buckets_at(runs));
    uint32_t next = 0;  // first bucket whose run is not set yet
    for (uint32_t k = 0; k < runs; ++k) {
        // run k holds the ids [run[k].x, end); it is the run of every bucket whose first id is among them
        const uint32_t end = k + 1 < runs ? run[k + 1].x : n;
        const uint32_t last = row_bucket(end - 1);
        for (; next <= last; ++next) bucket[next] = (uint16_t)k;
    }
    return img;
}

// The arrays of a graph: one allocation up to 1 MB per vertex array, from there on one
// each, in the order in which walks read them.  The line lies about where the walks'
// times cross, for a reason not known: DeepWalk, one walker per vertex, 80 positions, apart
// against in one, R-MAT scale 17 63 against 65 us, 18 (0.7 MB) 142 / 138, 19 (1.3 MB)
// 266 / 264, 20 565 / 576, 22 3,723 / 3,740; count walks the same up to 18, 19 74 / 76,
// 22 331 / 342.  One allocation spares a build of scale 10 20 us of 400 and its close
// 17 of 97, at scale 18 140 of 1,420 and 110 of 195.
int alloc_arrays(ptw_graph *g, uint32_t n, uint64_t m, uint32_t max_runs)
{
    DeviceGraph &dg = g->dg;
    struct Want {
        void **p;
        uint64_t bytes;
    };
    const Want want[] = {{(void **)&dg.adj, n * 8ull},       {(void **)&dg.col, m * 4},
                         {(void **)&dg.int2name, n * 4ull},  {(void **)&dg.idx2int, n * 4ull},
                         {(void **)&dg.int2idx, n * 4ull},   {(void **)&dg.names, n * 4ull},
                         {(void **)&g->sc.counts, n * 4ull}, {(void **)&g->sc.ctrl, 16 * sizeof(unsigned long long)},
                         {(void **)&g->row_space, row_words(max_runs, n) * 4ull}};
    const bool apart = n * 4ull >= (1ull << 20);
    uint64_t bytes = 0;
    for (const Want &w : want) bytes += (w.bytes + 255) & ~255ull;
    char *block = nullptr;
    g->arrays.reserve(sizeof(want) / sizeof(want[0]));
    if (!apart) {
        PTW_CUDA(device_malloc(&block, bytes));
        g->arrays.push_back(block);
    }
    for (const Want &w : want) {
        if (apart) {
            PTW_CUDA(device_malloc(&block, w.bytes));
            g->arrays.push_back(block);
        }
        *w.p = block;
        block += (w.bytes + 255) & ~255ull;
    }
    return PTW_OK;
}

}  // namespace

// Device time of 8 M edges, both directions, 3 M names below 12 M: names and keys
// from a table over the name range 0.26 ms (sorting all endpoints for the distinct
// ones and searching those for every endpoint: 1.6 ms), the sort of the keys 1.0
// ms (six passes at 1.7 TB/s of reads and writes), rows and columns 0.3 ms.
// R-MAT scale 20 7.8 -> 3.6 ms, 22 29 -> 16, 24 119 -> 69; 1,087 edges 449 -> 300 us.
int build_graph_from_device_edges(ptw_graph *g, uint32_t *d_src, uint32_t *d_dst, uint64_t m, bool as_undirected,
                                  bool clean, bool compact_names)
{
    cudaStream_t st = g->stream;
    AsyncBufs tmp(st);
    tmp.ptrs = {d_src, d_dst};
    if (m == 0) return fail(PTW_EINVAL, "edge list is empty");
    const unsigned wide = (unsigned)g->num_sms * 8;

    // Name range.
    unsigned *d_max = nullptr;
    unsigned long long *d_cnt = nullptr;  // {edges kept, vertices, entries after unique}
    PTW_CUDA(tmp.alloc(&d_cnt, 4));
    PTW_CUDA(cudaMemsetAsync(d_cnt, 0, 4 * sizeof(unsigned long long), st));
    d_max = reinterpret_cast<unsigned *>(d_cnt + 3);
    k_max2<<<std::min(grid_for(m / 4), wide), kThreads, 0, st>>>(d_src, d_dst, m, d_max);
    unsigned h_max = 0;
    PTW_CUDA(cudaMemcpyAsync(&h_max, d_max, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    PTW_CUDA(cudaStreamSynchronize(st));
    const uint64_t id_bound = (uint64_t)h_max + 1;
    const uint64_t cap = as_undirected ? 2 * m : m;

    // Names, and the index of each: over the name range while that is not far
    // above the number of entries (4 bytes of it against the two sorts' 32 per
    // entry), else by sorting the endpoints (edges of a clean graph come from the
    // generators, whose vertices are their range).
    const bool table = clean || id_bound <= 4 * cap;
    uint32_t *index_of = nullptr, *names = nullptr;
    unsigned long long h_cnt[2] = {m, 0};
    if (table) {
        PTW_CUDA(tmp.alloc(&index_of, id_bound + 1));
        PTW_CUDA(tmp.alloc(&names, std::min(id_bound, 2 * m)));
        PTW_CUDA(cudaMemsetAsync(index_of, 0, (id_bound + 1) * 4, st));
        k_mark_names<<<std::min(grid_for(m), wide), kThreads, 0, st>>>(d_src, d_dst, m, clean, index_of, d_cnt);
        PTW_CUDA(cub_call([&](void *t, size_t &b) {
            return cub::DeviceScan::ExclusiveSum(t, b, index_of, index_of, (int64_t)id_bound + 1, st);
        }, st));
        k_collect_names<<<grid_for(id_bound), kThreads, 0, st>>>(index_of, id_bound, names, d_cnt + 1);
        PTW_CUDA(cudaGetLastError());
        PTW_CUDA(cudaMemcpyAsync(h_cnt, d_cnt, sizeof(h_cnt), cudaMemcpyDeviceToHost, st));
    } else {
        uint32_t *ends = nullptr;
        PTW_CUDA(tmp.alloc(&ends, 2 * m));
        PTW_CUDA(tmp.alloc(&names, 2 * m));
        PTW_CUDA(cudaMemcpyAsync(ends, d_src, m * 4, cudaMemcpyDeviceToDevice, st));
        PTW_CUDA(cudaMemcpyAsync(ends + m, d_dst, m * 4, cudaMemcpyDeviceToDevice, st));
        cub::DoubleBuffer<uint32_t> db(ends, names);
        PTW_CUDA(cub_call([&](void *t, size_t &b) {
            return cub::DeviceRadixSort::SortKeys(t, b, db, (int64_t)(2 * m), 0, bits_for(id_bound), st);
        }, st));
        if (db.Current() == names) std::swap(ends, names);
        PTW_CUDA(cub_call([&](void *t, size_t &b) {
            return cub::DeviceSelect::Unique(t, b, ends, names, d_cnt + 1, (int64_t)(2 * m), st);
        }, st));
        tmp.release(ends);
        PTW_CUDA(cudaMemcpyAsync(h_cnt + 1, d_cnt + 1, sizeof(h_cnt[1]), cudaMemcpyDeviceToHost, st));
    }
    PTW_CUDA(cudaStreamSynchronize(st));
    uint64_t mm = as_undirected ? 2 * h_cnt[0] : h_cnt[0];
    const uint32_t n = (uint32_t)h_cnt[1];
    if (mm == 0) return fail(PTW_EINVAL, "graph has no edges after clean-up");
    if (mm >= (1ull << 32)) return fail(PTW_EINVAL, "graphs with 2^32 or more CSR entries are not supported");

    // Packed keys, sorted.
    const int bits = bits_for(n);
    unsigned long long *keys = nullptr, *keys_alt = nullptr;
    PTW_CUDA(tmp.alloc(&keys, cap));
    k_make_keys<<<grid_for(m), kThreads, 0, st>>>(d_src, d_dst, m, bits, as_undirected, clean, index_of, names, n, keys);
    PTW_CUDA(cudaGetLastError());
    tmp.release(d_src);
    tmp.release(d_dst);
    if (index_of) tmp.release(index_of);
    PTW_CUDA(tmp.alloc(&keys_alt, cap));
    {
        cub::DoubleBuffer<unsigned long long> db(keys, keys_alt);
        PTW_CUDA(cub_call([&](void *t, size_t &b) {
            return cub::DeviceRadixSort::SortKeys(t, b, db, (int64_t)cap, 0, 2 * bits, st);
        }, st));
        if (db.Current() != keys) std::swap(keys, keys_alt);
    }
    if (clean) {
        PTW_CUDA(cub_call([&](void *t, size_t &b) {
            return cub::DeviceSelect::Unique(t, b, keys, keys_alt, d_cnt + 2, (int64_t)mm, st);
        }, st));
        PTW_CUDA(cudaMemcpyAsync(h_cnt, d_cnt + 2, sizeof(h_cnt[0]), cudaMemcpyDeviceToHost, st));
        PTW_CUDA(cudaStreamSynchronize(st));
        std::swap(keys, keys_alt);
        mm = h_cnt[0];
    }
    tmp.release(keys_alt);

    // The distinct degrees d of a graph sum up to mm at most.
    const uint32_t max_runs =
        (uint32_t)std::min<uint64_t>(std::min<uint64_t>(n, kMaxRowRuns), (uint64_t)std::sqrt(2.0 * (double)mm) + 2);
    DeviceGraph &dg = g->dg;
    dg.n = n;
    dg.m = mm;
    dg.id_bound = compact_names ? n : (uint32_t)id_bound;
    if (const int rc = alloc_arrays(g, n, mm, max_runs)) return rc;

    // Degrees; internal order: stable sort of canonical indices by descending
    // degree; rows in that order.
    uint32_t *first = nullptr, *deg = nullptr, *deg_sorted = nullptr, *iota = nullptr;
    uint4 *d_run = nullptr;
    PTW_CUDA(tmp.alloc(&first, 2ull * n));
    deg = first + n;
    PTW_CUDA(tmp.alloc(&deg_sorted, n));
    PTW_CUDA(tmp.alloc(&iota, n));
    PTW_CUDA(tmp.alloc(&d_run, 1ull + max_runs));
    PTW_CUDA(cudaMemsetAsync(first, 0, n * 8ull, st));
    PTW_CUDA(cudaMemsetAsync(d_run, 0, sizeof(uint4), st));
    PTW_CUDA(cudaMemsetAsync(g->sc.ctrl, 0, 16 * sizeof(unsigned long long), st));  // [7]: index checks
    k_row_bounds<<<grid_for(mm), kThreads, 0, st>>>(keys, mm, bits, first, deg);
    k_degrees<<<grid_for(n), kThreads, 0, st>>>(deg, first, n, iota);
    PTW_CUDA(cub_call([&](void *t, size_t &b) {
        return cub::DeviceRadixSort::SortPairsDescending(t, b, deg, deg_sorted, iota, dg.int2idx, (int64_t)n, 0,
                                                         bits_for(mm + 1), st);
    }, st));
    uint32_t *off = iota, *shift = deg;  // reuse
    PTW_CUDA(cub_call([&](void *t, size_t &b) {
        return cub::DeviceScan::ExclusiveSum(t, b, deg_sorted, off, (int64_t)n, st);
    }, st));
    k_relabel<<<grid_for(n), kThreads, 0, st>>>(dg.int2idx, deg_sorted, off, first, names, compact_names, n, dg.idx2int,
                                                dg.int2name, dg.adj, shift, max_runs, d_run);
    if (compact_names) k_iota<<<grid_for(n), kThreads, 0, st>>>(dg.names, n);
    else PTW_CUDA(cudaMemcpyAsync(dg.names, names, n * 4ull, cudaMemcpyDeviceToDevice, st));
    PTW_CUDA(cudaGetLastError());
    std::vector<uint4> h_run(1 + max_runs);
    PTW_CUDA(cudaMemcpyAsync(h_run.data(), d_run, h_run.size() * sizeof(uint4), cudaMemcpyDeviceToHost, st));
    PTW_CUDA(cudaStreamSynchronize(st));

    // The host makes the row table while the columns are filled.
    k_fill_col<<<grid_for(mm), kThreads, 0, st>>>(keys, mm, bits, shift, dg.idx2int, dg.col);
    PTW_CUDA(cudaGetLastError());
    const std::vector<uint32_t> img = row_table_image(h_run, n);
    if (!img.empty()) {
        PTW_CUDA(cudaMemcpyAsync(g->row_space, img.data(), img.size() * 4, cudaMemcpyHostToDevice, st));
        dg.rows = g->row_space;
        dg.row_runs = h_run[0].x;
    }
    // Host copy of the ascending names for source lookups.
    g->h_names = new (std::nothrow) uint32_t[n];
    if (!g->h_names) return fail(PTW_ENOMEM, "host allocation of the name table failed");
    PTW_CUDA(cudaMemcpyAsync(g->h_names, dg.names, (uint64_t)n * 4, cudaMemcpyDeviceToHost, st));
    g->h_idx2int = new (std::nothrow) uint32_t[n];
    if (!g->h_idx2int) return fail(PTW_ENOMEM, "host allocation of the index table failed");
    PTW_CUDA(cudaMemcpyAsync(g->h_idx2int, dg.idx2int, (uint64_t)n * 4, cudaMemcpyDeviceToHost, st));
    PTW_CUDA(cudaStreamSynchronize(st));
    dg.max_degree = h_run[0].y;
    // symmetrised, self-loops dropped and duplicates removed: simple and
    // symmetric by construction (node2vec then skips its check)
    dg.simple_symmetric = as_undirected && clean ? 1 : -1;
    g->device_bytes = (uint64_t)n * (8 + 4 * 4 + 4) + mm * 4 + 64 + img.size() * 4;
    return PTW_OK;
}

}  // namespace ptw

using namespace ptw;

extern "C" int ptw_graph_get_info(const ptw_graph *g, ptw_graph_info *info)
try {
    if (!g || !info) return fail(PTW_EINVAL, "null argument");
    info->n_vertices = g->dg.n;
    info->id_bound = g->dg.id_bound;
    info->n_edges = g->dg.m;
    info->max_degree = g->dg.max_degree;
    info->reserved = 0;
    info->device_bytes = g->device_bytes;
    return PTW_OK;
} catch (...) {
    return host_exception();
}

extern "C" int ptw_graph_export_csr(const ptw_graph *g, uint32_t *h_names, uint64_t *h_row_ptr,
                                    uint32_t *h_col)
try {
    if (!g) return fail(PTW_EINVAL, "null graph");
    const DeviceGraph &dg = g->dg;
    cudaStream_t st = g->stream;
    PTW_CUDA(cudaSetDevice(g->device));
    PoolKeep pool(st);
    AsyncBufs tmp(st);
    // row offsets as the caller takes them, degrees, offsets, columns: one allocation
    const uint64_t n1 = dg.n + 1ull;
    unsigned long long *rows = nullptr;
    PTW_CUDA(tmp.alloc(&rows, (h_row_ptr ? n1 : 0) + n1 + (h_col ? (dg.m + 1) / 2 : 0)));
    uint32_t *const deg = reinterpret_cast<uint32_t *>(rows + (h_row_ptr ? n1 : 0)), *const off = deg + n1, *const c = off + n1;
    k_deg_by_index<<<grid_for(n1), kThreads, 0, st>>>(dg.adj, dg.idx2int, dg.n, deg);
    PTW_CUDA(cub_call([&](void *t, size_t &b) {
        return cub::DeviceScan::ExclusiveSum(t, b, deg, off, (int64_t)n1, st);
    }, st));
    if (h_col) {
        const uint64_t tiles = (dg.m + kExportTile - 1) / kExportTile;
        k_export<<<grid_for(tiles * 32), kThreads, 0, st>>>(dg.adj, dg.col, dg.int2idx, off, dg.n, dg.m, c);
        PTW_CUDA(cudaGetLastError());
    }
    if (h_row_ptr) {
        k_widen<<<grid_for(n1), kThreads, 0, st>>>(off, n1, rows);
        PTW_CUDA(cudaGetLastError());
        PTW_CUDA(cudaMemcpyAsync(h_row_ptr, rows, n1 * 8, cudaMemcpyDeviceToHost, st));
    }
    if (h_col) PTW_CUDA(cudaMemcpyAsync(h_col, c, dg.m * 4, cudaMemcpyDeviceToHost, st));
    if (h_names) std::memcpy(h_names, g->h_names, (uint64_t)dg.n * 4);
    PTW_CUDA(cudaStreamSynchronize(st));
    return PTW_OK;
} catch (...) {
    return host_exception();
}

extern "C" int ptw_graph_export_edges(const ptw_graph *g, uint32_t *h_src, uint32_t *h_dst)
try {
    if (!g || !h_src || !h_dst) return fail(PTW_EINVAL, "null argument");
    const DeviceGraph &dg = g->dg;
    std::vector<uint64_t> rp(dg.n + 1);
    int rc = ptw_graph_export_csr(g, nullptr, rp.data(), h_dst);
    if (rc) return rc;
    for (uint32_t i = 0; i < dg.n; ++i)
        for (uint64_t e = rp[i]; e < rp[i + 1]; ++e) h_src[e] = g->h_names[i];
    for (uint64_t e = 0; e < dg.m; ++e) h_dst[e] = g->h_names[h_dst[e]];
    return PTW_OK;
} catch (...) {
    return host_exception();
}

extern "C" int ptw_graph_sync(ptw_graph *g)
try {
    if (!g) return fail(PTW_EINVAL, "null graph");
    PTW_CUDA(cudaStreamSynchronize(g->stream));
    return PTW_OK;
} catch (...) {
    return host_exception();
}

extern "C" int ptw_graph_set_stream(ptw_graph *g, void *cuda_stream)
try {
    if (!g) return fail(PTW_EINVAL, "null graph");
    cudaStream_t s = cuda_stream ? (cudaStream_t)cuda_stream : g->own_stream;
    if (s != g->stream) {
        // Work already queued on the old stream completes before the switch.
        PTW_CUDA(cudaStreamSynchronize(g->stream));
    }
    g->stream = s;
    return PTW_OK;
} catch (...) {
    return host_exception();
}
