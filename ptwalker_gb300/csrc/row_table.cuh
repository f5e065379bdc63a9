// Row records without a memory access.
//
// Internal ids are ranks by descending degree and the rows are laid out in
// that order, so the vertices of one degree are a run of consecutive ids whose
// rows follow one another: first column = base + id * degree (mod 2^32; CSRs
// have fewer than 2^32 entries).  A graph has few distinct degrees (R-MAT
// scale 22: 1,447 for 2.4 M vertices; at most sqrt(2m) of any graph with m
// entries), so the runs fit in shared memory, and a kernel looks a vertex's
// row up there instead of loading adj[v] from L2 behind every gather.
//
// Device image (32-bit words): first[runs + 2], ascending, ~0 from first[runs]
// on; {base, degree} per run and once more for the last; one 16-bit entry per
// bucket with the run of the bucket's first id.  Buckets cut the ids as a
// 10-bit mantissa cuts a float: single ids below 2,048, then 1,024 buckets
// per octave.  Degrees come in clusters (R-MAT), so with 6 bits the slowest
// lane of a warp stepped over 5.3 runs on average at scale 20 (29 at the 99th
// percentile); with 10 bits it is 0.5 (3), for 2 KB of table per octave.
#pragma once

#include <stdint.h>

namespace ptw {

constexpr uint32_t kMaxRowRuns = 8192;

constexpr uint32_t kRowBits = 10;

__host__ __device__ __forceinline__ int max_int(int x, int y) { return x > y ? x : y; }

__host__ __device__ __forceinline__ uint32_t row_bucket(uint32_t id)
{
#ifdef __CUDA_ARCH__
    const int z = __clz(id);
#else
    const int z = id ? __builtin_clz(id) : 32;
#endif
    const uint32_t s = (uint32_t)max_int(31 - (int)kRowBits - z, 0);  // low bits cut off
    return (s << kRowBits) + (id >> s);
}

// First word of the {base, degree} pairs (8-byte aligned) and of the buckets.
__host__ __device__ __forceinline__ uint32_t row_pairs_at(uint32_t runs) { return (runs + 3) & ~1u; }
__host__ __device__ __forceinline__ uint32_t row_buckets_at(uint32_t runs) { return row_pairs_at(runs) + 2 * (runs + 1); }
// Words of the whole image, a multiple of 4.
__host__ __device__ __forceinline__ uint32_t row_words(uint32_t runs, uint32_t n)
{
    return (row_buckets_at(runs) + (row_bucket(n - 1) + 2) / 2 + 3) & ~3u;
}

#ifdef __CUDACC__
// Copies the image to shared memory (16-byte aligned); the caller synchronises.
__device__ __forceinline__ void row_table_load(uint32_t *s_rows, const uint32_t *rows, uint32_t words)
{
    for (uint32_t i = threadIdx.x; i < words / 4; i += blockDim.x)
        reinterpret_cast<uint4 *>(s_rows)[i] = reinterpret_cast<const uint4 *>(rows)[i];
}

// {first column, degree} of vertex v < n.
__device__ __forceinline__ uint2 row_of(const uint32_t *s_rows, uint32_t runs, uint32_t v)
{
    const uint2 *pairs = reinterpret_cast<const uint2 *>(s_rows + row_pairs_at(runs));
    uint32_t k = reinterpret_cast<const uint16_t *>(s_rows + row_buckets_at(runs))[row_bucket(v)];
    // the bucket's first run or the next one, nearly always: the loads of
    // both are issued together
    const uint32_t f1 = s_rows[k + 1], f2 = s_rows[k + 2];
    const uint2 p0 = pairs[k], p1 = pairs[k + 1];
    uint2 bd = v < f1 ? p0 : p1;
    if (v >= f2) {
        for (k += 2; s_rows[k + 1] <= v;) ++k;  // ends at the last run: first[runs] = ~0
        bd = pairs[k];
    }
    return make_uint2(bd.x + v * bd.y, bd.y);
}
#endif

}  // namespace ptw
