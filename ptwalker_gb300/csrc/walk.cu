// Walker-update kernels for sm_103a.
//
// K1/K2 k_walk: persistent walker pool.  Replaces the reference's per-thread
// walker containers, partition sweeps and migrations
// (src/core/solver.hpp:194-498, :850-1028) and the direct sampler
// (src/core/sampler.hpp:214-217).  Each lane holds ILP walkers.  A lane whose
// walker ended is refilled from a warp-private range of walker ids: the warp
// ballots the empty lanes, ranks them with a popcount prefix and takes ids
// from its range, drawing a new range of `chunk` ids from one global cursor
// when it runs dry.  Every draw is a pure function of (seed, walker id, step),
// so scheduling never changes a result.
//
// Per move (count apps, pagerank.cpp:86-89 / ppr.cpp:114-117):
//   {off, deg} = adj[v]                      one 8-byte random load
//   u = Philox4x32-10(key=seed, ctr=(wid_lo, wid_hi, step, "WALK"))
//   v = col[off + mulhi(u.x, deg)]           one 4-byte random load
//   counts[v] += 1                           one fire-and-forget reduction
//   stop iff u.y < floor(sp * 2^32)
// With the extended column copy (EXT) the column entry also carries the
// neighbour's {off, deg} (and name), so a move is one dependent 16-byte
// gather: the walker keeps {off, deg} of its vertex in registers and loads a
// row record only at its start vertex.
//
// A graph that still has the launch parameters it was built with walks in
// k_walk_queued (walk_queued.cuh) instead.
//
// K3 k_paths: DeepWalk (src/core/deepwalk.cpp:25-28) on the plain or
// name-paired columns.  One walker per lane, all walks the same length, so a
// warp stays converged.  Each warp stages the next 32 path positions of its
// 32 walkers in shared memory and writes them out row by row, so every store
// instruction writes 32 consecutive int32 of one path row.  On the extended
// columns DeepWalk runs in the per-lane loop of node2vec.cu.
#include <algorithm>

#include "path_rows.cuh"
#include "ptw_internal.cuh"

namespace ptw {
namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ uint64_t umin64(uint64_t x, uint64_t y) { return x < y ? x : y; }

struct WalkArgs {
    const uint2 *__restrict__ adj;
    const uint32_t *__restrict__ col;
    const uint4 *__restrict__ col_ext;       // EXT: {id, first column, degree, name} per entry
    const uint4 *__restrict__ vtx_ext;       // {id, first column, degree, name} by canonical index
    const uint32_t *__restrict__ start_map;  // canonical index -> internal
    const uint32_t *__restrict__ int2idx;    // internal -> canonical index
    const uint32_t *__restrict__ sources;    // internal ids
    const uint32_t *__restrict__ int2name;
    uint32_t *__restrict__ counts;
    uint32_t *__restrict__ pairs;            // endpoint app: [2 * walkers] names
    unsigned long long *__restrict__ ctrl;   // [0] cursor, [1] moves; k_walk_queued: [8] cursor, [9] moves so far,
                                             // [10] blocks that ended
    uint64_t w_begin;
    uint64_t n_walk;
    uint64_t thr;
    uint64_t m;  // CSR entries (index checks)
    uint32_t n;
    uint32_t key0, key1;
    uint32_t n_sources;
    uint32_t max_moves;
    uint32_t chunk;
    uint32_t hot_k;
    int start_mode;
    int hints;  // L2 eviction priorities on (see l2_policy)
    int by_name;  // EXT count walks: counts[] is indexed by vertex name (the caller's output)
};

// (of its own: k_walk's registers and time depend on the fields beside its own, up to 7%)
struct QueuedArgs : WalkArgs {
    const uint32_t *__restrict__ rows;  // row table (row_table.cuh)
    uint32_t row_runs, row_words;
    uint32_t source0;  // the only source (sources: more than one)
};

__device__ __forceinline__ uint32_t start_vertex(const WalkArgs &a, uint64_t wid)
{
    return walker_start(a.start_mode, a.start_map, a.sources, a.n, a.n_sources, a.key0, a.key1, wid);
}

__device__ __forceinline__ uint32_t start_index(const WalkArgs &a, uint64_t wid)
{
    return walker_start_index(a.start_mode, a.int2idx, a.sources, a.n, a.n_sources, a.key0, a.key1, wid);
}

// Counts a visit of internal vertex v (name nm): ids below hot_k in shared
// memory, the others in counts[] by internal id, or by name when by_name.
template <bool HOT>
__device__ __forceinline__ void count_visit(const WalkArgs &a, uint32_t *s_hot, uint32_t v, uint32_t nm,
                                            uint64_t pol)
{
    if (HOT && v < a.hot_k) atomicAdd(&s_hot[v], 1u);
    else if (a.by_name) red_add_hint(&a.counts[nm], 1u, pol);
    else red_add_hint(&a.counts[PTW_IDX(v, a.n, &a.ctrl[7], kCheckCounter)], 1u, pol);
}

// Warp-aggregated visit (all 32 lanes call it): lanes with `on` set count
// vertex v; lanes counting the same non-hot vertex merge into one reduction
// of the group's size by its lowest lane.
template <bool HOT>
__device__ __forceinline__ void count_visit_agg(const WalkArgs &a, uint32_t *s_hot, uint32_t v, bool on,
                                                uint32_t lt_mask, uint64_t pol)
{
    const bool hot = HOT && v < a.hot_k;
    const unsigned m = __ballot_sync(kFull, on && !hot);
    if (!on) return;
    if (hot) {
        atomicAdd(&s_hot[v], 1u);
        return;
    }
    const unsigned grp = __match_any_sync(m, v);
    if ((grp & lt_mask) == 0)
        red_add_hint(&a.counts[PTW_IDX(v, a.n, &a.ctrl[7], kCheckCounter)], (uint32_t)__popc(grp), pol);
}

template <bool ENDPOINT, int ILP, bool HOT, bool EXT, bool AGG = false>
__device__ __forceinline__ void walk_body(const WalkArgs &a, uint32_t *s_hot)
{
    if (HOT) {
        for (uint32_t i = threadIdx.x; i < a.hot_k; i += blockDim.x) s_hot[i] = 0;
        __syncthreads();
    }
    const uint64_t pol_keep = l2_policy(a.hints ? 1 : 0);   // row records, counters
    const uint64_t pol_stream = l2_policy(a.hints ? 2 : 0); // column array
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lt_mask = (1u << lane) - 1u;

    uint64_t wid[ILP];
    uint32_t v[ILP], step[ILP], s0[ILP];
    bool act[ILP], have[ILP];
    uint2 rec[ILP];  // {first column, degree} of v (kept across moves with EXT)
#pragma unroll
    for (int k = 0; k < ILP; ++k) {
        act[k] = have[k] = false;
        wid[k] = 0;
        v[k] = step[k] = s0[k] = 0;
        rec[k] = make_uint2(0u, 0u);
    }
    // Warp-uniform walker-id range [next, end) relative to w_begin.
    uint64_t next = 0, end = 0;
    bool exhausted = false;
    unsigned long long moves = 0;

    for (;;) {
        // ---- refill empty slots ------------------------------------------
#pragma unroll
        for (int k = 0; k < ILP; ++k) {
            const unsigned need = __ballot_sync(kFull, !act[k]);
            if (need == 0 || exhausted) continue;
            const uint32_t n_need = __popc(need);
            const uint32_t rank = __popc(need & lt_mask);
            uint64_t my = ~0ull;
            const uint64_t avail = end - next;
            const uint32_t took = (uint32_t)umin64(n_need, avail);
            if (!act[k] && rank < took) my = next + rank;
            next += took;
            if (took < n_need) {
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(&a.ctrl[0], (unsigned long long)a.chunk);
                base = __shfl_sync(kFull, base, 0);
                if (base >= a.n_walk) {
                    exhausted = true;
                    next = end = a.n_walk;
                } else {
                    next = base;
                    end = umin64(base + a.chunk, a.n_walk);
                    const uint32_t take2 = (uint32_t)umin64(n_need - took, end - next);
                    if (!act[k] && rank >= took && rank - took < take2) my = next + (rank - took);
                    next += take2;
                }
            }
            if (my != ~0ull) {
                wid[k] = a.w_begin + my;
                // EXT count walks by name hold the start's canonical index
                // until its record is loaded
                v[k] = EXT && a.by_name ? start_index(a, wid[k]) : start_vertex(a, wid[k]);
                s0[k] = v[k];
                step[k] = 0;
                act[k] = true;
                have[k] = false;
                if (!ENDPOINT && !(EXT && a.by_name)) count_visit<HOT>(a, s_hot, v[k], 0u, pol_keep);
            }
        }
        bool any = false;
#pragma unroll
        for (int k = 0; k < ILP; ++k) any |= act[k];
        if (!__any_sync(kFull, any)) break;

        // ---- one move for every active slot --------------------------------
#pragma unroll
        for (int k = 0; k < ILP; ++k) {
            if (!act[k] || (EXT && have[k])) continue;
            if (EXT && a.by_name) {
                // a walker's first move: its start record, with the start's name
                // for its start visit
                const uint4 vx = ld_hint_u4(&a.vtx_ext[PTW_IDX(v[k], a.n, &a.ctrl[7], kCheckRecord)], pol_keep);
                v[k] = vx.x;
                rec[k] = make_uint2(vx.y, vx.z);
                if (!ENDPOINT) count_visit<HOT>(a, s_hot, v[k], vx.w, pol_keep);
            } else {
                rec[k] = ld_hint_u2(&a.adj[PTW_IDX(v[k], a.n, &a.ctrl[7], kCheckRecord)], pol_keep);
            }
        }
        uint4 r[ILP];
#pragma unroll
        for (int k = 0; k < ILP; ++k)
            if (act[k])
                r[k] = philox(make_uint4((uint32_t)wid[k], (uint32_t)(wid[k] >> 32), step[k], PTW_TAG_WALK),
                              a.key0, a.key1);
        uint32_t nb[ILP], nnm[ILP];
        uint2 nrec[ILP];
#pragma unroll
        for (int k = 0; k < ILP; ++k) {
            nnm[k] = 0;
            if (act[k] && rec[k].y != 0) {
                const uint32_t e = rec[k].x + __umulhi(r[k].x, rec[k].y);
                if (EXT) {
                    const uint4 x = ld_hint_u4(&a.col_ext[PTW_IDX(e, a.m, &a.ctrl[7], kCheckColumn)], pol_stream);
                    nb[k] = x.x;
                    nrec[k] = make_uint2(x.y, x.z);
                    nnm[k] = x.w;
                } else {
                    nb[k] = ld_hint_u32(&a.col[PTW_IDX(e, a.m, &a.ctrl[7], kCheckColumn)], pol_stream);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < ILP; ++k) {
            bool counted = false;  // AGG: this lane moved and counts v[k] below
            if (act[k]) {
                bool done;
                if (rec[k].y == 0) {
                    done = true;  // no out-edge: the walk ends here
                } else {
                    v[k] = nb[k];
                    if (EXT) {
                        rec[k] = nrec[k];
                        have[k] = true;
                    }
                    ++step[k];
                    ++moves;
                    if (!ENDPOINT) {
                        if (AGG) counted = true;
                        else count_visit<HOT>(a, s_hot, v[k], nnm[k], pol_keep);
                    }
                    done = (uint64_t)r[k].y < a.thr || (a.max_moves && step[k] >= a.max_moves);
                }
                if (done) {
                    if (ENDPOINT) {
                        const uint64_t j = wid[k] - a.w_begin;
                        *reinterpret_cast<uint2 *>(&a.pairs[2 * j]) =
                            make_uint2(a.int2name[s0[k]], a.int2name[v[k]]);
                    }
                    act[k] = false;
                }
            }
            if (AGG && !ENDPOINT) count_visit_agg<HOT>(a, s_hot, v[k], counted, lt_mask, pol_keep);
        }
    }

    // ---- flush ------------------------------------------------------------
#pragma unroll
    for (int o = 16; o; o >>= 1) moves += __shfl_xor_sync(kFull, moves, o);
    if (lane == 0 && moves) atomicAdd(&a.ctrl[1], moves);
    if (HOT) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < a.hot_k; i += blockDim.x)
            if (s_hot[i]) atomicAdd(&a.counts[a.by_name ? a.int2name[i] : i], s_hot[i]);
    }
}

// Register budget chosen by the compiler (ILP=4: 72 registers, one
// 512-thread block per SM).
template <bool ENDPOINT, int ILP, bool HOT, bool EXT>
__global__ void k_walk(const WalkArgs a)
{
    extern __shared__ uint32_t s_hot[];
    walk_body<ENDPOINT, ILP, HOT, EXT>(a, s_hot);
}

// Count walks with warp-aggregated visits (tune.warp_agg).
template <int ILP, bool HOT, bool EXT>
__global__ void k_walk_agg(const WalkArgs a)
{
    extern __shared__ uint32_t s_hot[];
    walk_body<false, ILP, HOT, EXT, true>(a, s_hot);
}

// Register caps so that two blocks fit on an SM, for more walkers in flight:
// two 512-thread blocks (64 registers), two 768-thread blocks (42
// registers; ILP 2 holds 3072 walkers per SM) or two 1024-thread blocks
// (32 registers; 4096 walkers per SM at ILP 2, with a few spills).
template <bool ENDPOINT, int ILP, bool HOT, bool EXT>
__global__ void __launch_bounds__(512, 2) k_walk_b2(const WalkArgs a)
{
    extern __shared__ uint32_t s_hot[];
    walk_body<ENDPOINT, ILP, HOT, EXT>(a, s_hot);
}

template <bool ENDPOINT, int ILP, bool HOT, bool EXT>
__global__ void __launch_bounds__(768, 2) k_walk_b2_768(const WalkArgs a)
{
    extern __shared__ uint32_t s_hot[];
    walk_body<ENDPOINT, ILP, HOT, EXT>(a, s_hot);
}

template <bool ENDPOINT, int ILP, bool HOT, bool EXT>
__global__ void __launch_bounds__(1024, 2) k_walk_b2_1024(const WalkArgs a)
{
    extern __shared__ uint32_t s_hot[];
    walk_body<ENDPOINT, ILP, HOT, EXT>(a, s_hot);
}

// K1/K2 with walkers in shared memory.  Each thread owns S walker slots;
// a slot holds the walker's id, step, start name, flags and a 16-byte
// landing buffer with the record {id, first column, degree, name} of the
// vertex it stands on.  One round: refill empty slots (warp ballot, as in
// walk_body) and start their record gathers; for every other walker draw the
// move and start the gather of the chosen column entry; wait for all of the
// thread's gathers; count the landed vertices and apply the stop decisions.
// The gathers are cp.async copies into shared memory, so a thread has S of
// them in flight without holding S destination registers: with 4096
// walkers per SM in flight the random-gather rate of the GPU is reached,
// where register-resident walkers stop at about 2048.  Draws and semantics
// are those of walk_body, so results are identical.
constexpr uint32_t kSlotActive = 1, kSlotStart = 2, kSlotMoved = 4, kSlotStop = 8;

template <bool ENDPOINT, bool HOT, int S>
__global__ void __launch_bounds__(256) k_walk_async(const WalkArgs a)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t T = blockDim.x;
    const uint32_t tid = threadIdx.x;
    uint4 *land = reinterpret_cast<uint4 *>(smem);                              // [S*T]
    unsigned long long *wid = reinterpret_cast<unsigned long long *>(land + S * T); // [S*T]
    uint32_t *step = reinterpret_cast<uint32_t *>(wid + S * T);                  // [S*T]
    uint32_t *s0n = step + S * T;                                                // [S*T] start name
    uint32_t *flag = s0n + S * T;                                                // [S*T]
    uint32_t *s_hot = flag + S * T;                                              // [hot_k]
    if (HOT) {
        for (uint32_t i = tid; i < a.hot_k; i += T) s_hot[i] = 0;
    }
#pragma unroll
    for (int k = 0; k < S; ++k) flag[k * T + tid] = 0;
    __syncthreads();
    const uint64_t pol_keep = l2_policy(a.hints ? 1 : 0);
    const uint64_t pol_stream = l2_policy(a.hints ? 2 : 0);
    const uint32_t lane = tid & 31;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint64_t next = 0, end = 0;
    bool exhausted = false;
    unsigned long long moves = 0;

    for (;;) {
        // ---- refill empty slots; start their record gathers --------------
#pragma unroll 1
        for (int k = 0; k < S; ++k) {
            const uint32_t i = k * T + tid;
            const bool empty = (flag[i] & kSlotActive) == 0;
            const unsigned need = __ballot_sync(kFull, empty);
            if (need == 0 || exhausted) continue;
            const uint32_t n_need = __popc(need);
            const uint32_t rank = __popc(need & lt_mask);
            uint64_t my = ~0ull;
            const uint64_t avail = end - next;
            const uint32_t took = (uint32_t)umin64(n_need, avail);
            if (empty && rank < took) my = next + rank;
            next += took;
            if (took < n_need) {
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(&a.ctrl[0], (unsigned long long)a.chunk);
                base = __shfl_sync(kFull, base, 0);
                if (base >= a.n_walk) {
                    exhausted = true;
                    next = end = a.n_walk;
                } else {
                    next = base;
                    end = umin64(base + a.chunk, a.n_walk);
                    const uint32_t take2 = (uint32_t)umin64(n_need - took, end - next);
                    if (empty && rank >= took && rank - took < take2) my = next + (rank - took);
                    next += take2;
                }
            }
            if (my != ~0ull) {
                const uint64_t w = a.w_begin + my;
                wid[i] = w;
                step[i] = 0;
                flag[i] = kSlotActive | kSlotStart;
                cp_async16(&land[i], &a.vtx_ext[PTW_IDX(start_index(a, w), a.n, &a.ctrl[7], kCheckRecord)], pol_keep);
            }
        }
        bool any = false;
#pragma unroll 1
        for (int k = 0; k < S; ++k) any |= (flag[k * T + tid] & kSlotActive) != 0;
        if (!__any_sync(kFull, any)) break;

        // ---- draw and start one move for every walker standing on a record
#pragma unroll 1
        for (int k = 0; k < S; ++k) {
            const uint32_t i = k * T + tid;
            const uint32_t f = flag[i];
            if ((f & kSlotActive) == 0 || (f & kSlotStart)) continue;
            const uint4 x = land[i];  // {v, first column, degree, name}
            if (x.z == 0) {           // no out-edge: the walk ends here
                if (ENDPOINT) {
                    const uint64_t j = wid[i] - a.w_begin;
                    *reinterpret_cast<uint2 *>(&a.pairs[2 * j]) = make_uint2(s0n[i], x.w);
                }
                flag[i] = 0;
                continue;
            }
            const uint64_t w = wid[i];
            const uint32_t st = step[i];
            const uint4 r = philox(make_uint4((uint32_t)w, (uint32_t)(w >> 32), st, PTW_TAG_WALK), a.key0, a.key1);
            const bool stop = (uint64_t)r.y < a.thr || (a.max_moves && st + 1 >= a.max_moves);
            flag[i] = kSlotActive | kSlotMoved | (stop ? kSlotStop : 0u);
            cp_async16(&land[i], &a.col_ext[PTW_IDX((uint64_t)x.y + __umulhi(r.x, x.z), a.m, &a.ctrl[7], kCheckColumn)],
                       pol_stream);
        }
        cp_async_wait_all();

        // ---- count the landed vertices, apply the stop decisions -----------
#pragma unroll 1
        for (int k = 0; k < S; ++k) {
            const uint32_t i = k * T + tid;
            const uint32_t f = flag[i];
            if ((f & kSlotActive) == 0) continue;
            const uint4 x = land[i];
            if (f & kSlotStart) {
                s0n[i] = x.w;
                if (!ENDPOINT) count_visit<HOT>(a, s_hot, x.x, 0u, pol_keep);
                flag[i] = kSlotActive;
            } else if (f & kSlotMoved) {
                step[i] += 1;
                ++moves;
                if (!ENDPOINT) count_visit<HOT>(a, s_hot, x.x, 0u, pol_keep);
                if (f & kSlotStop) {
                    if (ENDPOINT) {
                        const uint64_t j = wid[i] - a.w_begin;
                        *reinterpret_cast<uint2 *>(&a.pairs[2 * j]) = make_uint2(s0n[i], x.w);
                    }
                    flag[i] = 0;
                } else {
                    flag[i] = kSlotActive;
                }
            }
        }
    }

#pragma unroll
    for (int o = 16; o; o >>= 1) moves += __shfl_xor_sync(kFull, moves, o);
    if (lane == 0 && moves) atomicAdd(&a.ctrl[1], moves);
    if (HOT) {
        __syncthreads();
        for (uint32_t i = tid; i < a.hot_k; i += T)
            if (s_hot[i]) atomicAdd(&a.counts[i], s_hot[i]);
    }
}

// Dynamic shared memory of k_walk_async: 36 bytes per slot + hot counters.
inline size_t async_smem(int slots, int block, uint32_t hot_k)
{
    return (size_t)slots * block * 36 + (size_t)hot_k * 4;
}

struct PathArgs {
    const uint2 *__restrict__ adj;
    const uint32_t *__restrict__ col;
    const uint2 *__restrict__ col_named;  // {internal id, name} per column entry
    const uint32_t *__restrict__ start_map;
    const uint32_t *__restrict__ sources;
    const uint32_t *__restrict__ int2name;
    int32_t *__restrict__ paths;
    unsigned long long *check;  // index-check word (checked build)
    uint64_t w_begin, n_walk;
    uint64_t m;  // CSR entries (index checks)
    uint32_t n, L;
    uint32_t key0, key1;
    uint32_t n_sources;
    int start_mode;
    int hints;
};

// (of its own: with these fields among the others k_paths<2> takes 67 registers
// instead of 52, and 10% longer)
struct PathRowsArgs : PathArgs {
    const uint32_t *__restrict__ rows;    // row table
    uint32_t row_runs, row_words;
    unsigned long long *counters;         // {moves, draws} of node2vec, or null
    uint32_t tag;                         // draw tag: "WALK" or "N2"
    const uint4 *__restrict__ col_ext;    // extended columns: {id, first column, degree, name} per entry
    const uint4 *__restrict__ vtx_ext;    // and per vertex, by canonical index
    const uint32_t *__restrict__ int2idx;
    bool hot_cols;                        // columns through L1
};

constexpr int kPathWarps = 4;  // warps per block

// G groups of 32 consecutive walkers per warp (one walker of each group per
// lane), stepped together so a lane has G gathers in flight.  MODE 0 reads
// the row record, the column entry and the neighbour's name (three random
// reads per move); MODE 1 reads {internal id, name} pairs from col_named (two:
// row record, pair).  With the extended columns (one read per move) DeepWalk
// runs in the per-lane loop of node2vec.cu instead.
template <int G, int MODE>
__global__ void __launch_bounds__(kPathWarps * 32) k_paths(const PathArgs a)
{
    // C path positions are staged per walker before a flush; rows are padded
    // to C+1 words so the per-lane column writes do not conflict on banks.
    constexpr uint32_t C = G == 1 ? 32 : 16;
    __shared__ int32_t stage[kPathWarps][G][32][C + 1];
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t wib = threadIdx.x >> 5;
    const uint64_t n_groups = (a.n_walk + 31) / 32;
    const uint64_t warps = (uint64_t)gridDim.x * kPathWarps;

    const uint64_t pol_keep = l2_policy(a.hints ? 1 : 0);   // row records, names
    const uint64_t pol_stream = l2_policy(a.hints ? 2 : 0); // column array

    for (uint64_t g0 = (blockIdx.x * (uint64_t)kPathWarps + wib) * G; g0 < n_groups; g0 += warps * G) {
        uint64_t wid[G];
        uint32_t v[G], rows[G];
        bool dead[G];
        uint2 rec[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const uint64_t grp = g0 + g;
            const uint64_t j = grp * 32 + lane;  // walker offset
            const bool valid = j < a.n_walk;
            wid[g] = a.w_begin + j;
            rows[g] = grp < n_groups ? (uint32_t)umin64(32, a.n_walk - grp * 32) : 0;
            v[g] = valid ? walker_start(a.start_mode, a.start_map, a.sources, a.n, a.n_sources, a.key0, a.key1, wid[g]) : 0;
            dead[g] = !valid;
            stage[wib][g][lane][0] = valid ? (int32_t)a.int2name[v[g]] : -1;
        }
        uint32_t c0 = 0;  // path position of stage column 0
        for (uint32_t p = 1; p <= a.L; ++p) {
            if (p == a.L || p % C == 0) {
                // flush columns [c0, p) of every group's rows; consecutive
                // lanes write consecutive positions of one path row
                __syncwarp();
                const uint32_t cols = p - c0;
#pragma unroll
                for (int g = 0; g < G; ++g)
                    for (uint32_t idx = lane; idx < rows[g] * cols; idx += 32) {
                        const uint32_t rr = idx / cols, cc = idx - rr * cols;
                        a.paths[((g0 + g) * 32 + rr) * (uint64_t)a.L + c0 + cc] = stage[wib][g][rr][cc];
                    }
                __syncwarp();
                c0 = p;
                if (p == a.L) break;
            }
#pragma unroll
            for (int g = 0; g < G; ++g)
                if (!dead[g]) rec[g] = ld_hint_u2(&a.adj[PTW_IDX(v[g], a.n, a.check, kCheckRecord)], pol_keep);
            uint4 r[G];
#pragma unroll
            for (int g = 0; g < G; ++g)
                if (!dead[g])
                    r[g] = philox(make_uint4((uint32_t)wid[g], (uint32_t)(wid[g] >> 32), p - 1, PTW_TAG_WALK),
                                  a.key0, a.key1);
            uint32_t nm[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                if (!dead[g]) {
                    if (rec[g].y == 0) {
                        dead[g] = true;
                    } else if (MODE == 1) {
                        const uint2 cn = ld_hint_u2(
                            &a.col_named[PTW_IDX((uint64_t)rec[g].x + __umulhi(r[g].x, rec[g].y), a.m, a.check,
                                                 kCheckColumn)],
                            pol_stream);
                        v[g] = cn.x;
                        nm[g] = cn.y;
                    } else {
                        v[g] = ld_hint_u32(&a.col[PTW_IDX((uint64_t)rec[g].x + __umulhi(r[g].x, rec[g].y), a.m, a.check,
                                                          kCheckColumn)],
                                           pol_stream);
                    }
                }
            }
#pragma unroll
            for (int g = 0; g < G; ++g) {
                int32_t out = -1;
                if (!dead[g])
                    out = MODE != 0 ? (int32_t)nm[g]
                                    : (int32_t)ld_hot_u32(&a.int2name[PTW_IDX(v[g], a.n, a.check, kCheckCounter)],
                                                          pol_keep);
                stage[wib][g][lane][p - c0] = out;
            }
        }
    }
}

constexpr int kPathRowsBlock = 768;   // many waves: 768 threads per SM (1,024: 5-15% slower)
constexpr int kPathWaveBlock = 1024;  // one wave
constexpr uint64_t kPathExtBytes = 512ull << 20;  // extended columns up to here: k_paths_rows
constexpr uint64_t kPathHotBytes = 1ull << 20;    // columns up to here: through L1
constexpr uint64_t kPathPairBytes = 512ull << 10; // columns up to here, many walkers: k_paths (short paths: twice)
constexpr uint32_t kPathStage = 32;   // positions collected before they are written

// DeepWalk of a graph whose path parameters are the ones it was built with
// (paths_launch_is_auto): one walker per lane, warps take groups of 32
// consecutive walkers in turn (all walks have one length), a move is one 4-byte
// gather from the plain columns; no column copy is built or read.  The
// neighbour's name is loaded beside the next gather, through L1 (the hubs'
// names are asked for by all SMs), and the draw of a move is made while the
// gather before it is on its way.  The columns come through L1 where their lines
// are shared (hot_cols): on small graphs and from given sources.
// MANY (more walkers than one wave): the row comes from the row table in shared
// memory, and a warp's paths are collected there and written 32 positions of
// one row at a time, first to be evicted from L2: in pieces of 16 bytes they
// leave it half-filled and cost DRAM a line each time (R-MAT scale 22, 80
// positions: 39 against 47 G moves/s), at normal priority they push out columns
// and names (scale 20: 54 against 79).  Otherwise the row record from L2 is as
// quick, the output fits L2, and paths are written from registers.
// Against k_paths on name-paired columns, one walker per vertex, 80 positions:
// scale 10 66 -> 41 us, 16 74 -> 51, 18 169 -> 138, 20 859 -> 588, 22 4,563 ->
// 3,800 us, 24 19.6 -> 18.5 ms.  At scale 22 a move without names and stores
// takes as long (50 G moves/s): it is one DRAM line.
// EXT (extended columns asked for): the record and the name come with the 16-byte
// entry.  Against k_lane_paths, scale 10 to 16 91 - 102 -> 31 - 37 us, 18 311 ->
// 216, 19 606 -> 475, 20 1,127 -> 1,080 us; of columns that DRAM holds for the most
// part (kPathExtBytes) k_lane_paths reads more (scale 22 4.1 against 4.7 ms).
// node2vec with p = q = 1 accepts every first draw: the same walk with its tag.
// Many walkers on columns of up to kPathPairBytes are left to k_paths, whose id and
// name come with one read that hits L1: 2 M walkers, 20 positions, scale 8 208 against
// 238 us, 11 247 / 282, 12 267 / 286; scale 13 (0.8 MB) 283 / 285, but 5 positions
// 94 / 104.
template <bool MANY, bool EXT>
__global__ void __launch_bounds__(MANY ? kPathRowsBlock : kPathWaveBlock, 1) k_paths_rows(const PathRowsArgs a)
{
    extern __shared__ __align__(16) uint32_t s_rows[];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t(*stage)[kPathStage + 1] =
        reinterpret_cast<int32_t(*)[kPathStage + 1]>(s_rows + a.row_words) + warp * 32;
    if (MANY && !EXT) {
        row_table_load(s_rows, a.rows, a.row_words);
        __syncthreads();
    }
    // the columns at normal priority: first to be evicted, they do not replace what
    // other kernels left in L2 (scale 20 after a build, whose temporaries stay mapped,
    // 810 -> 620 us; in a row of calls 40 positions 397 -> 302, scale 21 811 -> 741,
    // 22 and 23 the same)
    const uint64_t pol_keep = l2_policy(1), pol_col = l2_policy(0), pol_out = l2_policy(2);
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    const uint64_t n_groups = (a.n_walk + 31) / 32;
    unsigned long long moves = 0;
    for (uint64_t g = (uint64_t)blockIdx.x * (blockDim.x >> 5) + warp; g < n_groups; g += warps) {
        const uint64_t j = g * 32 + lane;
        bool alive = j < a.n_walk;
        const uint64_t wid = a.w_begin + j;
        PathOut out;
        uint32_t v = 0, rx = 0;
        uint2 rec = make_uint2(0u, 0u);
        int32_t name = -1;
        if (alive) {
            if (EXT) {
                const uint32_t i =
                    walker_start_index(a.start_mode, a.int2idx, a.sources, a.n, a.n_sources, a.key0, a.key1, wid);
                const uint4 x = ld_hint_u4(&a.vtx_ext[PTW_IDX(i, a.n, a.check, kCheckRecord)], pol_keep);
                rec = make_uint2(x.y, x.z);
                name = (int32_t)x.w;
            } else {
                v = walker_start(a.start_mode, a.start_map, a.sources, a.n, a.n_sources, a.key0, a.key1, wid);
                name = (int32_t)ld_hot_u32(&a.int2name[PTW_IDX(v, a.n, a.check, kCheckCounter)], pol_keep);
            }
            rx = philox(make_uint4((uint32_t)wid, (uint32_t)(wid >> 32), 0u, a.tag), a.key0, a.key1).x;
            if (!MANY) out.start(a.paths + j * a.L);
        }
        // Writes positions [c0, p) of the group's rows, consecutive lanes
        // consecutive positions of one row (fewer than 32: and of the next rows).
        auto flush = [&](uint32_t c0, uint32_t p) {
            __syncwarp();
            const uint32_t rows = (uint32_t)umin64(32, a.n_walk - g * 32), cols = p - c0;
            int32_t *o = a.paths + g * 32 * a.L + c0;
            if (cols == 32) {
#pragma unroll 4
                for (uint32_t r = 0; r < rows; ++r) st_hint_s32(o + (uint64_t)r * a.L + lane, stage[r][lane], pol_out);
            } else {
                for (uint32_t i = lane; i < rows * cols; i += 32) {
                    const uint32_t r = i / cols, c = i - r * cols;
                    st_hint_s32(o + (uint64_t)r * a.L + c, stage[r][c], pol_out);
                }
            }
            __syncwarp();
        };
        const bool valid = alive;
        for (uint32_t p = 1; p < a.L; ++p) {
            uint32_t next_name = ~0u;  // EXT
            if (alive) {
                if (!EXT) {
                    const uint32_t x = (uint32_t)PTW_IDX(v, a.n, a.check, kCheckRecord);
                    rec = MANY ? row_of(s_rows, a.row_runs, x) : ld_hint_u2(&a.adj[x], pol_keep);
                }
                alive = rec.y != 0;  // no out-edge: -1 from here on
                if (alive) {
                    const uint64_t e = PTW_IDX((uint64_t)rec.x + __umulhi(rx, rec.y), a.m, a.check, kCheckColumn);
                    if (EXT) {
                        const uint4 x = ld_line_u4(&a.col_ext[e], pol_col);
                        rec = make_uint2(x.y, x.z);
                        next_name = x.w;
                    } else {
                        v = a.hot_cols ? ld_hot_u32(&a.col[e], pol_col) : ld_line_u32(&a.col[e], pol_col);
                    }
                }
            }
            if (MANY) {
                stage[lane][(p - 1) % kPathStage] = name;
                if (p % kPathStage == 0) flush(p - kPathStage, p);
            } else if (valid) {
                out.put(p - 1, name);
            }
            if (alive) rx = philox(make_uint4((uint32_t)wid, (uint32_t)(wid >> 32), p, a.tag), a.key0, a.key1).x;
            if (EXT) name = (int32_t)next_name;
            else name = alive ? (int32_t)ld_hot_u32(&a.int2name[PTW_IDX(v, a.n, a.check, kCheckCounter)], pol_keep) : -1;
            moves += alive;
        }
        if (MANY) {
            stage[lane][(a.L - 1) % kPathStage] = name;
            flush((a.L - 1) / kPathStage * kPathStage, a.L);
        } else if (valid) {
            out.put(a.L - 1, name);
            out.finish(a.L);
        }
    }
    if (a.counters) {  // node2vec: every move is its first draw
#pragma unroll
        for (int o = 16; o; o >>= 1) moves += __shfl_xor_sync(~0u, moves, o);
        if (lane == 0 && moves) {
            atomicAdd(&a.counters[0], moves);
            atomicAdd(&a.counters[1], moves);
        }
    }
}

__global__ void k_name_columns(const uint32_t *col, const uint32_t *int2name, uint64_t m, uint2 *col_named)
{
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = col[e];
        col_named[e] = make_uint2(c, int2name[c]);
    }
}

// {neighbour id, its first column, its degree, its name} for every entry.
__global__ void k_ext_columns(const uint32_t *col, const uint2 *adj, const uint32_t *int2name, uint64_t m,
                              uint4 *col_ext)
{
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = col[e];
        const uint2 r = adj[c];
        col_ext[e] = make_uint4(c, r.x, r.y, int2name[c]);
    }
}

// The vertex records in canonical order (by name rank).
__global__ void k_vertex_ext(const uint2 *adj, const uint32_t *int2name, const uint32_t *idx2int, uint32_t n,
                             uint4 *vtx_ext)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t v = idx2int[i];
        const uint2 r = adj[v];
        vtx_ext[i] = make_uint4(v, r.x, r.y, int2name[v]);
    }
}

__global__ void k_counts_by_name(const uint32_t *counts, const uint32_t *int2name, uint32_t n,
                                 uint32_t *out)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[int2name[i]] = counts[i];
}

// cap: 0 = no register cap, 512 / 768 / 1024 = two blocks of that size per SM.
template <bool E, int ILP, bool H, bool X> void *walk_fn(int cap)
{
    switch (cap) {
    case 512: return (void *)k_walk_b2<E, ILP, H, X>;
    case 768: return (void *)k_walk_b2_768<E, ILP, H, X>;
    case 1024: return (void *)k_walk_b2_1024<E, ILP, H, X>;
    default: return (void *)k_walk<E, ILP, H, X>;
    }
}

template <bool E, bool H, bool X> void *walk_fn_ilp(int ilp, int cap)
{
    switch (ilp) {
    case 1: return walk_fn<E, 1, H, X>(cap);
    case 4: return walk_fn<E, 4, H, X>(cap);
    default: return walk_fn<E, 2, H, X>(cap);
    }
}

template <bool X> void *pick_walk_x(bool endpoint, int ilp, bool hot, int cap)
{
    if (endpoint) return walk_fn_ilp<true, false, X>(ilp, cap);
    if (hot) return walk_fn_ilp<false, true, X>(ilp, cap);
    return walk_fn_ilp<false, false, X>(ilp, cap);
}

void *pick_walk_async(bool endpoint, bool hot, int slots)
{
    if (slots == 16) {
        if (endpoint) return (void *)k_walk_async<true, false, 16>;
        return hot ? (void *)k_walk_async<false, true, 16> : (void *)k_walk_async<false, false, 16>;
    }
    if (endpoint) return (void *)k_walk_async<true, false, 8>;
    return hot ? (void *)k_walk_async<false, true, 8> : (void *)k_walk_async<false, false, 8>;
}

template <bool H, bool X> void *agg_fn(int ilp)
{
    switch (ilp) {
    case 1: return (void *)k_walk_agg<1, H, X>;
    case 4: return (void *)k_walk_agg<4, H, X>;
    default: return (void *)k_walk_agg<2, H, X>;
    }
}

void *pick_walk_agg(int ilp, bool hot, bool ext)
{
    if (ext) return hot ? agg_fn<true, true>(ilp) : agg_fn<false, true>(ilp);
    return hot ? agg_fn<true, false>(ilp) : agg_fn<false, false>(ilp);
}

// min_blocks 2 picks the register cap by block size (checked by check_tune).
void *pick_walk(bool endpoint, int ilp, bool hot, int min_blocks, int block, bool ext)
{
    const int cap = min_blocks != 2 ? 0 : block <= 512 ? 512 : block <= 768 ? 768 : 1024;
    return ext ? pick_walk_x<true>(endpoint, ilp, hot, cap) : pick_walk_x<false>(endpoint, ilp, hot, cap);
}

}  // namespace
}  // namespace ptw

#include "walk_queued.cuh"

namespace ptw {

constexpr uint64_t kColumnsStay = 192ull << 20;  // columns up to here stay in L2 for the most part
constexpr uint64_t kLocalBytes = 160 * 1024;     // row records and columns up to here are copied to shared memory

uint64_t one_wave_walkers(const ptw_graph *g) { return (uint64_t)g->num_sms * kQueuedBlock; }

ptw_tune default_tune()
{
    ptw_tune t{};
    t.block = 256;
    t.ilp = 2;
    t.chunk = 256;
    t.paths_ilp = 2;
    t.cache_hints = 1;
    t.paths_named = 1;
    return t;
}

bool walk_launch_is_auto(const ptw_tune &t)
{
    const ptw_tune d = default_tune();
    return t.block == d.block && t.ilp == d.ilp && t.chunk == d.chunk && t.hot_k == d.hot_k &&
           t.blocks_per_sm == d.blocks_per_sm && t.min_blocks == d.min_blocks && t.cache_hints == d.cache_hints &&
           !(t.ext_columns & 1) && t.gather_slots == d.gather_slots && t.warp_agg == d.warp_agg;
}

static bool paths_launch_is_auto(const ptw_tune &t)
{
    const ptw_tune d = default_tune();
    return t.paths_ilp == d.paths_ilp && t.paths_named == d.paths_named && t.cache_hints == d.cache_hints &&
           !(t.ext_columns & 2);
}

// k_walk_queued takes the walks of a graph whose launch parameters are untouched,
// and of others those of one wave, where block, chunk and layout only decide how
// few SMs share them: the launch that is best at scale 24 (768 threads, chunk 64,
// 8,192 hot counters, extended columns) took 16 to 100% longer for 300 to 155,000
// walkers on R-MAT scales 10 to 22 (30,000 at scale 16 77 us against 54, 100,000 at
// scale 20 94 against 73; of 300,000 on either may win).  Merged visits, walkers in
// shared memory and a limit on blocks stay what they say.
bool walk_is_queued(const ptw_graph *g, const ptw_tune &t, uint64_t n_walk)
{
    return walk_launch_is_auto(t) ||
           (n_walk <= one_wave_walkers(g) && !t.warp_agg && !t.gather_slots && !t.blocks_per_sm && t.cache_hints);
}

bool count_walk_by_name(ptw_graph *g, const ptw_tune &t, uint64_t n_walk)
{
    if (walk_is_queued(g, t, n_walk)) return n_walk <= one_wave_walkers(g);
    return !t.gather_slots && !t.warp_agg && (t.ext_columns & 1) && ensure_ext_columns(g);
}

// Builds the extended column copy on first use; false (and no error) when
// it does not fit in device memory, so the caller walks without it.
bool ensure_ext_columns(ptw_graph *g)
{
    if (g->dg.col_ext) return true;
    const DeviceGraph &dg = g->dg;
    uint4 *cx = nullptr;
    if (device_malloc(&cx, std::max<uint64_t>(dg.m, 1) * sizeof(uint4)) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const unsigned grid = (unsigned)std::min<uint64_t>((dg.m + 255) / 256, (uint64_t)g->num_sms * 64);
    k_ext_columns<<<std::max(grid, 1u), 256, 0, g->stream>>>(dg.col, dg.adj, dg.int2name, dg.m, cx);
    if (cudaGetLastError() != cudaSuccess) {
        cudaFree(cx);
        return false;
    }
    uint4 *vx = nullptr;
    if (device_malloc(&vx, std::max<uint32_t>(dg.n, 1) * sizeof(uint4)) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(cx);
        return false;
    }
    const unsigned vgrid = (unsigned)std::min<uint64_t>((dg.n + 255) / 256, (uint64_t)g->num_sms * 64);
    k_vertex_ext<<<std::max(vgrid, 1u), 256, 0, g->stream>>>(dg.adj, dg.int2name, dg.idx2int, dg.n, vx);
    if (cudaGetLastError() != cudaSuccess) {
        cudaFree(cx);
        cudaFree(vx);
        return false;
    }
    g->dg.col_ext = cx;
    g->dg.vtx_ext = vx;
    g->device_bytes += dg.m * sizeof(uint4) + (uint64_t)dg.n * sizeof(uint4);
    return true;
}

void drop_unused_columns(ptw_graph *g)
{
    DeviceGraph &dg = g->dg;
    if (dg.col_ext && !g->tune.ext_columns && !g->tune.gather_slots && g->ext_users == 0) {
        cudaStreamSynchronize(g->stream);
        cudaFree(dg.col_ext);
        cudaFree(dg.vtx_ext);
        dg.col_ext = nullptr;
        dg.vtx_ext = nullptr;
        g->device_bytes -= dg.m * sizeof(uint4) + (uint64_t)dg.n * sizeof(uint4);
    }
    if (dg.col_named && ((g->tune.ext_columns & 2) || !g->tune.paths_named)) {
        cudaStreamSynchronize(g->stream);
        cudaFree(dg.col_named);
        dg.col_named = nullptr;
        g->device_bytes -= dg.m * sizeof(uint2);
    }
}

int check_tune(const ptw_tune &t)
{
    if (t.block < 32 || t.block > 1024 || t.block % 32)
        return fail(PTW_EINVAL, "tune.block must be a multiple of 32 in [32, 1024]");
    if (t.ilp != 1 && t.ilp != 2 && t.ilp != 4) return fail(PTW_EINVAL, "tune.ilp must be 1, 2 or 4");
    if (t.chunk < 1 || t.chunk > (1 << 20)) return fail(PTW_EINVAL, "tune.chunk must be in [1, 2^20]");
    if (t.hot_k < 0 || t.hot_k > 48 * 1024)
        return fail(PTW_EINVAL, "tune.hot_k must be in [0, 49152]");
    if (t.blocks_per_sm < 0 || t.blocks_per_sm > 64) return fail(PTW_EINVAL, "tune.blocks_per_sm out of range");
    if (t.min_blocks != 0 && t.min_blocks != 1 && t.min_blocks != 2)
        return fail(PTW_EINVAL, "tune.min_blocks must be 0, 1 or 2");
    if (t.min_blocks == 2 && t.block > 512 && t.block != 768 && t.block != 1024)
        return fail(PTW_EINVAL, "tune.min_blocks = 2 needs tune.block <= 512, 768 or 1024");
    if (t.paths_ilp != 0 && t.paths_ilp != 1 && t.paths_ilp != 2 && t.paths_ilp != 4)
        return fail(PTW_EINVAL, "tune.paths_ilp must be 1, 2 or 4 (0 = default)");
    if (t.cache_hints != 0 && t.cache_hints != 1) return fail(PTW_EINVAL, "tune.cache_hints must be 0 or 1");
    if (t.paths_named != 0 && t.paths_named != 1) return fail(PTW_EINVAL, "tune.paths_named must be 0 or 1");
    if (t.ext_columns < 0 || t.ext_columns > 3) return fail(PTW_EINVAL, "tune.ext_columns must be in [0, 3]");
    if (t.gather_slots != 0 && t.gather_slots != 8 && t.gather_slots != 16)
        return fail(PTW_EINVAL, "tune.gather_slots must be 0, 8 or 16");
    if (t.gather_slots && t.block > 256) return fail(PTW_EINVAL, "tune.gather_slots needs tune.block <= 256");
    if (t.warp_agg != 0 && t.warp_agg != 1) return fail(PTW_EINVAL, "tune.warp_agg must be 0 or 1");
    if (t.warp_agg && (t.min_blocks == 2 || t.gather_slots))
        return fail(PTW_EINVAL, "tune.warp_agg needs min_blocks 0 and gather_slots 0");
    return PTW_OK;
}

namespace {

WalkArgs walk_args(ptw_graph *g, const WalkLaunch &wl)
{
    const DeviceGraph &dg = g->dg;
    WalkArgs a{};
    a.adj = dg.adj;
    a.col = dg.col;
    a.start_map = dg.idx2int;
    a.int2idx = dg.int2idx;
    a.sources = g->sc.sources;
    a.int2name = dg.int2name;
    a.counts = g->sc.counts;
    a.pairs = wl.pairs;
    a.ctrl = g->sc.ctrl;
    a.w_begin = wl.w_begin;
    a.n_walk = wl.w_end - wl.w_begin;
    a.thr = wl.thr;
    a.m = dg.m;
    a.n = dg.n;
    a.key0 = (uint32_t)wl.seed;
    a.key1 = (uint32_t)(wl.seed >> 32);
    a.n_sources = wl.n_sources;
    a.max_moves = wl.max_moves;
    a.start_mode = wl.start_mode;
    return a;
}

// The launch of a graph with the launch parameters it was built with.  Up to
// one walker per lane of 1,024 threads on every SM: as few threads per SM as
// that takes, so that all SMs share the walkers.
int launch_walk_queued(ptw_graph *g, const WalkLaunch &wl)
{
    QueuedArgs a{};
    static_cast<WalkArgs &>(a) = walk_args(g, wl);
    // Ids per take from the cursor: the takes of walks that end at once are the bound
    // (5.4 M walkers from a vertex without out-edges 140 us with 32 ids, 91 with 64, 70
    // with 128; 600,000 47, 41, 41); of longer walks (sp 0.15) all three are alike.
    const uint64_t per_lane = a.n_walk / one_wave_walkers(g);
    a.chunk = per_lane >= 4 ? 128 : per_lane >= 2 ? 64 : 32;
    a.source0 = g->h_idx2int[wl.source_index];
    if (wl.by_name) a.counts = wl.by_name;
    const bool one_wave = a.n_walk <= one_wave_walkers(g);
    const uint64_t per_sm = (a.n_walk + g->num_sms - 1) / g->num_sms;
    const bool group = wl.start_mode == PTW_START_SOURCES && !wl.endpoint;
    // A small graph is copied to shared memory by every block (of 256 threads at
    // least), and a move then waits on L2 for neither of its two accesses (8 KB, 5,000
    // walkers 54 -> 48 us a call, 150,000 90 -> 55; 153 KB 56 -> 51, 70 -> 63; of 210 KB
    // the copy takes as long).  Merging visits (group), 256 threads per block are slower
    // than the spread over all SMs (62 against 60 us).
    const bool local = one_wave && !group && local_words(g->dg.n, g->dg.m) * 4 <= kLocalBytes;
    const int block = std::max(local ? 256 : 32, (int)std::min<uint64_t>(kQueuedBlock, (per_sm + 31) / 32 * 32));
    const uint64_t grid = std::min<uint64_t>(g->num_sms, (a.n_walk + block - 1) / block);
    // Hot counters pay once their flush (hot_k words per block) is small
    // beside the visits: scale 14 (12,557 walkers) is quicker without any,
    // scale 16 (45,000) with 1,024, from one wave on 8,192 and 4,096 are alike.
    if (!wl.endpoint)
        a.hot_k = std::min<uint32_t>(!one_wave ? 8192u : a.n_walk >= 24576 ? 1024u : 0u, g->dg.n);
    // Columns that L2 holds for the most part stay at normal priority, to replace what
    // other kernels left there (scale 18 66 -> 64 us, 19 91 -> 81, 20 126 -> 116; behind
    // a kernel that filled L2 81 -> 64, 100 -> 87, 134 -> 128); larger ones are first to
    // be evicted (RWR, scale 21 94 us against 97, 23 347 against 470).
    a.hints = g->dg.m * sizeof(uint32_t) > kColumnsStay;
    const bool rows = !one_wave && g->dg.rows;
    if (rows) {
        a.rows = g->dg.rows;
        a.row_runs = g->dg.row_runs;
        a.row_words = row_words(g->dg.row_runs, g->dg.n);
    }
    void *fn = pick_walk_queued(wl.endpoint, a.hot_k > 0, one_wave, group, rows, local);
    const size_t smem = ((size_t)a.hot_k + a.row_words + (local ? local_words(g->dg.n, g->dg.m) : 0)) * 4;
    if (smem > 48 * 1024) PTW_CUDA(allow_shared(fn, kQueuedFixedBytes));
    void *args[] = {&a};
    PTW_CUDA(cudaLaunchKernel(fn, dim3((unsigned)std::max<uint64_t>(grid, 1)), dim3(block), args, smem, g->stream));
    return PTW_OK;
}

}  // namespace

int launch_walk(ptw_graph *g, const WalkLaunch &wl, const ptw_tune &t)
{
    int rc = check_tune(t);
    if (rc) return rc;
    if (walk_launch_is_auto(t)) return launch_walk_queued(g, wl);
    const DeviceGraph &dg = g->dg;
    WalkArgs a = walk_args(g, wl);
    a.chunk = (uint32_t)t.chunk;
    const bool hot = !wl.endpoint && t.hot_k > 0;
    a.hot_k = hot ? std::min<uint32_t>((uint32_t)t.hot_k, dg.n) : 0;
    a.hints = t.cache_hints;

    const bool slots = t.gather_slots != 0 && ensure_ext_columns(g);
    const bool ext = !slots && (t.ext_columns & 1) && ensure_ext_columns(g);
    a.col_ext = g->dg.col_ext;
    a.vtx_ext = g->dg.vtx_ext;
    void *fn = slots ? pick_walk_async(wl.endpoint, hot, t.gather_slots)
               : (t.warp_agg && !wl.endpoint) ? pick_walk_agg(t.ilp, hot, ext)
                                              : pick_walk(wl.endpoint, t.ilp, hot, t.min_blocks, t.block, ext);
    const size_t smem = slots ? async_smem(t.gather_slots, t.block, a.hot_k) : hot ? (size_t)a.hot_k * 4 : 0;
    if (smem > kMaxSharedBytes) return fail(PTW_EINVAL, "tune.gather_slots x tune.block x hot_k need too much shared memory");
    if (smem > 48 * 1024) PTW_CUDA(allow_shared(fn));
    int per_sm = 0;
    PTW_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, t.block, smem));
    if (per_sm < 1) return fail(PTW_EINVAL, "walk kernel does not fit on an SM with this tune");
    // (a launch that does not fit is refused whatever the number of walkers)
    if (walk_is_queued(g, t, a.n_walk)) return launch_walk_queued(g, wl);
    // extended columns carry each neighbour's name: count straight into the
    // caller's by-name array (no scatter after the walk)
    a.by_name = 0;
    if (wl.by_name) {
        if (!(ext && !t.warp_agg && !wl.endpoint)) return fail(PTW_EINVAL, "counting by name needs the plain walk on extended columns");
        a.by_name = 1;
        a.counts = wl.by_name;
    }
    if (t.blocks_per_sm > 0) per_sm = std::min(per_sm, (int)t.blocks_per_sm);
    uint64_t grid = (uint64_t)g->num_sms * per_sm;
    // No more warps than walker ranges to hand out.
    const uint64_t warps_needed = (a.n_walk + (uint64_t)a.chunk - 1) / a.chunk;
    const uint64_t max_blocks = std::max<uint64_t>(1, (warps_needed + t.block / 32 - 1) / (t.block / 32));
    grid = std::min(grid, max_blocks);

    // a single source: its entry of the index table is the list
    if (wl.start_mode == PTW_START_SOURCES && wl.n_sources == 1) a.sources = dg.idx2int + wl.source_index;
    PTW_CUDA(cudaMemsetAsync(g->sc.ctrl, 0, 2 * sizeof(unsigned long long), g->stream));
    void *args[] = {&a};
    PTW_CUDA(cudaLaunchKernel(fn, dim3((unsigned)grid), dim3(t.block), args, smem, g->stream));
    return PTW_OK;
}

namespace {

// k_paths_rows: walkers of one wave, or more of them with a row table whose
// copy fits beside the collected positions.
bool path_rows_many(const ptw_graph *g, uint64_t n_walk)
{
    return (n_walk + g->num_sms - 1) / g->num_sms > (uint64_t)kPathWaveBlock;
}

size_t path_rows_smem(uint32_t table_words)
{
    return (size_t)kPathRowsBlock * (kPathStage + 1) * 4 + table_words * 4ull;
}

}  // namespace

bool paths_rows_apply(const ptw_graph *g, uint64_t n_walk)
{
    return paths_launch_is_auto(g->tune) &&
           (!path_rows_many(g, n_walk) || (g->dg.rows && path_rows_smem(row_words(g->dg.row_runs, g->dg.n)) <= kMaxSharedBytes));
}

int launch_paths(ptw_graph *g, uint64_t w_begin, uint64_t w_end, uint32_t L, uint64_t seed,
                 int start_mode, uint32_t n_sources, int32_t *paths, uint32_t tag, unsigned long long *counters)
{
    const DeviceGraph &dg = g->dg;
    PathRowsArgs a{};
    a.adj = dg.adj;
    a.col = dg.col;
    a.start_map = dg.idx2int;
    a.sources = g->sc.sources;
    a.int2name = dg.int2name;
    a.paths = paths;
    a.check = g->sc.ctrl + 7;
    a.w_begin = w_begin;
    a.n_walk = w_end - w_begin;
    a.m = dg.m;
    a.n = dg.n;
    a.L = L;
    a.key0 = (uint32_t)seed;
    a.key1 = (uint32_t)(seed >> 32);
    a.n_sources = n_sources;
    a.start_mode = start_mode;
    a.hints = g->tune.cache_hints;
    a.tag = tag;
    a.counters = counters;
    const bool ext = (g->tune.ext_columns & 2) && ensure_ext_columns(g);
    const bool many = path_rows_many(g, a.n_walk);
    // On a small graph with walkers for many waves, the pairs of k_paths are in L1.
    const bool pairs = many && tag == PTW_TAG_WALK && dg.m * sizeof(uint32_t) <= (L <= 8 ? 2 : 1) * kPathPairBytes;
    if ((!pairs && paths_rows_apply(g, a.n_walk)) || (ext && (!many || dg.m * sizeof(uint4) <= kPathExtBytes))) {
        // One wave: as few threads per SM as the walkers take, so that all SMs
        // share them.
        const uint64_t sm_walkers = (a.n_walk + g->num_sms - 1) / g->num_sms;
        const int block = many ? kPathRowsBlock : (int)(std::max<uint64_t>(1, (sm_walkers + 31) / 32) * 32);
        const uint64_t blocks = std::max<uint64_t>(1, std::min<uint64_t>(g->num_sms, (a.n_walk + block - 1) / block));
        const void *fn = ext    ? (many ? (const void *)k_paths_rows<true, true> : (const void *)k_paths_rows<false, true>)
                         : many ? (const void *)k_paths_rows<true, false>
                                : (const void *)k_paths_rows<false, false>;
        a.rows = dg.rows;
        a.row_runs = dg.row_runs;
        a.row_words = many && !ext ? row_words(dg.row_runs, dg.n) : 0u;
        const size_t smem = many ? path_rows_smem(a.row_words) : 0;
        a.col_ext = g->dg.col_ext;
        a.vtx_ext = g->dg.vtx_ext;
        a.int2idx = dg.int2idx;
        a.hot_cols = dg.m * sizeof(uint32_t) <= kPathHotBytes || start_mode == PTW_START_SOURCES;
        if (smem > 48 * 1024) PTW_CUDA(allow_shared(fn));
        void *args[] = {&a};
        PTW_CUDA(cudaLaunchKernel(fn, dim3((unsigned)blocks), dim3(block), args, smem, g->stream));
        return PTW_OK;
    }
    // Extended columns (16 bytes per CSR entry) take precedence; then
    // name-paired columns, built once on the first path walk (8 bytes per
    // CSR entry); without either the kernel looks names up per move.
    bool named = !ext && g->tune.paths_named != 0;
    if (named && !g->dg.col_named) {
        uint2 *cn = nullptr;
        if (device_malloc(&cn, std::max<uint64_t>(dg.m, 1) * sizeof(uint2)) == cudaSuccess) {
            const unsigned grid = (unsigned)std::min<uint64_t>((dg.m + 255) / 256, (uint64_t)g->num_sms * 64);
            k_name_columns<<<std::max(grid, 1u), 256, 0, g->stream>>>(dg.col, dg.int2name, dg.m, cn);
            PTW_CUDA(cudaGetLastError());
            g->dg.col_named = cn;
            g->device_bytes += dg.m * sizeof(uint2);
        } else {
            cudaGetLastError();  // no room: walk with per-move name lookups
            named = false;
        }
    }
    a.col_named = g->dg.col_named;
    // With extended columns the walkers run in the per-lane loop of
    // node2vec.cu, each slot refilled as its walk ends (no warp lockstep).
    if (ext) return launch_lane_deepwalk(g, w_begin, w_end, L, seed, start_mode, n_sources, paths);
    const int G = g->tune.paths_ilp == 1 || g->tune.paths_ilp == 4 ? g->tune.paths_ilp : 2;
    const void *fn;
    if (named)
        fn = G == 1 ? (const void *)k_paths<1, 1> : G == 4 ? (const void *)k_paths<4, 1> : (const void *)k_paths<2, 1>;
    else
        fn = G == 1 ? (const void *)k_paths<1, 0> : G == 4 ? (const void *)k_paths<4, 0> : (const void *)k_paths<2, 0>;
    int per_sm = 0;
    PTW_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kPathWarps * 32, 0));
    per_sm = std::max(per_sm, 1);
    const uint64_t groups = (a.n_walk + 31) / 32;
    const uint64_t per_block = (uint64_t)kPathWarps * G;
    uint64_t grid = std::min<uint64_t>((uint64_t)g->num_sms * per_sm, (groups + per_block - 1) / per_block);
    grid = std::max<uint64_t>(grid, 1);
    PathArgs pa = a;
    void *args[] = {&pa};
    PTW_CUDA(cudaLaunchKernel(fn, dim3((unsigned)grid), dim3(kPathWarps * 32), args, 0, g->stream));
    return PTW_OK;
}

int launch_counts_by_name(ptw_graph *g, uint32_t *d_out)
{
    const DeviceGraph &dg = g->dg;
    if (dg.id_bound != dg.n)
        PTW_CUDA(cudaMemsetAsync(d_out, 0, (uint64_t)dg.id_bound * 4, g->stream));
    const unsigned grid = (unsigned)std::min<uint64_t>((dg.n + 255) / 256, (uint64_t)g->num_sms * 16);
    k_counts_by_name<<<std::max(grid, 1u), 256, 0, g->stream>>>(g->sc.counts, dg.int2name, dg.n, d_out);
    PTW_CUDA(cudaGetLastError());
    return PTW_OK;
}

}  // namespace ptw
