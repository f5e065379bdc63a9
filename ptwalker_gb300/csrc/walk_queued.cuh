// k_walk_queued: the count / endpoint walk of a graph whose walk launch
// parameters are the ones it was built with (walk_launch_is_auto), and of any
// graph the walks of one wave (walk_is_queued): kernel, layout and launch follow
// the number of walkers.  Included by walk.cu.
//
// What bounds such a walk is either the latency of a move (walkers for one
// wave at most: the longest walk, 75 moves for 10^5 walkers at sp 0.15, is
// the kernel's time) or, with many waves, the DRAM line that each move's
// column entry sits in.  So:
//  - one walker per lane, its first id fixed by the lane: a small call takes
//    nothing from the global cursor and spreads over all SMs.  Draws are made
//    while the gather of the move before them is on its way, and the stop
//    decision, known before the gather returns, spares the last move's draw
//    and row;
//  - with more walkers than lanes, a second walker waits behind each lane's
//    own, its start vertex loaded during an earlier move, and takes over in
//    the same round in which the first one ends;
//  - once the ids are used up, the lanes walk on in a loop without warp-wide
//    steps;
//  - ROWS: with more walkers than lanes the row of a vertex comes from the row
//    table in shared memory (row_table.cuh), which leaves one gather per move;
//    a 4-byte one, from the plain columns, through L1 (ld_hot_u32).  In one wave the L2 load of
//    adj[v] is as quick as the lookup and the table need not be copied;
//  - LOCAL: in one wave on a small graph, row records and columns are copied to
//    shared memory, and the chain of a move is its draw and two reads there;
//  - BYNAME: in one wave the visits are counted by name (an extra load off the
//    chain) and there is no second kernel after the walk;
//  - visits of the hottest ids are counted in shared memory: without it the
//    reductions on a few hub counters are the bound (2.1x slower at R-MAT
//    scale 22);
//  - GROUP (walkers from given sources): visits of one vertex by several lanes
//    are merged, and with a single source all start visits are one addition;
//  - the last block to end hands over the number of moves and clears the
//    cursor, so no launch or memset goes before or after the kernel for them.
//
// Measured on a GB300 against the launch these graphs had before (block 256,
// ILP 2, chunk 256, no hot counters), device time of the whole call, sp 0.15,
// one walker per vertex: R-MAT scale 10 61.5 -> 36 us, 14 80.9 -> 46, 18
// 120 -> 70, 20 260 -> 134, 22 759 -> 365 us; scale 20, 100,000 walkers from
// one source 158 -> 78 us.  With 8 walkers per vertex, scale 22 moves 61 G
// steps/s between W = 4n and 8n, which is the rate of independent random loads
// from an array of that size (57-61 G/s), against 54 for k_walk at its best.
#pragma once

#include "ptw_internal.cuh"

namespace ptw {
namespace {

constexpr size_t kQueuedFixedBytes = 16;  // shared memory of the kernel's own (s_moves), at most
constexpr int kQueuedBlock = 1024;  // largest block, one per SM: 768 x 2 and 1024 x 2 were 3-10% slower

// Row records and columns of a graph that is copied to shared memory whole, in
// words, each 16-byte aligned.
__host__ __device__ __forceinline__ uint32_t local_adj_words(uint32_t n) { return (2 * n + 3) & ~3u; }
__host__ __device__ __forceinline__ uint64_t local_words(uint32_t n, uint64_t m)
{
    return local_adj_words(n) + ((m + 3) & ~3ull);
}

__device__ __forceinline__ uint32_t queued_start(const QueuedArgs &a, uint64_t wid)
{
    if (a.start_mode == PTW_START_SOURCES && a.n_sources == 1) return a.source0;
    return start_vertex(a, wid);
}

// ROWS: row records from the row table in shared memory instead of adj; LOCAL: row
// records and columns from shared memory.
template <bool ENDPOINT, bool HOT, bool BYNAME, bool GROUP, bool ROWS, bool LOCAL = false>
__global__ void __launch_bounds__(kQueuedBlock, 1) k_walk_queued(const QueuedArgs a)
{
    extern __shared__ __align__(16) uint32_t s_mem[];
    const uint32_t *s_rows = s_mem;
    uint32_t *s_hot = s_mem + (ROWS ? a.row_words : LOCAL ? (uint32_t)local_words(a.n, a.m) : 0u);
    const uint2 *s_adj = reinterpret_cast<const uint2 *>(s_mem);
    const uint32_t *s_col = s_mem + local_adj_words(a.n);
    __shared__ unsigned long long s_moves;
    if (threadIdx.x == 0) s_moves = 0;
    if (ROWS) row_table_load(s_mem, a.rows, a.row_words);
    if (LOCAL) {
        // (the arrays' allocations end on 256-byte boundaries)
        const uint64_t pol = l2_policy(0);
        const uint32_t w = local_adj_words(a.n), all = (uint32_t)local_words(a.n, a.m);
        for (uint32_t i = 4 * threadIdx.x; i < w; i += 4 * blockDim.x)
            cp_async16(s_mem + i, reinterpret_cast<const uint32_t *>(a.adj) + i, pol);
        for (uint32_t i = w + 4 * threadIdx.x; i < all; i += 4 * blockDim.x) cp_async16(s_mem + i, a.col + (i - w), pol);
        cp_async_wait_all();
    }
    if (HOT)
        for (uint32_t i = threadIdx.x; i < a.hot_k; i += blockDim.x) s_hot[i] = 0;
    __syncthreads();
    const uint64_t pol_keep = l2_policy(1);    // row records, counters, names
    const uint64_t pol_stream = l2_policy(a.hints ? 2 : 0);  // column array
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lt_mask = (1u << lane) - 1u;

    // Walker ids: the first 32 per warp are its own, the others come from the
    // cursor ctrl[8] in ranges of a.chunk.
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    const uint64_t own = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32 + lane;
    const uint64_t first = warps * 32;  // ids handed out without the cursor
    uint64_t next = 0, end = 0;
    bool exhausted = first >= a.n_walk;

    // The walker of this lane: id, moves made, the draw of the next move, the
    // row it stands on (and its vertex and start, ENDPOINT).
    uint64_t wid = a.w_begin + own;
    uint32_t step = 0, rx = 0, ry = 0, v = 0, s0 = 0;
    uint2 rec = make_uint2(0u, 0u);
    bool act = own < a.n_walk;
    unsigned long long moves = 0;

    auto draw = [&](uint64_t w, uint32_t st) {
        const uint4 r = philox(make_uint4((uint32_t)w, (uint32_t)(w >> 32), st, PTW_TAG_WALK), a.key0, a.key1);
        rx = r.x;
        ry = r.y;
    };
    auto row = [&](uint32_t x) -> uint2 {
        if (ROWS) return row_of(s_rows, a.row_runs, (uint32_t)PTW_IDX(x, a.n, &a.ctrl[7], kCheckRecord));
        if (LOCAL) return s_adj[PTW_IDX(x, a.n, &a.ctrl[7], kCheckRecord)];
        return ld_hint_u2(&a.adj[PTW_IDX(x, a.n, &a.ctrl[7], kCheckRecord)], pol_keep);
    };
    auto gather = [&]() -> uint32_t {
        if (LOCAL) return s_col[PTW_IDX((uint64_t)rec.x + __umulhi(rx, rec.y), a.m, &a.ctrl[7], kCheckColumn)];
        return ld_hot_u32(&a.col[PTW_IDX((uint64_t)rec.x + __umulhi(rx, rec.y), a.m, &a.ctrl[7], kCheckColumn)],
                          pol_stream);
    };
    auto name_of = [&](uint32_t x) -> uint32_t {
        return ld_hot_u32(&a.int2name[PTW_IDX(x, a.n, &a.ctrl[7], kCheckCounter)], pol_keep);
    };
    // How much this lane has to add to the count of x (0: another lane adds
    // it, or shared memory took it).
    auto visit = [&](bool on, uint32_t x) -> uint32_t {
        const bool hot = HOT && x < a.hot_k;
        uint32_t inc = 1;
        if (GROUP) {
            const unsigned m = __ballot_sync(kFull, on && !hot);
            if (on && !hot) {
                const unsigned grp = __match_any_sync(m, x);
                inc = (grp & lt_mask) == 0 ? (uint32_t)__popc(grp) : 0u;
            }
        }
        if (!on) return 0;
        if (hot) {
            atomicAdd(&s_hot[x], 1u);
            return 0;
        }
        return inc;
    };
    auto add = [&](uint32_t x, uint32_t inc) {
        red_add_hint(&a.counts[PTW_IDX(x, a.n, &a.ctrl[7], kCheckCounter)], inc, pol_keep);
    };
    auto add_name = [&](uint32_t nm, uint32_t inc) { red_add_hint(&a.counts[nm], inc, pol_keep); };
    const bool count_start = !ENDPOINT && !(GROUP && a.n_sources == 1);

    // ---- the warp's own walkers -----------------------------------------------
    {
        uint32_t x = 0;
        if (act) {
            x = queued_start(a, wid);
            draw(wid, 0);
            rec = row(x);
            v = s0 = x;
        }
        if (count_start) {
            const uint32_t inc = visit(act, x);
            if (inc) {
                if (BYNAME) add_name(name_of(x), inc);
                else add(x, inc);
            }
        }
    }

    // ---- while there are more: one walker queued behind each lane's own -----------
    // (counting by name and LOCAL are launches of one wave, which has no more)
    if constexpr (!BYNAME && !LOCAL) if (!exhausted) {
        uint64_t qwid = 0;
        uint32_t qv = 0;
        bool queued = false;
        // ENDPOINT: the names of a walk's start and end on the way.
        bool pend = false;
        uint32_t pname = 0, sname = 0;
        uint64_t pj = 0;
        auto flush_names = [&] {
            if (pend) *reinterpret_cast<uint2 *>(&a.pairs[2 * pj]) = make_uint2(sname, pname);
            pend = false;
        };
        for (;;) {
            // 1. the move's gather
            const bool go = act && rec.y != 0;
            uint32_t nb = 0;
            if (go) nb = gather();
            const bool done = act && (!go || (uint64_t)ry < a.thr || (a.max_moves && step + 1 >= a.max_moves));

            // 2. names that arrived
            if (ENDPOINT) flush_names();

            // 3. the queue
            {
                const bool empty = !queued;
                const unsigned need = __ballot_sync(kFull, empty);
                const uint32_t n_need = __popc(need);
                const uint32_t rank = __popc(need & lt_mask);
                uint64_t my = ~0ull;
                const uint32_t took = (uint32_t)umin64(n_need, end - next);
                if (empty && rank < took) my = next + rank;
                next += took;
                if (took < n_need && !exhausted) {
                    unsigned long long base = 0;
                    if (lane == 0) base = atomicAdd(&a.ctrl[8], (unsigned long long)a.chunk) + first;
                    base = __shfl_sync(kFull, base, 0);
                    if (base >= a.n_walk) {
                        exhausted = true;
                        next = end = 0;
                    } else {
                        next = base;
                        end = umin64(base + a.chunk, a.n_walk);
                        const uint32_t take2 = (uint32_t)umin64(n_need - took, end - next);
                        if (empty && rank >= took && rank - took < take2) my = next + (rank - took);
                        next += take2;
                    }
                }
                if (my != ~0ull) {
                    qwid = a.w_begin + my;
                    qv = queued_start(a, qwid);
                    queued = true;
                }
            }

            // 4. the next draw, while the gather is on its way
            const bool adopt = queued && (done || !act);
            const bool go_on = act && !done;
            if (adopt || go_on) draw(adopt ? qwid : wid, adopt ? 0u : step + 1);

            // 5. arrival
            if (adopt || go_on) rec = row(adopt ? qv : nb);
            if (go) {
                ++step;
                ++moves;
                if (ENDPOINT) v = nb;
            }
            if (!ENDPOINT) {
                const uint32_t inc = visit(go, nb);
                if (inc) add(nb, inc);
            } else if (done) {
                pj = wid - a.w_begin;
                sname = name_of(s0);
                pname = name_of(v);
                pend = true;
            }
            if (count_start) {
                const uint32_t inc = visit(adopt, qv);
                if (inc) add(qv, inc);
            }
            if (done) act = false;
            if (adopt) {
                wid = qwid;
                step = 0;
                act = true;
                queued = false;
                if (ENDPOINT) v = s0 = qv;
            }
            if (exhausted && !__any_sync(kFull, queued || next < end)) break;
        }
        if (ENDPOINT) flush_names();
    }

    // ---- no more: every lane walks on by itself -------------------------------------
    uint32_t dname = 0, dinc = 0;  // BYNAME: the last visit, its name on the way
    while (GROUP ? __any_sync(kFull, act) : act) {
        const bool go = act && rec.y != 0;
        uint32_t nb = 0;
        if (go) nb = gather();
        if (BYNAME && dinc) add_name(dname, dinc);
        const bool done = act && (!go || (uint64_t)ry < a.thr || (a.max_moves && step + 1 >= a.max_moves));
        if (act && !done) {
            draw(wid, step + 1);
            rec = row(nb);
        }
        if (go) {
            ++step;
            ++moves;
            v = nb;
        }
        if (!ENDPOINT) {
            dinc = visit(go, nb);
            if (dinc) {
                if (BYNAME) dname = name_of(nb);
                else add(nb, dinc);
            }
        } else if (done) {
            *reinterpret_cast<uint2 *>(&a.pairs[2 * (wid - a.w_begin)]) = make_uint2(name_of(s0), name_of(v));
        }
        if (done) act = false;
    }
    if (BYNAME && dinc) add_name(dname, dinc);

    // ---- flush --------------------------------------------------------------
    __syncwarp();
#pragma unroll
    for (int o = 16; o; o >>= 1) moves += __shfl_xor_sync(kFull, moves, o);
    if (lane == 0 && moves) atomicAdd(&s_moves, moves);
    __syncthreads();
    if (HOT)
        for (uint32_t i = threadIdx.x; i < a.hot_k; i += blockDim.x)
            if (s_hot[i]) atomicAdd(&a.counts[BYNAME ? a.int2name[i] : i], s_hot[i]);
    if (threadIdx.x == 0) {
        // one source: every walker's start visit at once
        if (GROUP && !ENDPOINT && a.n_sources == 1 && blockIdx.x == 0)
            atomicAdd(&a.counts[BYNAME ? a.int2name[a.source0] : a.source0], (uint32_t)a.n_walk);
        if (s_moves) atomicAdd(&a.ctrl[9], s_moves);
        __threadfence();
        // the last block hands the total over and leaves the words at zero
        if (atomicInc(reinterpret_cast<unsigned *>(&a.ctrl[10]), gridDim.x - 1) == gridDim.x - 1) {
            __threadfence();
            a.ctrl[1] = atomicExch(&a.ctrl[9], 0ull);
            a.ctrl[8] = 0;
        }
    }
}

template <bool H, bool N, bool R> void *queued_fn(bool group)
{
    return group ? (void *)k_walk_queued<false, H, N, true, R> : (void *)k_walk_queued<false, H, N, false, R>;
}

// The count walks that launch_walk_queued asks for: by name without row table
// (one wave), or by internal id with hot counters (more).
void *pick_walk_queued(bool endpoint, bool hot, bool by_name, bool group, bool rows, bool local)
{
    if (local) {  // (one wave, not grouped)
        if (endpoint) return (void *)k_walk_queued<true, false, false, false, false, true>;
        return hot ? (void *)k_walk_queued<false, true, true, false, false, true>
                   : (void *)k_walk_queued<false, false, true, false, false, true>;
    }
    if (endpoint)
        return rows ? (void *)k_walk_queued<true, false, false, false, true>
                    : (void *)k_walk_queued<true, false, false, false, false>;
    if (by_name) return hot ? queued_fn<true, true, false>(group) : queued_fn<false, true, false>(group);
    return rows ? queued_fn<true, false, true>(group) : queued_fn<true, false, false>(group);
}

}  // namespace
}  // namespace ptw
