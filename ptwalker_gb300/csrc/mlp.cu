// Learned walker budgets: source features (K5) and a small FP32 MLP with
// hand-written forward, backward and Adam kernels (K6).  No reference
// counterpart: the reference runs every query with the same walker count.
//
// Network: x[8] -> (x - mu) / sigma -> z1 = W1^T x + b1 [64] -> relu ->
//          z2 = W2^T a1 + b2 [64] -> relu -> y = w3 . a2 + b3.
// Loss: mean squared error against normalised targets.  Parameters live in
// one flat FP32 array:
//   W1[8][64] @0, b1[64] @512, W2[64][64] @576, b2[64] @4672, w3[64] @4736, b3 @4800.
// Every reduction runs in a fixed order (one thread per parameter adding up
// the batch's samples one after the other), so gradients are deterministic and
// comparable with the FP64 reference in the tests.
//
// A training step is 3.6 MFLOP at batch 256: its time is latency.  As five
// launches per step with one thread per sample or parameter, each waiting on
// its own loads, and a copy of the loss per step, a step took 155 us.  Now one
// cluster of 16 CTAs runs the steps of several epochs in one launch (k_mlp_steps; one
// CTA where no such cluster fits): samples are spread over the CTAs in tiles of 16 (a thread makes four of the 64
// sums of a layer for two samples, weights in shared memory), then every
// CTA sums the gradients of a sixteenth of the parameters over the whole
// batch, with the optimiser's state of a parameter in its thread's registers.
// The two exchanges per step (per-sample terms, updated parameters) go through
// L2 between cluster barriers, copied to shared memory asynchronously; the
// next step's samples are read ahead.  Through distributed shared memory both
// were slower: its stores move 14 bytes per cycle and SM (terms 3,900 cycles
// against 2,500, parameters 3,000 against 900).
// Of the 17,800 cycles of a step at batch 256 the exchanges take 7,500, the layers
// 4,400 and the sums over the samples 3,600 -- both bound by their shared memory
// reads, 4 cycles per 16-byte read of a warp however many of its threads read the
// same --, the update 460.  A step takes 6 us at batch 16 and 9 us at 256;
// training 2,000 samples for 30 epochs of batch 256 went from 37.4 to 2.5 ms,
// model creation and prediction included.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "ptw_internal.cuh"

struct ptw_mlp {
    float *params = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;  // [PTW_MLP_NPARAMS], one allocation
    float norm[2 * PTW_MLP_IN + 2];  // mu[8], sigma[8], t_mu, t_sigma (host)
    uint64_t step = 0;
    int device = 0;
    cudaStream_t stream = nullptr;
};

namespace ptw {
namespace {

constexpr int IN = PTW_MLP_IN, H = PTW_MLP_HIDDEN;
constexpr int OW1 = 0, OB1 = IN * H, OW2 = OB1 + H, OB2 = OW2 + H * H, OW3 = OB2 + H, OB3 = OW3 + H;
static_assert(OB3 + 1 == PTW_MLP_NPARAMS, "parameter layout");

struct Norm {
    float mu[IN], sd[IN], tmu, tsd;
};

constexpr int kTile = 16;        // samples per tile
constexpr int kCluster = 16;     // CTAs of k_mlp_steps
constexpr int kTileThreads = 128;  // per tile: two samples and four units each
constexpr int kW2 = 256;           // W2 parameters of a CTA, and its others:
constexpr int kOthers = 4 * IN + 13;
constexpr int kStepThreads = kW2 + 64;  // one per parameter
constexpr int kRow = H + 4;      // row stride of the tile's per-sample arrays (16-byte rows, no bank conflicts)
constexpr int kChunk = kCluster * kTile;  // samples that the cluster takes at a time
constexpr int kChunkRow = kChunk + 4;

// One tile of samples.
struct Tile {
    float x[kTile][IN + 4];  // normalised inputs
    float a1[kTile][kRow];   // relu(z1)
    float z2[kTile][kRow];
    float g2[kTile][kRow];   // dL/dz2
    float e[kTile];          // dL/dy
    float y[kTile];
};

// Terms of a tile's samples, one row per unit: what the gradients add up.
constexpr int TA1 = 0, TD2 = H, TD1 = 2 * H, TA2 = 3 * H, TX = 4 * H, TE = TX + IN, kTermRows = TE + 1;
constexpr int kTermRow = kTile + 1;  // (odd: a tile's threads write columns)
constexpr int kTermsWords = (kTermRows * kTermRow + 3) & ~3;
// Rows that a CTA needs of every tile: 16 of a1 and of d2 for its W2 block; 4 of d1, d2 and
// a2, all of x, and e for its other parameters.
constexpr int kStageRows = 16 + 16 + 4 + 4 + 4 + IN + 1;

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// Asynchronous copy of n floats (a multiple of 4) to shared memory, from L2.
__device__ __forceinline__ void copy_async(float *dst, const float *src, int n, uint64_t pol)
{
    for (int i = 4 * threadIdx.x; i < n; i += 4 * blockDim.x) cp_async16(dst + i, src + i, pol);
}
constexpr int kParamsPadded = (PTW_MLP_NPARAMS + 3) & ~3;  // 16-byte copies

// acc[q][c] = fma chain over k of v[q][k] * m[k][4 * col + c], k in order.
template <int N>
__device__ __forceinline__ void dot24(float (&acc)[2][4], const float *v0, const float *v1, const float *m, int col)
{
#pragma unroll
    for (int k = 0; k < N; k += 4) {
        const float4 x0 = ld4(v0 + k), x1 = ld4(v1 + k);
        const float xs[2][4] = {{x0.x, x0.y, x0.z, x0.w}, {x1.x, x1.y, x1.z, x1.w}};
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float4 w = ld4(m + (k + r) * H + 4 * col);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                acc[q][0] = fmaf(xs[q][r], w.x, acc[q][0]);
                acc[q][1] = fmaf(xs[q][r], w.y, acc[q][1]);
                acc[q][2] = fmaf(xs[q][r], w.z, acc[q][2]);
                acc[q][3] = fmaf(xs[q][r], w.w, acc[q][3]);
            }
        }
    }
}

__device__ __forceinline__ void st4(float *p, const float (&v)[4])
{
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

__device__ __forceinline__ void load_bias(float (&z)[2][4], const float *b, int col)
{
    const float4 x = ld4(b + 4 * col);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        z[q][0] = x.x;
        z[q][1] = x.y;
        z[q][2] = x.z;
        z[q][3] = x.w;
    }
}

// Forward pass of a tile whose inputs are in t.x: a1, z2 and y, with the
// parameters w.  Called by the whole block (threads past kTileThreads only
// synchronise).
__device__ __forceinline__ void tile_forward(Tile &t, const float *w)
{
    const int s = threadIdx.x / 16 * 2, c = threadIdx.x % 16;
    const bool on = threadIdx.x < kTileThreads;
    float z[2][4];
    if (on) {
        load_bias(z, w + OB1, c);
        dot24<IN>(z, t.x[s], t.x[s + 1], w + OW1, c);
#pragma unroll
        for (int q = 0; q < 8; ++q) z[q / 4][q % 4] = z[q / 4][q % 4] > 0.f ? z[q / 4][q % 4] : 0.f;
        st4(t.a1[s] + 4 * c, z[0]);
        st4(t.a1[s + 1] + 4 * c, z[1]);
    }
    __syncthreads();
    if (on) {
        load_bias(z, w + OB2, c);
        dot24<H>(z, t.a1[s], t.a1[s + 1], w + OW2, c);
        st4(t.z2[s] + 4 * c, z[0]);
        st4(t.z2[s + 1] + 4 * c, z[1]);
    }
    __syncthreads();
    if (threadIdx.x < kTile) {
        const float *z2 = t.z2[threadIdx.x];
        float out = w[OB3];
#pragma unroll
        for (int j = 0; j < H; j += 4) {
            const float4 v = ld4(z2 + j), w3 = ld4(w + OW3 + j);
            out = fmaf(v.x > 0.f ? v.x : 0.f, w3.x, out);
            out = fmaf(v.y > 0.f ? v.y : 0.f, w3.y, out);
            out = fmaf(v.z > 0.f ? v.z : 0.f, w3.z, out);
            out = fmaf(v.w > 0.f ? v.w : 0.f, w3.w, out);
        }
        t.y[threadIdx.x] = out;
    }
}

// y of every sample, one tile per block.
__global__ void __launch_bounds__(kTileThreads) k_mlp_fwd(const float *__restrict__ P,
                                                          const __grid_constant__ Norm nm,
                                                          const float *__restrict__ x, uint32_t B, float *y)
{
    __shared__ __align__(16) float w[kParamsPadded];
    __shared__ __align__(16) Tile t;
    copy_async(w, P, kParamsPadded, l2_policy(0));
    const int s = threadIdx.x / IN, k = threadIdx.x % IN;
    const uint32_t b = blockIdx.x * kTile + s;
    t.x[s][k] = b < B ? (x[(uint64_t)b * IN + k] - nm.mu[k]) / nm.sd[k] : 0.f;
    cp_async_wait_all();
    __syncthreads();
    tile_forward(t, w);
    const uint32_t o = blockIdx.x * kTile + threadIdx.x;
    if (threadIdx.x < kTile && o < B) y[o] = t.y[threadIdx.x];
}
static_assert(kTileThreads == kTile * IN, "one input per thread");

__device__ __forceinline__ void adam(float &P, float &M, float &V, float g, float lr, float b1, float b2, float eps,
                                     float c1, float c2)
{
    // which products are rounded is spelled out: a trained model does not
    // depend on how the compiler contracts these sums here
    const float m = __fmaf_rn(1.f - b1, g, __fmul_rn(b1, M));
    const float v = __fmaf_rn(__fmul_rn(1.f - b2, g), g, __fmul_rn(b2, V));
    M = m;
    V = v;
    P -= lr * (m / c1) / (sqrtf(v / c2) + eps);
}

__device__ __forceinline__ void cluster_arrive()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

struct StepArgs {
    const float *x, *t;        // all samples
    const uint32_t *idx;       // sample of every position of every epoch (null: the position itself)
    const float *corr;         // Adam's bias corrections {c1, c2} per step
    float *P, *PT, *M, *V, *G; // parameters, W2 transposed, Adam's state, gradient
    float *terms;              // of a chunk's tiles, [2][kCluster][kTermRows][kTile]
    float *loss_terms;         // squared error of every position
    uint32_t n, batch, epochs; // positions of an epoch, positions per step
    float lr, b1, b2, eps;
};

// Parameter of a thread, -1 = none.  The CTA of rank r has W2 rows
// 16 (r / 4) .. + 15, columns 16 (r % 4) .. + 15, and columns 4 r .. 4 r + 3 of W1,
// b1, b2 and w3, and b3 (rank 0).
__device__ __forceinline__ int param_of(int rank, int tid)
{
    if (tid < kW2) return OW2 + (16 * (rank / 4) + tid / 16) * H + 16 * (rank % 4) + tid % 16;
    const int q = tid - kW2, col = 4 * rank + q % 4;
    if (q < 4 * IN) return OW1 + (q / 4) * H + col;
    if (q < 4 * IN + 12) return (q < 4 * IN + 4 ? OB1 : q < 4 * IN + 8 ? OB2 : OW3) + col;
    return q == 4 * IN + 12 && rank == 0 ? OB3 : -1;
}

// The terms row that row r of the CTA of rank `rank` holds.
__device__ __forceinline__ int staged_row(int rank, int r)
{
    if (r < 16) return TA1 + 16 * (rank / 4) + r;
    if (r < 32) return TD2 + 16 * (rank % 4) + r - 16;
    if (r < 36) return TD1 + 4 * rank + r - 32;
    if (r < 40) return TD2 + 4 * rank + r - 36;
    if (r < 44) return TA2 + 4 * rank + r - 40;
    return TX + r - 44;  // x, then e
}

// acc = v * u + acc where v > 0, as a predicated instruction (a branch per sample
// took 26 cycles of it).
__device__ __forceinline__ void fma_if_positive(float &acc, float v, float u)
{
    asm("{\n\t.reg .pred p;\n\tsetp.gt.f32 p, %1, 0f00000000;\n\t@p fma.rn.f32 %0, %1, %2, %0;\n\t}"
        : "+f"(acc)
        : "f"(v), "f"(u));
}

// acc[i][j] += the sums over n samples (a multiple of 16) of v[i] * u[j], in order;
// GATE: of those with v[i] > 0.  Two rows of each: four chains of additions keep a
// scheduler busy, with one read per addition.  The next samples are read while
// these are added.
template <bool GATE>
__device__ __forceinline__ void sum_quad(float (&acc)[2][2], const float *u, const float *v, uint32_t n)
{
    constexpr int kFar = 8 * kChunkRow;  // the second row of each
    __align__(16) float x[4][8], y[4][8];
    auto load = [&](float (&f)[4][8], uint32_t k) {
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
            *reinterpret_cast<float4 *>(f[0] + h) = ld4(u + k + h);
            *reinterpret_cast<float4 *>(f[1] + h) = ld4(u + kFar + k + h);
            *reinterpret_cast<float4 *>(f[2] + h) = ld4(v + k + h);
            *reinterpret_cast<float4 *>(f[3] + h) = ld4(v + kFar + k + h);
        }
    };
    auto add = [&](const float (&f)[4][8]) {
#pragma unroll
        for (int c = 0; c < 8; ++c)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (GATE) fma_if_positive(acc[i][j], f[2 + i][c], f[j][c]);
                    else acc[i][j] = fmaf(f[2 + i][c], f[j][c], acc[i][j]);
                }
    };
    load(x, 0);
    for (uint32_t k = 0; k < n; k += 16) {
        load(y, k + 8);
        add(x);
        if (k + 16 < n) load(x, k + 16);
        add(y);
    }
}

// The same for one pair of rows.
template <bool GATE>
__device__ __forceinline__ void sum_one(float &acc, const float *u, const float *v, uint32_t n)
{
    __align__(16) float x[2][8], y[2][8];
    auto load = [&](float (&f)[2][8], uint32_t k) {
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
            *reinterpret_cast<float4 *>(f[0] + h) = ld4(u + k + h);
            *reinterpret_cast<float4 *>(f[1] + h) = ld4(v + k + h);
        }
    };
    auto add = [&](const float (&f)[2][8]) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            if (GATE) fma_if_positive(acc, f[1][c], f[0][c]);
            else acc = fmaf(f[1][c], f[0][c], acc);
        }
    };
    load(x, 0);
    for (uint32_t k = 0; k < n; k += 16) {
        load(y, k + 8);
        add(x);
        if (k + 16 < n) load(x, k + 16);
        add(y);
    }
}

// f(0) .. f(V - 1).
template <int V, typename F> __device__ __forceinline__ void each(F f)
{
    if constexpr (V == 1) {
        f(0);
    } else {
#pragma unroll 1
        for (int v = 0; v < V; ++v) f(v);
    }
}

// TRAIN: one Adam step per batch of positions; otherwise the gradient of the
// first batch, into G.  CTAS: kCluster, the work of one rank each, or 1 where no
// such cluster fits (a partition of the device): one CTA does that of all ranks in
// turn, with the same sums in the same order (a step 31 us at batch 16 and 114 at
// 256, against the cluster's 6 and 9).
template <bool TRAIN, int CTAS>
__global__ void __launch_bounds__(kStepThreads, 1) k_mlp_steps(const StepArgs a, const __grid_constant__ Norm nm)
{
    constexpr int V = kCluster / CTAS;  // ranks per CTA
    static_assert(V == 1 || CTAS == 1, "one rank per CTA or all in one");
    extern __shared__ __align__(16) float smem[];
    float *w = smem;                     // parameters
    float *w2t = w + kParamsPadded;      // W2 transposed
    float *terms = w2t + H * H;          // of this CTA's tile, [kTermRows][kTermRow]
    float *stage = terms + kTermsWords;  // of the cluster's tiles, what this CTA adds up
    float *ones = stage + kStageRows * kChunkRow;  // a row of ones
    float *grad = ones + kChunkRow;      // sums, one per thread
    Tile &t = *reinterpret_cast<Tile *>(grad + kStepThreads);
    auto rank_of = [](int v) { return V == 1 ? (int)blockIdx.x : v; };  // one cluster
    const int tid = threadIdx.x;
    const uint64_t pol = l2_policy(0);
    for (int i = tid; i < kChunkRow; i += kStepThreads) ones[i] = 1.f;

    // This thread's parameter (of each rank), with its optimiser state.
    const int own = param_of(rank_of(0), tid);
    auto param_at = [&](int v) { return V == 1 ? own : param_of(v, tid); };
    float pP[V] = {}, pM[V] = {}, pV[V] = {};
    each<V>([&](int v) {
        const int param = param_at(v);
        if (TRAIN && param >= 0) {
            pP[v] = a.P[param];
            pM[v] = a.M[param];
            pV[v] = a.V[param];
        }
    });

    // What it copies of a tile's terms: 16 bytes of row r for r = tid / 64, + 5, ...
    // of tile tid % 64 / 4.
    constexpr int kRowStep = kStepThreads / (4 * kCluster), kRowRounds = (kStageRows + kRowStep - 1) / kRowStep;
    const int c_row = tid / (4 * kCluster), c_tile = tid / 4 % kCluster, c_part = 4 * (tid % 4);
    uint16_t c_from[kRowRounds];
    auto copied_rows = [&](int rank) {
#pragma unroll
        for (int i = 0; i < kRowRounds; ++i) {
            const int r = c_row + i * kRowStep;
            c_from[i] = (uint16_t)(r < kStageRows ? staged_row(rank, r) : 0);
        }
    };
    if (V == 1) copied_rows(rank_of(0));

    // What this thread adds up: threads 0 .. 63 W2 rows i, i + 8 and columns j, j + 8,
    // threads 64 .. 95 W1, threads 96 .. 108 b1, b2, w3 and b3 (sums of d1, d2, a2 e
    // and e; products with 1 where there is one factor).
    constexpr int SA1 = 0, SD2 = 16, SD1 = 32, SE2 = 36, SA2 = 40, SX = 44, SE = SX + IN;
    int ru = 0, rv = -1;  // staged rows (-1: ones)
    if (tid < 64) {
        ru = SD2 + tid % 8;
        rv = SA1 + tid / 8;
    } else if (tid < 96) {
        ru = SD1 + tid % 4;
        rv = SX + (tid - 64) / 4;
    } else if (tid < 96 + 13) {
        const int q = (tid - 96) / 4, c = tid % 4;
        ru = q == 0 ? SD1 + c : q == 1 ? SE2 + c : SE;
        rv = q == 2 ? SA2 + c : -1;
    }

    // Input and target of this thread in the CTA's tile of a chunk (sample
    // tid / IN, input tid % IN; sample tid), read a chunk ahead.
    const int xs = tid / IN, xk = tid % IN;
    const float mu = nm.mu[xk], sd = nm.sd[xk];
    uint32_t ix = 0, it = 0;  // their samples
    float xv = 0.f, tv = 0.f;
    // position b of epoch ep (the first of the next epoch behind the last)
    auto ahead_index = [&](int rank, uint32_t ep, uint32_t b) {
        if (b >= a.n) {
            if (!TRAIN || ++ep >= a.epochs) return;
            b = 0;
        }
        const uint64_t e0 = (uint64_t)ep * a.n;
        const uint32_t bx = b + rank * kTile + xs, bt = b + rank * kTile + tid;
        if (tid < kTileThreads && bx < a.n) ix = a.idx ? a.idx[e0 + bx] : bx;
        if (tid < kTile && bt < a.n) it = a.idx ? a.idx[e0 + bt] : bt;
    };
    auto ahead_values = [&] {
        if (tid < kTileThreads) xv = a.x[(uint64_t)ix * IN + xk];
        if (tid < kTile) tv = a.t[it];
    };
    if (V == 1) {
        ahead_index(rank_of(0), 0, 0);
        ahead_values();
    }

    uint32_t flip = 0;
    for (uint32_t ep = 0, step = 0; ep < a.epochs; ++ep)
    for (uint32_t b0 = 0; b0 < a.n; b0 += a.batch, ++step) {
        const uint32_t B = a.n - b0 < a.batch ? a.n - b0 : a.batch;
        float c1 = 0.f, c2 = 0.f;
        if (TRAIN) {
            c1 = a.corr[2 * step];
            c2 = a.corr[2 * step + 1];
        }
        // W2 transposed is not needed before the backward pass
        copy_async(w, a.P, kParamsPadded, pol);
        asm volatile("cp.async.commit_group;" ::: "memory");
        copy_async(w2t, a.PT, H * H, pol);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        float accs[V][2][2] = {};
        for (uint32_t k0 = 0; k0 < B; k0 += kChunk, flip ^= 1) {
            float *const all = a.terms + (uint64_t)flip * (kCluster * kTermRows * kTile);
            const uint32_t n = B - k0 < kChunk ? (B - k0 + kTile - 1) / kTile * kTile : kChunk;
            // ---- forward and backward of this CTA's tile ------------------------------
            each<V>([&](int v) {
                const int rank = rank_of(v);
                const uint32_t t0 = k0 + rank * kTile;  // its first sample within the batch
                if (t0 >= B) return;
                if (V != 1) {
                    ahead_index(rank, ep, b0 + k0);
                    ahead_values();
                }
                if (tid < kTileThreads) t.x[xs][xk] = t0 + xs < B ? (xv - mu) / sd : 0.f;
                __syncthreads();
                tile_forward(t, w);
                if (tid < kTile) {
                    const uint32_t b = t0 + tid;
                    float eb = 0.f;
                    if (b < B) {
                        const float tn = (tv - nm.tmu) / nm.tsd;
                        const float d = t.y[tid] - tn;
                        if (a.loss_terms) a.loss_terms[(uint64_t)ep * a.n + b0 + b] = d * d;
                        eb = 2.f * d / (float)B;
                    }
                    t.e[tid] = eb;
                    terms[TE * kTermRow + tid] = eb;
                }
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                __syncthreads();
                const int s = tid / 16 * 2, c = tid % 16;
                if (tid < kTileThreads) {
                    const float4 w3 = ld4(w + OW3 + 4 * c);
#pragma unroll
                    for (int r = s; r < s + 2; ++r) {
                        const float4 z2 = ld4(t.z2[r] + 4 * c);
                        const float e = t.e[r];
                        const float g[4] = {z2.x > 0.f ? e * w3.x : 0.f, z2.y > 0.f ? e * w3.y : 0.f,
                                            z2.z > 0.f ? e * w3.z : 0.f, z2.w > 0.f ? e * w3.w : 0.f};
                        st4(t.g2[r] + 4 * c, g);
                    }
                }
                __syncthreads();
                if (tid < kTileThreads) {
                    float g[2][4] = {};
                    dot24<H>(g, t.g2[s], t.g2[s + 1], w2t, c);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int r = s + h;
                        const bool live = t0 + r < B;  // all terms of the samples past the batch are 0
                        const float4 a1 = ld4(t.a1[r] + 4 * c), z2 = ld4(t.z2[r] + 4 * c), g2 = ld4(t.g2[r] + 4 * c);
                        const float va[4] = {a1.x, a1.y, a1.z, a1.w}, vz[4] = {z2.x, z2.y, z2.z, z2.w},
                                    vg[4] = {g2.x, g2.y, g2.z, g2.w};
                        float *o = terms + 4 * c * kTermRow + r;
#pragma unroll
                        for (int q = 0; q < 4; ++q, o += kTermRow) {
                            o[TA1 * kTermRow] = live ? va[q] : 0.f;
                            o[TD1 * kTermRow] = live && va[q] > 0.f ? g[h][q] : 0.f;
                            o[TD2 * kTermRow] = live ? vg[q] : 0.f;
                            o[TA2 * kTermRow] = live && vz[q] > 0.f ? vz[q] : 0.f;
                        }
                    }
                    terms[(TX + xk) * kTermRow + xs] = t.x[xs][xk];
                }
                __syncthreads();
                for (int i = tid; i < kTermRows * kTile / 4; i += kStepThreads) {
                    const float *f = terms + i / 4 * kTermRow + 4 * (i % 4);
                    __stcg(reinterpret_cast<float4 *>(all + (uint64_t)rank * (kTermRows * kTile)) + i,
                           make_float4(f[0], f[1], f[2], f[3]));
                }
            });
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            cluster_arrive();
            if (V == 1) ahead_index(rank_of(0), ep, k0 + kChunk < B ? b0 + k0 + kChunk : b0 + a.batch);
            cluster_wait();
            if (V == 1) ahead_values();
            // ---- gradient of this CTA's share, samples in order -----------------------
            // (the next chunk's terms go to the other half of a.terms; whoever writes to
            // this one again has passed the barrier after this copy in every CTA)
            each<V>([&](int i_rank) {
                float(&acc)[2][2] = accs[i_rank];
                if (V != 1) copied_rows(rank_of(i_rank));
                if (c_tile * kTile < n) {
                    const float *from = all + c_tile * (kTermRows * kTile) + c_part;
                    float *to = stage + c_row * kChunkRow + c_tile * kTile + c_part;
#pragma unroll
                    for (int i = 0; i < kRowRounds; ++i)
                        if (c_row + i * kRowStep < kStageRows)
                            cp_async16(to + i * (kRowStep * kChunkRow), from + c_from[i] * kTile, pol);
                }
                cp_async_wait_all();
                __syncthreads();
                const float *u = stage + ru * kChunkRow, *v = rv < 0 ? ones : stage + rv * kChunkRow;
                if (tid < 64) {
                    // A sample whose a1 is 0 adds 0 times d2, which only differs from
                    // leaving it out where d2 is not finite: then the sum is NaN and is
                    // made again with the others only (a test per sample doubles it).
                    float q[2][2] = {{acc[0][0], acc[0][1]}, {acc[1][0], acc[1][1]}};
                    sum_quad<false>(q, u, v, n);
                    if (isnan(q[0][0]) || isnan(q[0][1]) || isnan(q[1][0]) || isnan(q[1][1])) sum_quad<true>(acc, u, v, n);
                    else {
                        acc[0][0] = q[0][0];
                        acc[0][1] = q[0][1];
                        acc[1][0] = q[1][0];
                        acc[1][1] = q[1][1];
                    }
                } else if (tid < 96) {
                    sum_one<false>(acc[0][0], u, v, n);
                } else if (tid < 96 + 13) {
                    float q = acc[0][0];
                    sum_one<false>(q, u, v, n);
                    if (isnan(q)) sum_one<true>(acc[0][0], u, v, n);
                    else acc[0][0] = q;
                }
                if (V != 1) __syncthreads();
            });
        }
        each<V>([&](int v) {
            const float(&acc)[2][2] = accs[v];
            const int param = param_at(v);
            if (tid < 64) {
                float *g = grad + tid / 8 * 16 + tid % 8;
                g[0] = acc[0][0];
                g[8] = acc[0][1];
                g[8 * 16] = acc[1][0];
                g[8 * 16 + 8] = acc[1][1];
            } else if (tid < 96 + 13) {
                grad[kW2 + tid - 64] = acc[0][0];
            }
            __syncthreads();
            if (!TRAIN) {
                if (param >= 0) a.G[param] = grad[tid];
            } else if (param >= 0) {
                adam(pP[v], pM[v], pV[v], grad[tid], a.lr, a.b1, a.b2, a.eps, c1, c2);
                __stcg(a.P + param, pP[v]);
                if (tid < kW2) __stcg(a.PT + (param - OW2) % H * H + (param - OW2) / H, pP[v]);
            }
            if (V != 1) __syncthreads();
        });
        if (!TRAIN) return;
        cluster_arrive();
        cluster_wait();
    }
    each<V>([&](int v) {
        const int param = param_at(v);
        if (TRAIN && param >= 0) {
            a.M[param] = pM[v];
            a.V[param] = pV[v];
        }
    });
}

constexpr size_t kStepSmem =
    (kParamsPadded + H * H + kTermsWords + (kStageRows + 1) * kChunkRow + kStepThreads) * 4 + sizeof(Tile);

// PT = W2 transposed.
__global__ void k_mlp_transpose(const float *P, float *PT)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < H * H) PT[(p % H) * H + p / H] = P[OW2 + p];
}

// ---- K5: source features, one warp per source -----------------------------
//  f0 log(1+deg)          f1 mean log(1+deg(u))    f2 max log(1+deg(u))
//  f3 min log(1+deg(u))   f4 log(1+sum deg(u))     f5 std log(1+deg(u))
//  f6 fraction of neighbours of degree 1          f7 log(1+sum deg(u)/deg)
__global__ void k_features(const uint2 *adj, const uint32_t *col, const uint32_t *src, uint32_t ns, float *f)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t q = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; q < ns; q += warps) {
        const uint2 a = adj[src[q]];
        double s1 = 0, s2 = 0, sdeg = 0;
        float mx = -1e30f, mn = 1e30f;
        uint32_t ones = 0;
        for (uint32_t r = lane; r < a.y; r += 32) {
            const uint32_t du = adj[col[a.x + r]].y;
            const double l = log1p((double)du);
            s1 += l;
            s2 += l * l;
            sdeg += du;
            mx = fmaxf(mx, (float)l);
            mn = fminf(mn, (float)l);
            ones += du == 1;
        }
        for (int o = 16; o; o >>= 1) {
            s1 += __shfl_xor_sync(0xffffffffu, s1, o);
            s2 += __shfl_xor_sync(0xffffffffu, s2, o);
            sdeg += __shfl_xor_sync(0xffffffffu, sdeg, o);
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            ones += __shfl_xor_sync(0xffffffffu, ones, o);
        }
        if (lane == 0) {
            const double d = a.y ? (double)a.y : 1.0;
            const double mean = a.y ? s1 / d : 0.0;
            const double var = a.y ? fmax(s2 / d - mean * mean, 0.0) : 0.0;
            float *o = f + q * IN;
            o[0] = (float)log1p((double)a.y);
            o[1] = (float)mean;
            o[2] = a.y ? mx : 0.f;
            o[3] = a.y ? mn : 0.f;
            o[4] = (float)log1p(sdeg);
            o[5] = (float)sqrt(var);
            o[6] = a.y ? (float)(ones / d) : 0.f;
            o[7] = (float)log1p(sdeg / d);
        }
    }
}

Norm host_norm(const ptw_mlp *m)
{
    Norm n;
    for (int k = 0; k < IN; ++k) {
        n.mu[k] = m->norm[k];
        n.sd[k] = m->norm[IN + k] > 0 ? m->norm[IN + k] : 1.f;
    }
    n.tmu = m->norm[2 * IN];
    n.tsd = m->norm[2 * IN + 1] > 0 ? m->norm[2 * IN + 1] : 1.f;
    return n;
}

// Device buffers of a training or gradient call, from one allocation.
struct MlpScratch {
    float *base = nullptr, *x = nullptr, *t = nullptr, *pt = nullptr, *terms = nullptr, *lt = nullptr;
    cudaStream_t st;
    explicit MlpScratch(cudaStream_t s) : st(s) {}
    // N samples, `loss` squared errors.
    cudaError_t alloc(uint64_t N, uint64_t loss)
    {
        uint64_t at = 0;
        auto take = [&](uint64_t n) {
            const uint64_t o = at;
            at += (n + 3) & ~3ull;  // 16-byte rows
            return o;
        };
        const uint64_t ox = take(N * IN), ot = take(N), opt = take(H * H), otr = take(2 * kCluster * kTermRows * kTile), olt = take(loss);
        const cudaError_t e = cudaMallocAsync((void **)&base, at * 4, st);
        if (e != cudaSuccess) return e;
        x = base + ox;
        t = base + ot;
        pt = base + opt;
        terms = base + otr;
        lt = base + olt;
        return cudaSuccess;
    }
    ~MlpScratch()
    {
        if (base) cudaFreeAsync(base, st);
    }
};

// A launch of k_mlp_steps: one cluster, or one CTA where the device (a partition of
// it) has no room for a cluster of that size.  Made once per call, used for each
// of its launches.
template <bool TRAIN> struct StepLaunch {
    cudaLaunchAttribute attr{};
    cudaLaunchConfig_t cfg{};
    int init(cudaStream_t st)
    {
        const void *fn = (const void *)k_mlp_steps<TRAIN, kCluster>;
        PTW_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStepSmem));
        PTW_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kCluster;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.gridDim = dim3(kCluster);
        cfg.blockDim = dim3(kStepThreads);
        cfg.dynamicSmemBytes = kStepSmem;
        cfg.stream = st;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) != cudaSuccess) {
            cudaGetLastError();
            clusters = 0;
        }
        if (clusters) return PTW_OK;
        cfg.gridDim = dim3(1);
        cfg.attrs = nullptr;
        cfg.numAttrs = 0;
        PTW_CUDA(cudaFuncSetAttribute((const void *)k_mlp_steps<TRAIN, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kStepSmem));
        return PTW_OK;
    }
    int run(const StepArgs &a, const Norm &nm) const
    {
        if (cfg.numAttrs) PTW_CUDA(cudaLaunchKernelEx(&cfg, k_mlp_steps<TRAIN, kCluster>, a, nm));
        else PTW_CUDA(cudaLaunchKernelEx(&cfg, k_mlp_steps<TRAIN, 1>, a, nm));
        return PTW_OK;
    }
};

// Sum of n squared errors as the loss of a batch takes it.
double mean_loss(const float *lt, uint32_t n)
{
    double acc = 0;
    for (uint32_t i = 0; i < n; ++i) acc += lt[i];
    return acc / n;
}

}  // namespace
}  // namespace ptw

using namespace ptw;

extern "C" int ptw_source_features(ptw_graph *g, const uint32_t *h_sources, uint32_t ns, float *h_feat)
try {
    if (!g || (ns && (!h_sources || !h_feat))) return fail(PTW_EINVAL, "null argument");
    if (!ns) return PTW_OK;
    PTW_CUDA(cudaSetDevice(g->device));
    const uint32_t n = g->dg.n;
    std::vector<uint32_t> ids(ns);
    for (uint32_t i = 0; i < ns; ++i) {
        const uint32_t *p = std::lower_bound(g->h_names, g->h_names + n, h_sources[i]);
        if (p == g->h_names + n || *p != h_sources[i])
            return fail(PTW_EINVAL, "source " + std::to_string(h_sources[i]) + " is not a vertex of the graph");
        ids[i] = g->h_idx2int[p - g->h_names];
    }
    cudaStream_t st = g->stream;
    uint32_t *d_src = nullptr;
    float *d_f = nullptr;
    PTW_CUDA(cudaMallocAsync(&d_src, ns * 4ull, st));
    cudaError_t e = cudaMallocAsync(&d_f, ns * 4ull * IN, st);
    if (e != cudaSuccess) {
        cudaFreeAsync(d_src, st);
        return cuda_fail(e, "feature buffer");
    }
    e = cudaMemcpyAsync(d_src, ids.data(), ns * 4ull, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        const unsigned grid = (unsigned)std::min<uint64_t>(((uint64_t)ns * 32 + 255) / 256, 65535);
        k_features<<<std::max(grid, 1u), 256, 0, st>>>(g->dg.adj, g->dg.col, d_src, ns, d_f);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h_feat, d_f, ns * 4ull * IN, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFreeAsync(d_src, st);
    cudaFreeAsync(d_f, st);
    if (e != cudaSuccess) return cuda_fail(e, "source features");
    return PTW_OK;
} catch (...) {
    return host_exception();
}

extern "C" int ptw_mlp_create(uint64_t seed, ptw_mlp **out)
try {
    if (!out) return fail(PTW_EINVAL, "null argument");
    *out = nullptr;
    ptw_mlp *m = new (std::nothrow) ptw_mlp();
    if (!m) return fail(PTW_ENOMEM, "host allocation failed");
    std::memset(m->norm, 0, sizeof(m->norm));
    for (int k = 0; k < IN; ++k) m->norm[IN + k] = 1.f;
    m->norm[2 * IN + 1] = 1.f;
    int rc = PTW_OK;
    cudaError_t e = cudaGetDevice(&m->device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
    constexpr size_t row = (PTW_MLP_NPARAMS + 3) & ~3;  // 16-byte rows of one allocation
    if (e == cudaSuccess) e = device_malloc(&m->params, 4 * row * sizeof(float));
    if (e == cudaSuccess) {
        m->grad = m->params + row;
        m->m = m->params + 2 * row;
        m->v = m->params + 3 * row;
    }
    if (e != cudaSuccess) {
        rc = cuda_fail(e, "MLP allocation");
    } else {
        // He-uniform initialisation from a 64-bit LCG (Knuth MMIX constants);
        // biases zero.
        std::vector<float> h(PTW_MLP_NPARAMS, 0.f);
        uint64_t st = seed * 6364136223846793005ull + 1442695040888963407ull;
        auto uni = [&]() {
            st = st * 6364136223846793005ull + 1442695040888963407ull;
            return (double)(st >> 11) / 9007199254740992.0 * 2.0 - 1.0;
        };
        for (int i = OW1; i < OB1; ++i) h[i] = (float)(uni() * std::sqrt(6.0 / IN));
        for (int i = OW2; i < OB2; ++i) h[i] = (float)(uni() * std::sqrt(6.0 / H));
        for (int i = OW3; i < OB3; ++i) h[i] = (float)(uni() * std::sqrt(3.0 / H));
        e = cudaMemcpy(m->params, h.data(), PTW_MLP_NPARAMS * 4, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemset(m->m, 0, 2 * row * sizeof(float));
        if (e != cudaSuccess) rc = cuda_fail(e, "MLP init");
    }
    if (rc != PTW_OK) {
        ptw_mlp_free(m);
        return rc;
    }
    *out = m;
    return PTW_OK;
} catch (...) {
    return host_exception();
}

extern "C" int ptw_mlp_set_params(ptw_mlp *m, const float *h_params, const float *h_norm)
try {
    if (!m) return fail(PTW_EINVAL, "null model");
    PTW_CUDA(cudaSetDevice(m->device));
    if (h_params) PTW_CUDA(cudaMemcpy(m->params, h_params, PTW_MLP_NPARAMS * 4, cudaMemcpyHostToDevice));
    if (h_norm) std::memcpy(m->norm, h_norm, sizeof(m->norm));
    return PTW_OK;
} catch (...) {
    return host_exception();
}

extern "C" int ptw_mlp_get_params(const ptw_mlp *m, float *h_params, float *h_norm)
try {
    if (!m) return fail(PTW_EINVAL, "null model");
    PTW_CUDA(cudaSetDevice(m->device));
    if (h_params) PTW_CUDA(cudaMemcpy(h_params, m->params, PTW_MLP_NPARAMS * 4, cudaMemcpyDeviceToHost));
    if (h_norm) std::memcpy(h_norm, m->norm, sizeof(m->norm));
    return PTW_OK;
} catch (...) {
    return host_exception();
}

extern "C" int ptw_mlp_forward(ptw_mlp *m, const float *h_x, uint32_t B, float *h_y)
try {
    if (!m || (B && (!h_x || !h_y))) return fail(PTW_EINVAL, "null argument");
    if (!B) return PTW_OK;
    PTW_CUDA(cudaSetDevice(m->device));
    float *d = nullptr;  // inputs, then outputs
    PTW_CUDA(cudaMallocAsync((void **)&d, (uint64_t)B * (IN + 1) * 4, m->stream));
    struct Free {
        float *p;
        cudaStream_t st;
        ~Free() { cudaFreeAsync(p, st); }
    } guard{d, m->stream};
    float *d_y = d + (uint64_t)B * IN;
    PTW_CUDA(cudaMemcpyAsync(d, h_x, (uint64_t)B * IN * 4, cudaMemcpyHostToDevice, m->stream));
    const Norm nm = host_norm(m);
    k_mlp_fwd<<<(B + kTile - 1) / kTile, kTileThreads, 0, m->stream>>>(m->params, nm, d, B, d_y);
    PTW_CUDA(cudaGetLastError());
    PTW_CUDA(cudaMemcpyAsync(h_y, d_y, B * 4ull, cudaMemcpyDeviceToHost, m->stream));
    PTW_CUDA(cudaStreamSynchronize(m->stream));
    for (uint32_t b = 0; b < B; ++b) h_y[b] = h_y[b] * nm.tsd + nm.tmu;  // de-normalised prediction
    return PTW_OK;
} catch (...) {
    return host_exception();
}

extern "C" int ptw_mlp_grad(ptw_mlp *m, const float *h_x, const float *h_t, uint32_t B, double *h_loss,
                            float *h_grad)
try {
    if (!m || !B || !h_x || !h_t) return fail(PTW_EINVAL, "null argument or empty batch");
    PTW_CUDA(cudaSetDevice(m->device));
    cudaStream_t st = m->stream;
    MlpScratch s(st);
    PTW_CUDA(s.alloc(B, B));
    PTW_CUDA(cudaMemcpyAsync(s.x, h_x, (uint64_t)B * IN * 4, cudaMemcpyHostToDevice, st));
    PTW_CUDA(cudaMemcpyAsync(s.t, h_t, B * 4ull, cudaMemcpyHostToDevice, st));
    k_mlp_transpose<<<(H * H + 255) / 256, 256, 0, st>>>(m->params, s.pt);
    StepArgs a{};
    a.x = s.x;
    a.t = s.t;
    a.P = m->params;
    a.PT = s.pt;
    a.terms = s.terms;
    a.G = m->grad;
    a.loss_terms = s.lt;
    a.n = a.batch = B;
    a.epochs = 1;
    StepLaunch<false> steps;
    if (const int rc = steps.init(st)) return rc;
    if (const int rc = steps.run(a, host_norm(m))) return rc;
    std::vector<float> lt(h_loss ? B : 0);
    if (h_loss) PTW_CUDA(cudaMemcpyAsync(lt.data(), s.lt, B * 4ull, cudaMemcpyDeviceToHost, st));
    if (h_grad) PTW_CUDA(cudaMemcpyAsync(h_grad, m->grad, PTW_MLP_NPARAMS * 4, cudaMemcpyDeviceToHost, st));
    PTW_CUDA(cudaStreamSynchronize(st));
    if (h_loss) *h_loss = mean_loss(lt.data(), B);
    return PTW_OK;
} catch (...) {
    return host_exception();
}

extern "C" int ptw_mlp_train(ptw_mlp *m, const float *h_x, const float *h_t, uint32_t N, uint32_t batch,
                             uint32_t epochs, float lr, uint64_t seed, float *h_loss_curve)
try {
    if (!m || !N || !h_x || !h_t || !batch) return fail(PTW_EINVAL, "null argument or empty data");
    PTW_CUDA(cudaSetDevice(m->device));
    // Normalisation from the training data (features and target).
    for (int k = 0; k < IN; ++k) {
        double s = 0, s2 = 0;
        for (uint32_t i = 0; i < N; ++i) {
            s += h_x[(uint64_t)i * IN + k];
            s2 += (double)h_x[(uint64_t)i * IN + k] * h_x[(uint64_t)i * IN + k];
        }
        const double mu = s / N, var = std::max(s2 / N - mu * mu, 1e-12);
        m->norm[k] = (float)mu;
        m->norm[IN + k] = (float)std::sqrt(var);
    }
    {
        double s = 0, s2 = 0;
        for (uint32_t i = 0; i < N; ++i) {
            s += h_t[i];
            s2 += (double)h_t[i] * h_t[i];
        }
        const double mu = s / N, var = std::max(s2 / N - mu * mu, 1e-12);
        m->norm[2 * IN] = (float)mu;
        m->norm[2 * IN + 1] = (float)std::sqrt(var);
    }
    if (!epochs) return PTW_OK;
    batch = std::min(batch, N);
    cudaStream_t st = m->stream;
    const uint32_t nb = (N + batch - 1) / batch;  // steps per epoch
    // The squared errors of a run of epochs stay on the device until the run is
    // copied (64 MB at most at a time).
    const uint32_t run = h_loss_curve ? (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(epochs, (16ull << 20) / N)) : 0;
    MlpScratch s(st);
    PTW_CUDA(s.alloc(N, (uint64_t)run * N));
    // A launch runs `group` epochs, from their order of the samples and bias
    // corrections: first one, then twice as many each time (the host makes the next
    // ones meanwhile), 64 MB at most.
    const uint64_t words = (uint64_t)N + 2ull * nb;  // per epoch
    const uint32_t most = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((epochs + 1) / 2, (16ull << 20) / words));
    uint32_t *d_plan = nullptr;
    PTW_CUDA(cudaMallocAsync((void **)&d_plan, most * words * 4, st));
    struct Free {
        void *p;
        cudaStream_t st;
        ~Free() { cudaFreeAsync(p, st); }
    } guard{d_plan, st};
    PTW_CUDA(cudaMemcpyAsync(s.x, h_x, (uint64_t)N * IN * 4, cudaMemcpyHostToDevice, st));
    PTW_CUDA(cudaMemcpyAsync(s.t, h_t, N * 4ull, cudaMemcpyHostToDevice, st));
    k_mlp_transpose<<<(H * H + 255) / 256, 256, 0, st>>>(m->params, s.pt);
    StepArgs a{};
    a.x = s.x;
    a.t = s.t;
    a.idx = d_plan;
    a.P = m->params;
    a.PT = s.pt;
    a.terms = s.terms;
    a.M = m->m;
    a.V = m->v;
    a.n = N;
    a.batch = batch;
    a.lr = lr;
    a.b1 = 0.9f;
    a.b2 = 0.999f;
    a.eps = 1e-8f;
    const Norm nm = host_norm(m);
    StepLaunch<true> steps;
    if (const int rc = steps.init(st)) return rc;
    // Two plans in turn, each filled again once its last copy has read it: the copies
    // come from pageable memory, which need not have been read when a call returns.
    struct Plan {
        std::vector<uint32_t> words;
        cudaEvent_t copied = nullptr;
        ~Plan()
        {
            if (copied) cudaEventDestroy(copied);
        }
    } plans[2];
    struct Drain {  // a call that fails, before the plans go
        cudaStream_t st;
        bool on = true;
        ~Drain()
        {
            if (on) cudaStreamSynchronize(st);
        }
    } drain{st};
    std::vector<uint32_t> order(N);
    std::vector<float> lt((uint64_t)run * N);
    for (uint32_t i = 0; i < N; ++i) order[i] = i;
    uint64_t rs = seed * 0x9E3779B97F4A7C15ull + 1;
    uint32_t ep0 = 0;  // first epoch whose squared errors are not copied yet
    uint32_t group = 1;
    for (uint32_t ep = 0, turn = 0; ep < epochs; group = std::min(2 * group, most), turn ^= 1) {
        uint32_t E = std::min(group, epochs - ep);
        if (run) E = std::min(E, run - (ep - ep0));
        std::vector<uint32_t> &plan = plans[turn].words;
        if (plans[turn].copied) PTW_CUDA(cudaEventSynchronize(plans[turn].copied));
        plan.resize(std::max<uint64_t>(plan.size(), E * words));
        float *corr = reinterpret_cast<float *>(plan.data() + (uint64_t)E * N);
        for (uint32_t e = 0; e < E; ++e) {
            for (uint32_t i = N - 1; i > 0; --i) {  // Fisher-Yates with an LCG
                rs = rs * 6364136223846793005ull + 1442695040888963407ull;
                std::swap(order[i], order[(rs >> 33) % (i + 1)]);
            }
            std::copy(order.begin(), order.end(), plan.begin() + (uint64_t)e * N);
            for (uint32_t k = 0; k < nb; ++k) {
                ++m->step;
                *corr++ = 1.f - std::pow(a.b1, (float)m->step);
                *corr++ = 1.f - std::pow(a.b2, (float)m->step);
            }
        }
        PTW_CUDA(cudaMemcpyAsync(d_plan, plan.data(), E * words * 4, cudaMemcpyHostToDevice, st));
        if (ep + E < epochs) {
            if (!plans[turn].copied) PTW_CUDA(cudaEventCreateWithFlags(&plans[turn].copied, cudaEventDisableTiming));
            PTW_CUDA(cudaEventRecord(plans[turn].copied, st));
        }
        a.corr = reinterpret_cast<const float *>(d_plan + (uint64_t)E * N);
        a.loss_terms = run ? s.lt + (uint64_t)(ep - ep0) * N : nullptr;
        a.epochs = E;
        if (const int rc = steps.run(a, nm)) return rc;
        ep += E;
        if (run && (ep == epochs || ep - ep0 == run)) {
            PTW_CUDA(cudaMemcpyAsync(lt.data(), s.lt, (uint64_t)(ep - ep0) * N * 4, cudaMemcpyDeviceToHost, st));
            PTW_CUDA(cudaStreamSynchronize(st));
            for (uint32_t e = ep0; e < ep; ++e) {
                double loss = 0;
                for (uint32_t b0 = 0; b0 < N; b0 += batch)
                    loss += mean_loss(lt.data() + (uint64_t)(e - ep0) * N + b0, std::min(batch, N - b0));
                h_loss_curve[e] = (float)(loss / nb);
            }
            ep0 = ep;
        }
    }
    PTW_CUDA(cudaStreamSynchronize(st));
    drain.on = false;
    return PTW_OK;
} catch (...) {
    return host_exception();
}

extern "C" void ptw_mlp_free(ptw_mlp *m)
try {
    if (!m) return;
    cudaSetDevice(m->device);
    if (m->stream) cudaStreamSynchronize(m->stream);
    cudaFree(m->params);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
} catch (...) {
    host_exception();
}
