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
// cluster of 16 CTAs runs all steps of an epoch in one launch (k_mlp_steps):
// samples are spread over the CTAs in tiles of 16 (a thread makes four of the 64
// sums of a layer for two samples, weights in shared memory), then every
// CTA sums the gradients of a sixteenth of the parameters over the whole
// batch, with the optimiser's state of a parameter in its thread's registers.
// The two exchanges per step (per-sample terms, updated parameters) go through
// L2 between cluster barriers, copied to shared memory asynchronously; the
// next step's samples are read ahead.  A step takes 7 us at batch 16 and 11 us
// at 256; training 2,000 samples for 30 epochs of batch 256 went from 37.4 to
// 3.3 ms, model creation and prediction included.
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
constexpr int kW2Threads = 256;    // one per W2 gradient of a CTA
constexpr int kStepThreads = kW2Threads + 64;  // and two warps for its other gradients
constexpr int kRow = H + 4;      // row stride of the tile's per-sample arrays (16-byte rows, no bank conflicts)
constexpr int kChunk = 256;      // samples whose terms are staged at a time
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

// Terms of the batch's samples in device memory, exchanged between the CTAs:
// rows of n_pad values (the batch rounded up to whole tiles), one per unit.
constexpr int TA1 = 0, TD2 = H, TD1 = 2 * H, TA2 = 3 * H, TX = 4 * H, TE = TX + IN, kTermRows = TE + 1;
// Rows that a CTA stages: 16 of a1 and of d2 for its W2 block; 4 of d1, d2 and
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
#pragma unroll 4
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

// Forward pass of a tile whose inputs are in t.x: a1, z2 and y, with the
// parameters w.  Called by the whole block (threads past kTileThreads only
// synchronise).
__device__ __forceinline__ void tile_forward(Tile &t, const float *w)
{
    const int s = threadIdx.x / 16 * 2, c = threadIdx.x % 16;
    const bool on = threadIdx.x < kTileThreads;
    float z[2][4];
    if (on) {
#pragma unroll
        for (int q = 0; q < 8; ++q) z[q / 4][q % 4] = w[OB1 + 4 * c + q % 4];
        dot24<IN>(z, t.x[s], t.x[s + 1], w + OW1, c);
#pragma unroll
        for (int q = 0; q < 8; ++q) t.a1[s + q / 4][4 * c + q % 4] = z[q / 4][q % 4] > 0.f ? z[q / 4][q % 4] : 0.f;
    }
    __syncthreads();
    if (on) {
#pragma unroll
        for (int q = 0; q < 8; ++q) z[q / 4][q % 4] = w[OB2 + 4 * c + q % 4];
        dot24<H>(z, t.a1[s], t.a1[s + 1], w + OW2, c);
#pragma unroll
        for (int q = 0; q < 8; ++q) t.z2[s + q / 4][4 * c + q % 4] = z[q / 4][q % 4];
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

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

struct StepArgs {
    const float *x, *t;        // all samples
    const uint32_t *idx;       // sample of every position (null: the position itself)
    const float *corr;         // Adam's bias corrections {c1, c2} per step
    float *P, *PT, *M, *V, *G; // parameters, W2 transposed, Adam's state, gradient
    float *loss_terms;         // squared error of every position
    float *terms;              // [kTermRows][n_pad]
    uint32_t n_pad;
    uint32_t n, batch;         // positions, positions per step
    float lr, b1, b2, eps;
};

// A thread's share of the gradient.  The CTA of rank r has W2 rows
// 16 (r / 4) .. + 15, columns 16 (r % 4) .. + 15 (one per thread), and, by two
// warps of their own, columns 4 r .. 4 r + 3 of W1, b1, b2 and w3, and b3 (rank 0).
struct Share {
    int p;    // parameter of this thread, -1 = none
    int u, v; // staged rows: its gradient is the sum over the samples of u[b] * v[b], v < 0: of u[b]
    bool gate; // only of the samples with v[b] > 0 (v is an activation)
};

__device__ __forceinline__ Share share_of(int rank, int tid)
{
    constexpr int SA1 = 0, SD2 = 16, SD1 = 32, SE2 = 36, SA2 = 40, SX = 44, SE = SX + IN;
    if (tid < kW2Threads) {
        const int i = tid / 16, j = tid % 16;
        return Share{OW2 + (16 * (rank / 4) + i) * H + 16 * (rank % 4) + j, SD2 + j, SA1 + i, true};
    }
    const int q = tid - kW2Threads, c = q % 4, col = 4 * rank + c;
    if (q < 4 * IN) return Share{OW1 + (q / 4) * H + col, SD1 + c, SX + q / 4, false};
    if (q < 4 * IN + 4) return Share{OB1 + col, SD1 + c, -1, false};
    if (q < 4 * IN + 8) return Share{OB2 + col, SE2 + c, -1, false};
    if (q < 4 * IN + 12) return Share{OW3 + col, SE, SA2 + c, true};
    if (q == 4 * IN + 12 && rank == 0) return Share{OB3, SE, -1, false};
    return Share{-1, 0, -1, false};
}

// The terms row that staged row r holds.
__device__ __forceinline__ int staged_row(int rank, int r)
{
    if (r < 16) return TA1 + 16 * (rank / 4) + r;
    if (r < 32) return TD2 + 16 * (rank % 4) + r - 16;
    if (r < 36) return TD1 + 4 * rank + r - 32;
    if (r < 40) return TD2 + 4 * rank + r - 36;
    if (r < 44) return TA2 + 4 * rank + r - 40;
    return TX + r - 44;  // x, then e
}

// TRAIN: one Adam step per batch of positions; otherwise the gradient of the
// first batch, into G.
template <bool TRAIN>
__global__ void __launch_bounds__(kStepThreads) k_mlp_steps(const StepArgs a, const __grid_constant__ Norm nm)
{
    extern __shared__ __align__(16) float smem[];
    float *w = smem;                     // parameters
    float *w2t = w + kParamsPadded;      // W2 transposed
    Tile &t = *reinterpret_cast<Tile *>(w2t + H * H);
    float *stage = w2t + H * H + sizeof(Tile) / 4;
    const int rank = blockIdx.x;  // one cluster
    const int tid = threadIdx.x;
    const uint64_t pol = l2_policy(0);

    const Share sh = share_of(rank, tid);
    float pP = 0.f, pM = 0.f, pV = 0.f;
    if (TRAIN && sh.p >= 0) {
        pP = a.P[sh.p];
        pM = a.M[sh.p];
        pV = a.V[sh.p];
    }
    const float *us = stage + sh.u * kChunkRow, *vs = stage + (sh.v < 0 ? 0 : sh.v) * kChunkRow;

    // Inputs and target of this thread in the CTA's first tile of a step
    // (sample tid / IN, input tid % IN; sample tid), read ahead of the step.
    const int xs = tid / IN, xk = tid % IN;
    uint32_t ix = 0, it = 0;  // their samples
    float xv = 0.f, tv = 0.f;
    auto ahead_index = [&](uint32_t b0) {
        const uint32_t bx = b0 + rank * kTile + xs, bt = b0 + rank * kTile + tid;
        if (tid < kTileThreads && bx < a.n) ix = a.idx ? a.idx[bx] : bx;
        if (tid < kTile && bt < a.n) it = a.idx ? a.idx[bt] : bt;
    };
    auto ahead_values = [&] {
        if (tid < kTileThreads) xv = a.x[(uint64_t)ix * IN + xk];
        if (tid < kTile) tv = a.t[it];
    };
    ahead_index(0);
    ahead_values();

    const uint32_t np = a.n_pad;
    for (uint32_t b0 = 0, step = 0; b0 < a.n; b0 += a.batch, ++step) {
        const uint32_t B = a.n - b0 < a.batch ? a.n - b0 : a.batch;
        const uint32_t tiles = (B + kTile - 1) / kTile;
        // W2 transposed is not needed before the backward pass
        copy_async(w, a.P, kParamsPadded, pol);
        asm volatile("cp.async.commit_group;" ::: "memory");
        copy_async(w2t, a.PT, H * H, pol);
        asm volatile("cp.async.commit_group;" ::: "memory");
        float c1 = 0.f, c2 = 0.f;
        if (TRAIN) {
            c1 = a.corr[2 * step];
            c2 = a.corr[2 * step + 1];
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        // ---- forward and backward of this CTA's tiles ----------------------------
        for (uint32_t tl = rank; tl < tiles; tl += kCluster) {
            const uint32_t t0 = tl * kTile;  // first sample within the batch
            if (tl != (uint32_t)rank) {
                const uint32_t bx = b0 + t0 + xs, bt = b0 + t0 + tid;
                if (tid < kTileThreads && bx < a.n) xv = a.x[(uint64_t)(a.idx ? a.idx[bx] : bx) * IN + xk];
                if (tid < kTile && bt < a.n) tv = a.t[a.idx ? a.idx[bt] : bt];
                __syncthreads();  // the tile before is done with t
            }
            if (tid < kTileThreads) t.x[xs][xk] = t0 + xs < B ? (xv - nm.mu[xk]) / nm.sd[xk] : 0.f;
            __syncthreads();
            tile_forward(t, w);
            if (tid < kTile) {
                const uint32_t b = t0 + tid;
                float eb = 0.f;
                if (b < B) {
                    const float tn = (tv - nm.tmu) / nm.tsd;
                    const float d = t.y[tid] - tn;
                    if (a.loss_terms) a.loss_terms[b0 + b] = d * d;
                    eb = 2.f * d / (float)B;
                }
                t.e[tid] = eb;
                __stcg(a.terms + (uint64_t)TE * np + t0 + tid, eb);
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            const int s = tid / 16 * 2, c = tid % 16;
            if (tid < kTileThreads) {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int r = s + q / 4, j = 4 * c + q % 4;
                    t.g2[r][j] = t.z2[r][j] > 0.f ? t.e[r] * w[OW3 + j] : 0.f;
                }
            }
            __syncthreads();
            if (tid < kTileThreads) {
                float g[2][4] = {};
                dot24<H>(g, t.g2[s], t.g2[s + 1], w2t, c);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int r = s + q / 4, i = 4 * c + q % 4;
                    const bool live = t0 + r < B;  // all terms of the samples past the batch are 0
                    const float a1 = t.a1[r][i], z2 = t.z2[r][i];
                    float *o = a.terms + (uint64_t)i * np + t0 + r;
                    __stcg(o + (uint64_t)TA1 * np, live ? a1 : 0.f);
                    __stcg(o + (uint64_t)TD1 * np, live && a1 > 0.f ? g[q / 4][q % 4] : 0.f);
                    __stcg(o + (uint64_t)TD2 * np, live ? t.g2[r][i] : 0.f);
                    __stcg(o + (uint64_t)TA2 * np, live && z2 > 0.f ? z2 : 0.f);
                }
                __stcg(a.terms + (uint64_t)(TX + xk) * np + t0 + xs, t.x[xs][xk]);
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        cluster_arrive();
        if (TRAIN) ahead_index(b0 + a.batch);
        cluster_wait();
        // ---- gradient of this CTA's share, samples in order -----------------------
        float acc = 0.f;
        for (uint32_t k0 = 0; k0 < tiles * kTile; k0 += kChunk) {
            const uint32_t left = tiles * kTile - k0, n = left < kChunk ? left : kChunk;
            if (k0) __syncthreads();  // the chunk before is summed
            for (uint32_t v = tid; v < kStageRows * (n / 4); v += blockDim.x) {
                const uint32_t r = v / (n / 4), q = 4 * (v - r * (n / 4));
                cp_async16(stage + r * kChunkRow + q, a.terms + (uint64_t)staged_row(rank, r) * np + k0 + q, pol);
            }
            if (TRAIN && !k0) ahead_values();
            cp_async_wait_all();
            __syncthreads();
            if (sh.p >= 0) {
                if (sh.v >= 0) {
#pragma unroll 4
                    for (uint32_t k = 0; k < n; k += 4) {
                        const float4 u = ld4(us + k), v = ld4(vs + k);
                        if (!sh.gate || v.x > 0.f) acc = fmaf(v.x, u.x, acc);
                        if (!sh.gate || v.y > 0.f) acc = fmaf(v.y, u.y, acc);
                        if (!sh.gate || v.z > 0.f) acc = fmaf(v.z, u.z, acc);
                        if (!sh.gate || v.w > 0.f) acc = fmaf(v.w, u.w, acc);
                    }
                } else {
#pragma unroll 4
                    for (uint32_t k = 0; k < n; k += 4) {
                        const float4 u = ld4(us + k);
                        acc += u.x;
                        acc += u.y;
                        acc += u.z;
                        acc += u.w;
                    }
                }
            }
        }
        if (!TRAIN) {
            if (sh.p >= 0) a.G[sh.p] = acc;
            break;
        }
        if (sh.p >= 0) {
            adam(pP, pM, pV, acc, a.lr, a.b1, a.b2, a.eps, c1, c2);
            __stcg(a.P + sh.p, pP);
            if (sh.p >= OW2 && sh.p < OB2) __stcg(a.PT + ((sh.p - OW2) % H) * H + (sh.p - OW2) / H, pP);
        }
        cluster_arrive();
        cluster_wait();
    }
    if (TRAIN && sh.p >= 0) {
        a.M[sh.p] = pM;
        a.V[sh.p] = pV;
    }
}

constexpr size_t kStepSmem = (kParamsPadded + H * H + kStageRows * kChunkRow) * 4 + sizeof(Tile);

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
    float *base = nullptr, *x = nullptr, *t = nullptr, *pt = nullptr, *lt = nullptr, *terms = nullptr;
    uint32_t n_pad = 0;
    cudaStream_t st;
    explicit MlpScratch(cudaStream_t s) : st(s) {}
    // N samples, batches of at most B, `loss` squared errors.
    cudaError_t alloc(uint64_t N, uint32_t B, uint64_t loss)
    {
        const uint64_t np = ((uint64_t)B + kTile - 1) / kTile * kTile;
        uint64_t at = 0;
        auto take = [&](uint64_t n) {
            const uint64_t o = at;
            at += (n + 3) & ~3ull;  // 16-byte rows
            return o;
        };
        const uint64_t ox = take(N * IN), ot = take(N), opt = take(H * H), olt = take(loss), otr = take(kTermRows * np);
        const cudaError_t e = cudaMallocAsync((void **)&base, at * 4, st);
        if (e != cudaSuccess) return e;
        x = base + ox;
        t = base + ot;
        pt = base + opt;
        lt = base + olt;
        terms = base + otr;
        n_pad = (uint32_t)np;
        return cudaSuccess;
    }
    ~MlpScratch()
    {
        if (base) cudaFreeAsync(base, st);
    }
};

// Launches k_mlp_steps as one cluster.
template <bool TRAIN> int launch_steps(const StepArgs &a, const Norm &nm, cudaStream_t st)
{
    const void *fn = (const void *)k_mlp_steps<TRAIN>;
    PTW_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStepSmem));
    PTW_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = kCluster;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kCluster);
    cfg.blockDim = dim3(kStepThreads);
    cfg.dynamicSmemBytes = kStepSmem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    PTW_CUDA(cudaLaunchKernelEx(&cfg, k_mlp_steps<TRAIN>, a, nm));
    return PTW_OK;
}

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
    PTW_CUDA(s.alloc(B, B, B));
    PTW_CUDA(cudaMemcpyAsync(s.x, h_x, (uint64_t)B * IN * 4, cudaMemcpyHostToDevice, st));
    PTW_CUDA(cudaMemcpyAsync(s.t, h_t, B * 4ull, cudaMemcpyHostToDevice, st));
    k_mlp_transpose<<<(H * H + 255) / 256, 256, 0, st>>>(m->params, s.pt);
    StepArgs a{};
    a.x = s.x;
    a.t = s.t;
    a.P = m->params;
    a.PT = s.pt;
    a.G = m->grad;
    a.loss_terms = s.lt;
    a.terms = s.terms;
    a.n_pad = s.n_pad;
    a.n = a.batch = B;
    const int rc = launch_steps<false>(a, host_norm(m), st);
    if (rc) return rc;
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
    PTW_CUDA(s.alloc(N, batch, (uint64_t)run * N));
    // Per epoch: the order of the samples and the steps' bias corrections.
    const uint64_t words = (uint64_t)N + 2ull * nb;
    uint32_t *d_plan = nullptr;
    PTW_CUDA(cudaMallocAsync((void **)&d_plan, words * 4, st));
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
    a.corr = reinterpret_cast<const float *>(d_plan + N);
    a.P = m->params;
    a.PT = s.pt;
    a.M = m->m;
    a.V = m->v;
    a.terms = s.terms;
    a.n_pad = s.n_pad;
    a.n = N;
    a.batch = batch;
    a.lr = lr;
    a.b1 = 0.9f;
    a.b2 = 0.999f;
    a.eps = 1e-8f;
    const Norm nm = host_norm(m);
    std::vector<uint32_t> plan(words);
    std::vector<float> lt((uint64_t)run * N);
    for (uint32_t i = 0; i < N; ++i) plan[i] = i;
    uint64_t rs = seed * 0x9E3779B97F4A7C15ull + 1;
    uint32_t ep0 = 0;  // first epoch whose squared errors are not copied yet
    for (uint32_t ep = 0; ep < epochs; ++ep) {
        for (uint32_t i = N - 1; i > 0; --i) {  // Fisher-Yates with an LCG
            rs = rs * 6364136223846793005ull + 1442695040888963407ull;
            std::swap(plan[i], plan[(rs >> 33) % (i + 1)]);
        }
        float *corr = reinterpret_cast<float *>(plan.data() + N);
        for (uint32_t k = 0; k < nb; ++k) {
            ++m->step;
            corr[2 * k] = 1.f - std::pow(a.b1, (float)m->step);
            corr[2 * k + 1] = 1.f - std::pow(a.b2, (float)m->step);
        }
        // (the copy has left `plan` when the call returns: pageable memory)
        PTW_CUDA(cudaMemcpyAsync(d_plan, plan.data(), words * 4, cudaMemcpyHostToDevice, st));
        a.loss_terms = run ? s.lt + (uint64_t)(ep - ep0) * N : nullptr;
        const int rc = launch_steps<true>(a, nm, st);
        if (rc) return rc;
        if (run && (ep + 1 == epochs || ep + 1 - ep0 == run)) {
            PTW_CUDA(cudaMemcpyAsync(lt.data(), s.lt, (uint64_t)(ep + 1 - ep0) * N * 4, cudaMemcpyDeviceToHost, st));
            PTW_CUDA(cudaStreamSynchronize(st));
            for (uint32_t e = ep0; e <= ep; ++e) {
                double loss = 0;
                for (uint32_t b0 = 0; b0 < N; b0 += batch)
                    loss += mean_loss(lt.data() + (uint64_t)(e - ep0) * N + b0, std::min(batch, N - b0));
                h_loss_curve[e] = (float)(loss / nb);
            }
            ep0 = ep + 1;
        }
    }
    PTW_CUDA(cudaStreamSynchronize(st));
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
