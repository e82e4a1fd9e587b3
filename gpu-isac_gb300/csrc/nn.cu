// nn.cu -- kernels of the learned reference proposal: rotation-invariant
// features from ring spectra, and the forward / backward / update steps of a
// small embedding network (dense layers, ReLU, row L2 normalisation, softmax
// cross-entropy over reference scores, Adam) plus per-row top-k.
//
// The network has no counterpart in the reference; it only decides which
// references the exhaustive search visits first.  All buffers are row-major
// FP32 device arrays owned by the caller; every entry point is asynchronous on
// the given stream.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/gpu_aln_pack.h"
#include "gpuisac_kernels.h"

namespace gpuisac {
namespace {

// ---------------------------------------------------------------- features
// feat[i][r*nk + k] = log(1 + |F_r[k]|) for k < nk (k = 0 from slot 0's F[0]),
// then the whole row scaled to unit L2 norm, then (when given) standardised
// per column, (v - mu[f]) * inv_sd[f].  Magnitudes of ring spectra do not
// change when the image turns (a circular shift of every ring) or is mirrored
// (conjugate spectra).
__global__ void features_kernel(const float2* __restrict__ sp, unsigned n, unsigned ring_num, unsigned nk,
                                const float* __restrict__ mu, const float* __restrict__ inv_sd,
                                float* __restrict__ feat)
{
    const unsigned i = blockIdx.x;
    if (i >= n)
        return;
    const unsigned nf = ring_num * nk;
    const float2* row = sp + (size_t)i * ring_num * kSlots;
    float* out = feat + (size_t)i * nf;
    float ss = 0.f;
    for (unsigned f = threadIdx.x; f < nf; f += blockDim.x) {
        const unsigned r = f / nk, k = f - r * nk;
        const float2 ab = row[r * kSlots + k];
        // stored basis (Re+Im, Re-Im); slot 0 holds (F[0], F[128])
        float re = 0.5f * (ab.x + ab.y), im = 0.5f * (ab.x - ab.y);
        if (k == 0)
            im = 0.f;
        const float v = log1pf(sqrtf(re * re + im * im));
        out[f] = v;
        ss += v * v;
    }
    __shared__ float red[32];
    for (int o = 16; o > 0; o >>= 1)
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x < 32) {
        float t = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
        for (int o = 16; o > 0; o >>= 1)
            t += __shfl_xor_sync(0xffffffffu, t, o);
        if (threadIdx.x == 0)
            red[0] = t;
    }
    __syncthreads();
    const float inv = rsqrtf(fmaxf(red[0], 1e-30f));
    if (mu) {
        for (unsigned f = threadIdx.x; f < nf; f += blockDim.x)
            out[f] = (out[f] * inv - mu[f]) * inv_sd[f];
    } else {
        for (unsigned f = threadIdx.x; f < nf; f += blockDim.x)
            out[f] *= inv;
    }
}

// ---------------------------------------------------------------- column statistics
// acc[2j], acc[2j+1] += sum, sum of squares of column j over a chunk of rows
__global__ void col_stats_kernel(const float* __restrict__ X, long rows, int cols, long rows_per_chunk,
                                 double* __restrict__ acc)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cols)
        return;
    const long r0 = (long)blockIdx.y * rows_per_chunk;
    const long r1 = min(rows, r0 + rows_per_chunk);
    double s = 0.0, ss = 0.0;
    for (long i = r0; i < r1; i++) {
        const double v = X[i * cols + j];
        s += v;
        ss += v * v;
    }
    atomicAdd(&acc[2 * j], s);
    atomicAdd(&acc[2 * j + 1], ss);
}

__global__ void col_stats_final_kernel(const double* __restrict__ acc, long rows, int cols, float eps,
                                       float* __restrict__ mean, float* __restrict__ inv_sd)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cols)
        return;
    const double m = acc[2 * j] / (double)rows;
    const double var = fmax(acc[2 * j + 1] / (double)rows - m * m, 0.0);
    mean[j] = (float)m;
    inv_sd[j] = (float)(1.0 / sqrt(var + (double)eps));
}

// X[i][j] = (X[i][j] - mu[j]) * inv_sd[j]
__global__ void affine_cols_kernel(float* __restrict__ X, long rows, int cols, const float* __restrict__ mu,
                                   const float* __restrict__ inv_sd)
{
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= rows * cols)
        return;
    const int j = (int)(idx % cols);
    X[idx] = (X[idx] - mu[j]) * inv_sd[j];
}

// out[i][j] = max over s < group of G[i*group + s][j]
__global__ void group_max_kernel(const float* __restrict__ G, long n, int group, int cols, float* __restrict__ out)
{
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n * cols)
        return;
    const long i = idx / cols;
    const int j = (int)(idx - i * cols);
    const float* g = G + (i * group) * cols + j;
    float m = g[0];
    for (int s = 1; s < group; s++)
        m = fmaxf(m, g[(long)s * cols]);
    out[idx] = m;
}

// ---------------------------------------------------------------- GEMM
// C[m][n] = alpha * sum_k A(m,k) B(k,n) + beta * C[m][n], with A(m,k) at
// A[m*sam + k*sak] and B(k,n) at B[k*sbk + n*sbn] (strides give transposes).
// A launch runs up to kMaxProblems of them (tiles numbered through), each with
// an optional second product added to it (a weight's gradient from particles
// and references), bias + ReLU or a ReLU mask.  Every output is summed by one
// thread in the order of k.
//
// What bounds it: the network's products are small (500 x 256 x 560 at most in
// a training step of 500 particles and 200 references), so the time is the
// latency of one tile's K loop.  64 x 64 tiles over 8 to 32 CTAs, loading each
// K step of 16 between two barriers, took 44 us a product, 573 of a step's 640
// us on the device; 32 x 32 tiles with the next 64 of K in flight, and
// independent products sharing a launch, take 91 of 102 us (15 us a launch; 27
// with 128 threads a tile and the operand's layout told apart at every load).
// Products with at least one 64 x 64 tile per SM keep that tile (half the
// loads per FMA).
constexpr int kMaxProblems = 4;
struct GemmPart {
    const float *A, *B;
    long sam, sak, sbk, sbn;
    int K;
};
struct GemmProblem {
    int M, N;
    float alpha, beta;
    GemmPart part[2]; // (part[1].K = 0: none)
    float* C;
    long ldc;
    const float* bias; // added per column, then ReLU if relu; or null
    int relu;
    const float* mask; // zero C where mask[m * ldc + n] is not positive; or null
    int tiles_n, tile_begin;
};
// sums of columns: db[j] = sum_i dY[i][j] (+ the same of dY2), by the last CTAs
struct ColSum {
    const float *dY, *dY2;
    long rows, rows2;
    int cols;
    float* db;
};
struct GemmGroup {
    GemmProblem p[kMaxProblems];
    int n, tiles;
    ColSum cs[2];
};

// sum of a column in row order (16 loads in flight)
__device__ __forceinline__ float col_sum(const float* __restrict__ dY, long rows, int cols, int j)
{
    float s = 0.f;
#pragma unroll 16
    for (long i = 0; i < rows; i++)
        s += dY[i * cols + j];
    return s;
}

// One operand's loads of a K step: T outer indices (rows of A, columns of B) x
// TK of k by 256 threads, kN each, along the operand's unit-stride dimension:
// k fastest (kK: a warp reads 8 k of 4 outer indices, whole sectors) or the
// outer index fastest (32 in a row).  No two lanes of a warp store to one bank
// of s[k][outer] (row length T + 4).
template <int T, int TK, bool kK>
struct GemmLoad {
    static constexpr int kN = T * TK / 256;
    static constexpr int kOuter = kK ? T / 32 : 1, kPer = kN / kOuter;
    const float* p[kOuter];
    bool in[kOuter];
    long step_k; // between the thread's successive k
    int o0, kk0, K;
    __device__ __forceinline__ GemmLoad(const float* base, long so, long sk, int first, int n, int k_count)
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        if (kK) {
            o0 = (lane >> 3) + 4 * warp;
            kk0 = lane & 7;
        } else {
            constexpr int kStrips = T / 32; // warps side by side
            o0 = lane + 32 * (warp % kStrips);
            kk0 = warp / kStrips;
        }
        K = k_count;
        step_k = sk;
#pragma unroll
        for (int j = 0; j < kOuter; j++) {
            in[j] = first + o0 + 32 * j < n;
            p[j] = base + (in[j] ? (long)(first + o0 + 32 * j) * so + (long)kk0 * sk : 0);
        }
    }
    static constexpr int kStep = kK ? 8 : 8 / (T / 32); // k between a thread's loads
    __device__ __forceinline__ void fetch(float (&r)[kN], int k0) const
    {
#pragma unroll
        for (int j = 0; j < kOuter; j++)
#pragma unroll
            for (int i = 0; i < kPer; i++)
                r[j * kPer + i] =
                    in[j] && k0 + kk0 + kStep * i < K ? __ldg(p[j] + (long)(k0 + kStep * i) * (kK ? 1 : step_k)) : 0.f;
    }
    __device__ __forceinline__ void store(const float (&r)[kN], float (*s)[T + 4]) const
    {
#pragma unroll
        for (int j = 0; j < kOuter; j++)
#pragma unroll
            for (int i = 0; i < kPer; i++)
                s[kk0 + kStep * i][o0 + 32 * j] = r[j * kPer + i];
    }
};

// one product of a tile, added to acc
template <int T, int TK, bool kA, bool kB>
__device__ __forceinline__ void gemm_part(const GemmPart& q, int m0, int M, int n0, int N, float (*As)[TK][T + 4],
                                          float (*Bs)[TK][T + 4], float (&acc)[T / 16][T / 16])
{
    constexpr int U = T / 16; // outputs per thread and dimension
    const GemmLoad<T, TK, kA> la(q.A, q.sam, q.sak, m0, M, q.K);
    const GemmLoad<T, TK, kB> lb(q.B, q.sbn, q.sbk, n0, N, q.K);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float ra[la.kN], rb[lb.kN];
    la.fetch(ra, 0);
    lb.fetch(rb, 0);
    int buf = 0;
    __syncthreads(); // (a previous product's last readers)
    for (int k0 = 0; k0 < q.K; k0 += TK, buf ^= 1) {
        la.store(ra, As[buf]);
        lb.store(rb, Bs[buf]);
        __syncthreads(); // (the other buffer's readers passed the barrier before)
        if (k0 + TK < q.K) {
            la.fetch(ra, k0 + TK);
            lb.fetch(rb, k0 + TK);
        }
#pragma unroll 8
        for (int kk = 0; kk < TK; kk++) {
            float a[U], b[U];
#pragma unroll
            for (int i = 0; i < U; i++) {
                a[i] = As[buf][kk][ty * U + i];
                b[i] = Bs[buf][kk][tx * U + i];
            }
#pragma unroll
            for (int i = 0; i < U; i++)
#pragma unroll
                for (int j = 0; j < U; j++)
                    acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
    }
}

// tiles of T x T, 256 threads
template <int T, int TK>
__global__ void __launch_bounds__(256) gemm_kernel(const __grid_constant__ GemmGroup g)
{
    constexpr int U = T / 16;
    __shared__ __align__(16) float As[2][TK][T + 4];
    __shared__ __align__(16) float Bs[2][TK][T + 4];
    const int tid = threadIdx.x;
    const int tile = blockIdx.x;
    if (tile >= g.tiles) { // column sums, 32 columns per CTA (its first warp)
        int j = (tile - g.tiles) * 32 + tid;
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const ColSum& cs = g.cs[c];
            if (tid < 32 && j >= 0 && j < cs.cols) {
                const float s1 = col_sum(cs.dY, cs.rows, cs.cols, j);
                cs.db[j] = cs.dY2 ? s1 + col_sum(cs.dY2, cs.rows2, cs.cols, j) : s1;
            }
            j -= (cs.cols + 31) / 32 * 32;
        }
        return;
    }
    int pi = 0;
    while (pi + 1 < g.n && g.p[pi + 1].tile_begin <= tile)
        pi++;
    const GemmProblem& p = g.p[pi];
    const int lt = tile - p.tile_begin;
    const int m0 = lt / p.tiles_n * T, n0 = lt % p.tiles_n * T;
    const int tx = tid & 15, ty = tid >> 4;
    float acc[U][U], prev[U][U];
#pragma unroll
    for (int i = 0; i < U; i++)
#pragma unroll
        for (int j = 0; j < U; j++)
            acc[i][j] = prev[i][j] = 0.f;
    const int n_parts = p.part[1].K > 0 ? 2 : 1;
    for (int h = 0; h < n_parts; h++) {
        const GemmPart& q = p.part[h];
        if (h == 1) { // the first product is complete
#pragma unroll
            for (int i = 0; i < U; i++)
#pragma unroll
                for (int j = 0; j < U; j++) {
                    prev[i][j] = p.alpha * acc[i][j];
                    acc[i][j] = 0.f;
                }
        }
        if (q.sak == 1) {
            if (q.sbk == 1)
                gemm_part<T, TK, true, true>(q, m0, p.M, n0, p.N, As, Bs, acc);
            else
                gemm_part<T, TK, true, false>(q, m0, p.M, n0, p.N, As, Bs, acc);
        } else {
            if (q.sbk == 1)
                gemm_part<T, TK, false, true>(q, m0, p.M, n0, p.N, As, Bs, acc);
            else
                gemm_part<T, TK, false, false>(q, m0, p.M, n0, p.N, As, Bs, acc);
        }
    }
#pragma unroll
    for (int i = 0; i < U; i++) {
        const int gm = m0 + ty * U + i;
        if (gm >= p.M)
            continue;
#pragma unroll
        for (int j = 0; j < U; j++) {
            const int gn = n0 + tx * U + j;
            if (gn >= p.N)
                continue;
            float* c = p.C + (long)gm * p.ldc + gn;
            float v = p.alpha * acc[i][j] + (n_parts == 2 ? prev[i][j] : p.beta != 0.f ? p.beta * *c : 0.f);
            if (p.bias) {
                v = v + p.bias[gn];
                v = p.relu ? fmaxf(v, 0.f) : v;
            }
            if (p.mask && !(p.mask[(long)gm * p.ldc + gn] > 0.f))
                v = 0.f;
            *c = v;
        }
    }
}

// One product with a short K and nothing added: 64 x 64 tiles, K steps of 16 through one
// buffer, 4 x 4 outputs per thread, the same order of k.  There is no K loop to hide
// behind, so what counts is how many tiles an SM has at a time: 48 registers and 9 KB
// against 80 and 35, and no zeros summed up to a step of 32 or 64.
constexpr int kShortT = 64, kShortK = 16;

__global__ void __launch_bounds__(256)
gemm_short_kernel(int M, int N, int K, float alpha, const float* __restrict__ A, long sam, long sak,
                  const float* __restrict__ B, long sbk, long sbn, float beta, float* __restrict__ C, long ldc)
{
    __shared__ float As[kShortK][kShortT + 4];
    __shared__ float Bs[kShortK][kShortT + 4];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int m0 = (int)blockIdx.y * kShortT, n0 = (int)blockIdx.x * kShortT;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < K; k0 += kShortK) {
        for (int e = threadIdx.x; e < kShortK * kShortT; e += 256) {
            const int kk = e / kShortT, o = e % kShortT, gk = k0 + kk;
            As[kk][o] = m0 + o < M && gk < K ? A[(long)(m0 + o) * sam + (long)gk * sak] : 0.f;
        }
        for (int e = threadIdx.x; e < kShortK * kShortT; e += 256) {
            const int kk = e / kShortT, o = e % kShortT, gk = k0 + kk;
            Bs[kk][o] = n0 + o < N && gk < K ? B[(long)gk * sbk + (long)(n0 + o) * sbn] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kShortK; kk++) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                a[i] = As[kk][ty * 4 + i];
                b[i] = Bs[kk][tx * 4 + i];
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++)
                    acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= M)
            continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int gn = n0 + tx * 4 + j;
            if (gn >= N)
                continue;
            float* c = C + (long)gm * ldc + gn;
            *c = alpha * acc[i][j] + (beta != 0.f ? beta * *c : 0.f);
        }
    }
}

// ---------------------------------------------------------------- elementwise
// Y[i][j] += b[j]; optionally ReLU
__global__ void bias_act_kernel(float* __restrict__ Y, const float* __restrict__ b, long rows, int cols, int relu)
{
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= rows * cols)
        return;
    float v = Y[idx] + b[idx % cols];
    Y[idx] = relu ? fmaxf(v, 0.f) : v;
}

// dY *= (Y > 0)
__global__ void relu_bwd_kernel(float* __restrict__ dY, const float* __restrict__ Y, long n)
{
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < n && !(Y[idx] > 0.f))
        dY[idx] = 0.f;
}

// db[j] = sum_i dY[i][j] (added to db when accumulate)
__global__ void colsum_kernel(const float* __restrict__ dY, long rows, int cols, float* __restrict__ db,
                              int accumulate)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cols)
        return;
    const float s = col_sum(dY, rows, cols, j);
    db[j] = accumulate ? db[j] + s : s;
}

// one warp per row: E = X / |X| (norm stored)
__global__ void l2norm_kernel(const float* __restrict__ X, long rows, int cols, float* __restrict__ E,
                              float* __restrict__ norm)
{
    const long r = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= rows)
        return;
    float ss = 0.f;
    for (int j = lane; j < cols; j += 32) {
        const float v = X[r * cols + j];
        ss += v * v;
    }
    for (int o = 16; o > 0; o >>= 1)
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float nr = sqrtf(fmaxf(ss, 1e-24f));
    for (int j = lane; j < cols; j += 32)
        E[r * cols + j] = X[r * cols + j] / nr;
    if (lane == 0)
        norm[r] = nr;
}

// dX = (dE - E (E . dE)) / norm
__global__ void l2norm_bwd_kernel(const float* __restrict__ E, const float* __restrict__ dE,
                                  const float* __restrict__ norm, long rows, int cols, float* __restrict__ dX)
{
    const long r = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= rows)
        return;
    float dot = 0.f;
    for (int j = lane; j < cols; j += 32)
        dot += E[r * cols + j] * dE[r * cols + j];
    for (int o = 16; o > 0; o >>= 1)
        dot += __shfl_xor_sync(0xffffffffu, dot, o);
    const float inv = 1.f / norm[r];
    for (int j = lane; j < cols; j += 32)
        dX[r * cols + j] = (dE[r * cols + j] - E[r * cols + j] * dot) * inv;
}

// one warp per row: softmax over the row's scores, cross-entropy against the
// label; dS = (softmax - onehot) / rows when dS is given
__global__ void softmax_xent_kernel(const float* __restrict__ S, const int* __restrict__ labels, long rows, int cols,
                                    float* __restrict__ loss, float* __restrict__ dS)
{
    const long r = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= rows)
        return;
    const float* s = S + r * cols;
    float mx = -INFINITY;
    for (int j = lane; j < cols; j += 32)
        mx = fmaxf(mx, s[j]);
    for (int o = 16; o > 0; o >>= 1)
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float se = 0.f;
    for (int j = lane; j < cols; j += 32)
        se += expf(s[j] - mx);
    for (int o = 16; o > 0; o >>= 1)
        se += __shfl_xor_sync(0xffffffffu, se, o);
    const int lab = labels[r];
    if (lane == 0)
        loss[r] = logf(se) + mx - s[lab];
    if (dS) {
        const float inv = 1.f / (se * (float)rows);
        for (int j = lane; j < cols; j += 32)
            dS[r * cols + j] = expf(s[j] - mx) * inv - (j == lab ? 1.f / (float)rows : 0.f);
    }
}

// AdamW step on n parameters (step counts from 1)
__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, long n, float lr, float b1, float b2, float eps, float wd, float c1,
                            float c2)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * ((mi / c1) / (sqrtf(vi / c2) + eps) + wd * p[i]);
}

// one warp per row: indices of the k largest scores, best first (ties: the
// smaller index); cols <= 1024, k <= 64
__global__ void topk_kernel(const float* __restrict__ S, long rows, int cols, int k, unsigned* __restrict__ idx)
{
    const long r = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= rows)
        return;
    const float* s = S + r * cols;
    unsigned taken = 0; // bit t: column lane + 32 t already chosen
    for (int pick = 0; pick < k; pick++) {
        float bv = -INFINITY;
        int bj = 0x7fffffff;
        for (int t = 0; t < 32; t++) {
            const int j = lane + 32 * t;
            if (j >= cols)
                break;
            if (taken & (1u << t))
                continue;
            const float v = s[j];
            if (v > bv || (v == bv && j < bj) || bj == 0x7fffffff) {
                bv = v;
                bj = j;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oj = __shfl_xor_sync(0xffffffffu, bj, o);
            if (oj != 0x7fffffff && (bj == 0x7fffffff || ov > bv || (ov == bv && oj < bj))) {
                bv = ov;
                bj = oj;
            }
        }
        if (bj == 0x7fffffff)
            bj = 0;
        if ((bj & 31) == lane)
            taken |= 1u << (bj >> 5);
        if (lane == 0)
            idx[r * k + pick] = (unsigned)bj;
    }
}

inline unsigned blocks(long n, int per) { return (unsigned)((n + per - 1) / per); }

int device_sms()
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

// numbers the tiles of g's problems and launches them with its column sums
cudaError_t launch_gemms(GemmGroup& g, cudaStream_t st)
{
    auto count = [&](int t) {
        long tiles = 0;
        for (int i = 0; i < g.n; i++) {
            GemmProblem& p = g.p[i];
            p.tiles_n = (p.N + t - 1) / t;
            p.tile_begin = (int)tiles;
            tiles += (long)p.tiles_n * ((p.M + t - 1) / t);
        }
        return tiles;
    };
    int t = 64;
    long tiles = count(t);
    // A product by itself with a short K: us here / in 64 x 64 tiles with two buffers,
    // columns x K at 300,000 rows: 8 x 8 37 / 82, 200 x 16 164 / 290, 64 x 24 66 / 83,
    // 64 x 32 114 / 89, 8 x 32 81 / 84, 64 x 40 94 / 118 (of its second 32 most are zeros),
    // 8 x 48 91 / 113, 200 x 48 402 / 421, 8 x 64 142 / 118; small products to K = 16 13.9 /
    // 15.0, 500 x 200 x 24 16.4 / 15.0.
    const GemmProblem& p0 = g.p[0];
    const int K = p0.part[0].K;
    const bool plain = g.n == 1 && p0.part[1].K == 0 && !p0.bias && !p0.mask && !g.cs[0].dY && !g.cs[1].dY;
    const int rows = (p0.M + kShortT - 1) / kShortT;
    if (plain && rows <= 65535 &&
        (K <= 16 || (tiles >= device_sms() && (K <= 24 || (K <= 48 && (K > 32 || p0.N <= 32)))))) {
        const GemmPart& q = p0.part[0];
        gemm_short_kernel<<<dim3((unsigned)p0.tiles_n, (unsigned)rows), 256, 0, st>>>(
            p0.M, p0.N, K, p0.alpha, q.A, q.sam, q.sak, q.B, q.sbk, q.sbn, p0.beta, p0.C, p0.ldc);
        g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
        return cudaGetLastError();
    }
    if (tiles < device_sms())
        tiles = count(t = 32);
    long grid = tiles;
    for (const ColSum& c : g.cs)
        grid += (c.cols + 31) / 32;
    if (grid > 0x7FFFFFFFl)
        return cudaErrorInvalidValue;
    g.tiles = (int)tiles;
    if (t == 64)
        gemm_kernel<64, 32><<<(unsigned)grid, 256, 0, st>>>(g);
    else
        gemm_kernel<32, 64><<<(unsigned)grid, 256, 0, st>>>(g);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError();
}

GemmProblem gemm_problem(int M, int N, int K, float alpha, const float* A, long sam, long sak, const float* B, long sbk,
                         long sbn, float beta, float* C, long ldc)
{
    GemmProblem p{};
    p.M = M;
    p.N = N;
    p.alpha = alpha;
    p.beta = beta;
    p.part[0] = GemmPart{A, B, sam, sak, sbk, sbn, K};
    p.C = C;
    p.ldc = ldc;
    return p;
}

} // namespace
} // namespace gpuisac

using namespace gpuisac;

// ============================================================ C-ABI
extern "C" {

int gpuisac_nn_features(const float* spectra, unsigned int n, unsigned int ring_num, unsigned int nk,
                        const float* mu, const float* inv_sd, float* feat, void* stream)
{
    if (!spectra || !feat || nk == 0 || nk > kSlots || ring_num == 0 || (!mu) != (!inv_sd))
        return 2;
    if (n == 0)
        return 0;
    features_kernel<<<n, 256, 0, (cudaStream_t)stream>>>(reinterpret_cast<const float2*>(spectra), n, ring_num, nk,
                                                          mu, inv_sd, feat);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

int gpuisac_nn_gemm(int M, int N, int K, float alpha, const float* A, long sam, long sak, const float* B, long sbk,
                    long sbn, float beta, float* C, long ldc, void* stream)
{
    if (M < 0 || N < 0 || K < 0 || !A || !B || !C)
        return 2;
    if (M == 0 || N == 0)
        return 0;
    GemmGroup g{};
    g.n = 1;
    g.p[0] = gemm_problem(M, N, K, alpha, A, sam, sak, B, sbk, sbn, beta, C, ldc);
    return launch_gemms(g, (cudaStream_t)stream) == cudaSuccess ? 0 : 1;
}

// One training batch: the forward pass of particles and references, the
// cross-entropy of their scores and its gradient.  Independent products of
// particles and references share launches: nine kernels.
int gpuisac_nn_loss_grad(const GpuisacNnTrain* t, void* stream)
{
    if (!t || !t->Xp || !t->Xr || !t->labels || !t->params || !t->grad || !t->loss || !t->work || t->n_in <= 0 ||
        t->hidden <= 0 || t->emb <= 0 || t->n_part <= 0 || t->n_ref <= 0)
        return 2;
    cudaStream_t st = (cudaStream_t)stream;
    const int P = t->n_part, R = t->n_ref, I = t->n_in, H = t->hidden, E = t->emb;
    const float *W1 = t->params, *b1 = W1 + (size_t)H * I, *W2 = b1 + H, *b2 = W2 + (size_t)E * H;
    float *gW1 = t->grad, *gb1 = gW1 + (size_t)H * I, *gW2 = gb1 + H, *gb2 = gW2 + (size_t)E * H;
    // rows of particles, then of references (one normalisation launch for both)
    const size_t n = (size_t)P + R;
    float* w = t->work;
    auto take = [&](size_t k) {
        float* r = w;
        w += k;
        return r;
    };
    float *Hb = take(n * H), *Z = take(n * E), *Eb = take(n * E), *nrm = take(n), *S = take((size_t)P * R),
          *dS = take((size_t)P * R), *dE = take(n * E), *dZ = take(n * E), *dH = take(n * H);
    const size_t rH = (size_t)P * H, rE = (size_t)P * E;
    GemmGroup g{};
    auto dense = [&](const float* X, int rows, int k, const float* W, int out, const float* b, int relu, float* Y) {
        GemmProblem p = gemm_problem(rows, out, k, 1.f, X, k, 1, W, 1, k, 0.f, Y, out);
        p.bias = b;
        p.relu = relu;
        return p;
    };
    // H = relu(X W1^T + b1), Z = H W2^T + b2, E = Z / |Z|
    g.n = 2;
    g.p[0] = dense(t->Xp, P, I, W1, H, b1, 1, Hb);
    g.p[1] = dense(t->Xr, R, I, W1, H, b1, 1, Hb + rH);
    if (launch_gemms(g, st) != cudaSuccess)
        return 1;
    g = GemmGroup{};
    g.n = 1;
    g.p[0] = dense(Hb, (int)n, H, W2, E, b2, 0, Z);
    if (launch_gemms(g, st) != cudaSuccess)
        return 1;
    l2norm_kernel<<<blocks((long)n, 8), 256, 0, st>>>(Z, (long)n, E, Eb, nrm);
    // S = scale Ep Er^T, its cross-entropy and dS
    g = GemmGroup{};
    g.n = 1;
    g.p[0] = gemm_problem(P, R, E, t->scale, Eb, E, 1, Eb + rE, 1, E, 0.f, S, R);
    if (launch_gemms(g, st) != cudaSuccess)
        return 1;
    softmax_xent_kernel<<<blocks(P, 8), 256, 0, st>>>(S, t->labels, P, R, t->loss, dS);
    // dEp = scale dS Er, dEr = scale dS^T Ep
    g = GemmGroup{};
    g.n = 2;
    g.p[0] = gemm_problem(P, E, R, t->scale, dS, R, 1, Eb + rE, E, 1, 0.f, dE, E);
    g.p[1] = gemm_problem(R, E, P, t->scale, dS, 1, R, Eb, E, 1, 0.f, dE + rE, E);
    if (launch_gemms(g, st) != cudaSuccess)
        return 1;
    l2norm_bwd_kernel<<<blocks((long)n, 8), 256, 0, st>>>(Eb, dE, nrm, (long)n, E, dZ);
    // dH = dZ W2 where H > 0; gW2 = dZ^T H, particles then references
    g = GemmGroup{};
    g.n = 2;
    g.p[0] = gemm_problem((int)n, H, E, 1.f, dZ, E, 1, W2, H, 1, 0.f, dH, H);
    g.p[0].mask = Hb;
    g.p[1] = gemm_problem(E, H, P, 1.f, dZ, 1, E, Hb, H, 1, 0.f, gW2, H);
    g.p[1].part[1] = GemmPart{dZ + rE, Hb + rH, 1, E, H, 1, R};
    g.cs[0] = ColSum{dZ, dZ + rE, P, R, E, gb2};
    if (launch_gemms(g, st) != cudaSuccess)
        return 1;
    g = GemmGroup{};
    g.n = 1;
    g.p[0] = gemm_problem(H, I, P, 1.f, dH, 1, H, t->Xp, I, 1, 0.f, gW1, I);
    g.p[0].part[1] = GemmPart{dH + rH, t->Xr, 1, H, I, 1, R};
    g.cs[0] = ColSum{dH, dH + rH, P, R, H, gb1};
    if (launch_gemms(g, st) != cudaSuccess)
        return 1;
    g_kernel_launches.fetch_add(3, std::memory_order_relaxed);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

int gpuisac_nn_bias_act(float* Y, const float* b, long rows, int cols, int relu, void* stream)
{
    if (!Y || !b || rows < 0 || cols <= 0)
        return 2;
    if (rows == 0)
        return 0;
    bias_act_kernel<<<blocks(rows * cols, 256), 256, 0, (cudaStream_t)stream>>>(Y, b, rows, cols, relu);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

int gpuisac_nn_relu_backward(float* dY, const float* Y, long n, void* stream)
{
    if (!dY || !Y || n < 0)
        return 2;
    if (n == 0)
        return 0;
    relu_bwd_kernel<<<blocks(n, 256), 256, 0, (cudaStream_t)stream>>>(dY, Y, n);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

int gpuisac_nn_colsum(const float* dY, long rows, int cols, float* db, int accumulate, void* stream)
{
    if (!dY || !db || rows < 0 || cols <= 0)
        return 2;
    colsum_kernel<<<blocks(cols, 32), 32, 0, (cudaStream_t)stream>>>(dY, rows, cols, db, accumulate);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

int gpuisac_nn_l2norm(const float* X, long rows, int cols, float* E, float* norm, void* stream)
{
    if (!X || !E || !norm || rows < 0 || cols <= 0)
        return 2;
    if (rows == 0)
        return 0;
    l2norm_kernel<<<blocks(rows, 8), 256, 0, (cudaStream_t)stream>>>(X, rows, cols, E, norm);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

int gpuisac_nn_l2norm_backward(const float* E, const float* dE, const float* norm, long rows, int cols, float* dX,
                               void* stream)
{
    if (!E || !dE || !norm || !dX || rows < 0 || cols <= 0)
        return 2;
    if (rows == 0)
        return 0;
    l2norm_bwd_kernel<<<blocks(rows, 8), 256, 0, (cudaStream_t)stream>>>(E, dE, norm, rows, cols, dX);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

int gpuisac_nn_softmax_xent(const float* S, const int* labels, long rows, int cols, float* loss, float* dS,
                            void* stream)
{
    if (!S || !labels || !loss || rows < 0 || cols <= 0)
        return 2;
    if (rows == 0)
        return 0;
    softmax_xent_kernel<<<blocks(rows, 8), 256, 0, (cudaStream_t)stream>>>(S, labels, rows, cols, loss, dS);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

int gpuisac_nn_adam(float* p, const float* g, float* m, float* v, long n, float lr, float b1, float b2, float eps,
                    float wd, int step, void* stream)
{
    if (!p || !g || !m || !v || n < 0 || step < 1)
        return 2;
    if (n == 0)
        return 0;
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    adam_kernel<<<blocks(n, 256), 256, 0, (cudaStream_t)stream>>>(p, g, m, v, n, lr, b1, b2, eps, wd, c1, c2);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

int gpuisac_nn_topk(const float* S, long rows, int cols, int k, unsigned int* idx, void* stream)
{
    if (!S || !idx || rows < 0 || cols <= 0 || cols > 1024 || k <= 0 || k > 64 || k > cols)
        return 2;
    if (rows == 0)
        return 0;
    topk_kernel<<<blocks(rows, 8), 256, 0, (cudaStream_t)stream>>>(S, rows, cols, k, idx);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

int gpuisac_nn_col_stats(const float* X, long rows, int cols, float eps, float* mean, float* inv_sd, void* stream)
{
    if (!X || !mean || !inv_sd || rows <= 0 || cols <= 0)
        return 2;
    cudaStream_t st = (cudaStream_t)stream;
    double* acc = nullptr;
    if (cudaMallocAsync(&acc, 2 * (size_t)cols * sizeof(double), st) != cudaSuccess)
        return 1;
    cudaMemsetAsync(acc, 0, 2 * (size_t)cols * sizeof(double), st);
    const long chunk = 512;
    dim3 grid(blocks(cols, 128), (unsigned)((rows + chunk - 1) / chunk));
    col_stats_kernel<<<grid, 128, 0, st>>>(X, rows, cols, chunk, acc);
    col_stats_final_kernel<<<blocks(cols, 128), 128, 0, st>>>(acc, rows, cols, eps, mean, inv_sd);
    g_kernel_launches.fetch_add(2, std::memory_order_relaxed);
    cudaFreeAsync(acc, st);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

int gpuisac_nn_affine_cols(float* X, long rows, int cols, const float* mu, const float* inv_sd, void* stream)
{
    if (!X || !mu || !inv_sd || rows < 0 || cols <= 0)
        return 2;
    if (rows == 0)
        return 0;
    affine_cols_kernel<<<blocks(rows * cols, 256), 256, 0, (cudaStream_t)stream>>>(X, rows, cols, mu, inv_sd);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

int gpuisac_nn_group_max(const float* G, long n, int group, int cols, float* out, void* stream)
{
    if (!G || !out || n < 0 || group <= 0 || cols <= 0)
        return 2;
    if (n == 0)
        return 0;
    group_max_kernel<<<blocks(n * cols, 256), 256, 0, (cudaStream_t)stream>>>(G, n, group, cols, out);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

} // extern "C"
