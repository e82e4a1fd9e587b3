// averages.cu -- the averaging step of ISAC's main iteration, after the
// equal-size group assignment (bin/sp_isac2_gpu.py:1153-1234): every particle
// rot_shift2D'd by the alignment parameters of its pair with its group's
// reference and added to the group's sum; the groups' mean shifts; every
// particle's parameters re-centred by them; each sum times 1/members,
// low-passed (filt_tanl) and moved by minus its mean shift (fshift).  The
// reference runs these steps on the host through EMAN2 (not part of the
// reference tree): rot_shift2D with its default quadratic interpolation in
// "background" mode and the x-mirror after it, add_img, mul_scalar,
// filt_tanl, fshift; the caller's conversion of the peak parameters
// (:1015-1022) comes first.
//
// Kernels, in stream order:
//  1. avg_count_kernel       members per (chunk of 1024 particles, group)
//  2. avg_chunk_scan_kernel  per group: exclusive offsets over the chunks
//  3. avg_group_scan_kernel  per group: first member, first piece, totals
//  4. avg_convert_kernel     thread per particle: its converted parameters
//  5. avg_scatter_kernel     stable counting sort: each group's members in
//                            particle order
//  6. avg_shift_kernel       one warp per group: mean shifts, parameters
//  7. avg_sum_kernel         one CTA per piece (a run of one group's members):
//                            each member image staged in shared memory by bulk
//                            copies (two buffers), every thread one column of
//                            two halves of the output, the quadratic
//                            interpolation from shared memory, FP32 sums in
//                            registers, one partial image per piece
//  8. avg_mean_kernel        each group's pieces summed in order, times
//                            float(1/members)
//  9. avg_rows_kernel, avg_cols_kernel, avg_inverse_kernel
//                            with a filter or centring: real 2D DFT, filter
//                            and phase shift, inverse DFT
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <mutex>
#include <vector>

#include "../../include/gpu_aln_pack.h"
#include "ccf_device.cuh"
#include "gpuisac_kernels.h"
#include "host_geometry.h"

namespace gpuisac {
namespace {

constexpr unsigned kAvgChunk = 1024;      // particles per counting-sort chunk
constexpr unsigned kSmemGroups = 16384;   // scatter: a chunk's group offsets in shared memory up to this
constexpr unsigned kMaxDim = 256;         // image side limit
constexpr unsigned kMinPiece = 2, kMaxPiece = 256; // members of a piece
constexpr unsigned kStagedMaxDim = 160;   // member images staged in shared memory (two buffers) up to this
constexpr double kPi = 3.141592653589793;

// error words: [0] belongsto entries outside [0, n_class), [1] the first such
// particle, [2] empty groups, [3] the first empty group, [4] bulk-copy waits
// that ran out
enum { kErrBad = 0, kErrBadFirst, kErrEmpty, kErrEmptyFirst, kErrWait, kErrWords };

// one member of a group, in the group's particle order (32 bytes)
struct AvgMember {
    float c, s;   // cos, sin of the angle (FP64 values rounded to float)
    float sx, sy; // the caller's converted shift, float as its peak_list
    float ang;
    unsigned img;
    unsigned mirror;
    unsigned pad;
};

__global__ void __launch_bounds__(256)
avg_count_kernel(const int* __restrict__ bel, unsigned P, unsigned R, unsigned* __restrict__ cnt,
                 unsigned* __restrict__ err)
{
    const unsigned c = blockIdx.x;
    const unsigned i1 = min(P, (c + 1) * kAvgChunk);
    for (unsigned i = c * kAvgChunk + threadIdx.x; i < i1; i += blockDim.x) {
        const int r = bel[i];
        if (r < 0 || (unsigned)r >= R) {
            atomicAdd(err + kErrBad, 1u);
            atomicMin(err + kErrBadFirst, i);
        } else {
            atomicAdd(cnt + (size_t)c * R + r, 1u);
        }
    }
}

// thread per group: cnt[c][r] <- members of r in chunks before c; total[r]
__global__ void __launch_bounds__(256)
avg_chunk_scan_kernel(unsigned* __restrict__ cnt, unsigned n_chunks, unsigned R, unsigned* __restrict__ total)
{
    const unsigned r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= R)
        return;
    unsigned run = 0;
    for (unsigned c0 = 0; c0 < n_chunks; c0 += 8) {
        unsigned v[8];
#pragma unroll
        for (unsigned k = 0; k < 8; k++)
            v[k] = c0 + k < n_chunks ? cnt[(size_t)(c0 + k) * R + r] : 0u;
#pragma unroll
        for (unsigned k = 0; k < 8; k++)
            if (c0 + k < n_chunks) {
                cnt[(size_t)(c0 + k) * R + r] = run;
                run += v[k];
            }
    }
    total[r] = run;
}

// one CTA of 1024 threads: start[r] = members of the groups before r,
// pstart[r] = pieces of the groups before r (pstart[R] = all pieces),
// members[r] (optional output), empty groups flagged
__global__ void __launch_bounds__(1024)
avg_group_scan_kernel(const unsigned* __restrict__ total, unsigned R, unsigned piece, unsigned* __restrict__ start,
                      unsigned* __restrict__ pstart, int* __restrict__ members, unsigned* __restrict__ err)
{
    __shared__ unsigned wa[32], wb[32], carry[2];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0)
        carry[0] = carry[1] = 0;
    __syncthreads();
    for (unsigned r0 = 0; r0 < R; r0 += 1024) {
        const unsigned r = r0 + threadIdx.x;
        const unsigned m = r < R ? total[r] : 0u;
        const unsigned np = (m + piece - 1) / piece;
        unsigned a = m, b = np;
#pragma unroll
        for (unsigned o = 1; o < 32; o <<= 1) {
            const unsigned ta = __shfl_up_sync(0xffffffffu, a, o), tb = __shfl_up_sync(0xffffffffu, b, o);
            if (lane >= o) {
                a += ta;
                b += tb;
            }
        }
        if (lane == 31)
            wa[warp] = a, wb[warp] = b;
        __syncthreads();
        if (warp == 0) {
            unsigned x = wa[lane], y = wb[lane];
#pragma unroll
            for (unsigned o = 1; o < 32; o <<= 1) {
                const unsigned tx = __shfl_up_sync(0xffffffffu, x, o), ty = __shfl_up_sync(0xffffffffu, y, o);
                if (lane >= o) {
                    x += tx;
                    y += ty;
                }
            }
            wa[lane] = x;
            wb[lane] = y;
        }
        __syncthreads();
        const unsigned ca = carry[0], cb = carry[1];
        if (r < R) {
            start[r] = ca + (warp ? wa[warp - 1] : 0u) + a - m;
            pstart[r] = cb + (warp ? wb[warp - 1] : 0u) + b - np;
            if (members)
                members[r] = (int)m;
            if (m == 0) {
                atomicAdd(err + kErrEmpty, 1u);
                atomicMin(err + kErrEmptyFirst, r);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            carry[0] = ca + wa[31];
            carry[1] = cb + wb[31];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        pstart[R] = carry[1];
}

// thread per particle: its member record from the peak of its group's pair,
// with the caller's conversion (bin/sp_isac2_gpu.py:1015-1022):
// sx = -sx_peak cos(a) - sy_peak sin(a), sy = sx_peak sin(a) - sy_peak cos(a),
// in FP64 (one rounding per operation), rounded to float
__global__ void __launch_bounds__(256)
avg_convert_kernel(const int* __restrict__ bel, unsigned P, unsigned R, const float4* __restrict__ peaks,
                   unsigned long long pitch, AvgMember* __restrict__ rec)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P)
        return;
    const int r = bel[i];
    if (r < 0 || (unsigned)r >= R)
        return;
    const float4 pk = peaks[(size_t)r * pitch + i];
    const double t = __dmul_rn((double)pk.x, kPi / 180.0);
    double sn, cs;
    sincos(t, &sn, &cs);
    const double sxn = -(double)pk.y, syn = -(double)pk.z, ss = -sn;
    AvgMember m;
    m.sx = (float)__dsub_rn(__dmul_rn(sxn, cs), __dmul_rn(syn, ss));
    m.sy = (float)__dadd_rn(__dmul_rn(sxn, ss), __dmul_rn(syn, cs));
    m.c = (float)cs;
    m.s = (float)sn;
    m.ang = pk.x;
    m.img = i;
    m.mirror = pk.w != 0.0f;
    m.pad = 0;
    rec[i] = m;
}

// one warp per chunk, particles in order: order[slot] = particle, the slot
// its group's first member + the members of its group in earlier chunks +
// those earlier in this chunk (match_any within each 32 particles, then the
// group's running count in shared memory).  The chunk's groups are loaded
// first, 32 per lane, so the 32 steps wait on no global load.
__global__ void __launch_bounds__(32)
avg_scatter_kernel(const int* __restrict__ bel, unsigned P, unsigned R, unsigned* __restrict__ cnt,
                   const unsigned* __restrict__ start, unsigned* __restrict__ order)
{
    extern __shared__ unsigned row_s[];
    const unsigned c = blockIdx.x, lane = threadIdx.x;
    const bool in_smem = R <= kSmemGroups;
    unsigned* row = in_smem ? row_s : cnt + (size_t)c * R;
    if (in_smem)
        for (unsigned r = lane; r < R; r += 32)
            row_s[r] = cnt[(size_t)c * R + r] + start[r];
    const unsigned i0 = c * kAvgChunk, i1 = min(P, i0 + kAvgChunk);
    int g[kAvgChunk / 32];
#pragma unroll
    for (unsigned s = 0; s < kAvgChunk / 32; s++) {
        const unsigned i = i0 + s * 32 + lane;
        g[s] = i < i1 ? bel[i] : -1;
    }
    __syncwarp();
#pragma unroll
    for (unsigned s = 0; s < kAvgChunk / 32; s++) {
        const unsigned i = i0 + s * 32 + lane;
        const bool ok = g[s] >= 0 && (unsigned)g[s] < R;
        const unsigned r = ok ? (unsigned)g[s] : 0xffffffffu;
        const unsigned peers = __match_any_sync(0xffffffffu, r);
        const unsigned leader = __ffs(peers) - 1;
        const unsigned rank = __popc(peers & ((1u << lane) - 1u));
        unsigned base = (ok && lane == leader) ? row[r] : 0u;
        base = __shfl_sync(0xffffffffu, base, leader);
        __syncwarp();
        if (ok && lane == leader)
            row[r] = base + __popc(peers);
        if (ok)
            order[base + rank + (in_smem ? 0u : start[r])] = i;
        __syncwarp();
    }
}

// one warp per group: the shift sums in FP64 (a mirrored particle's sx
// subtracted), rounded to float and divided by the member count; every
// member's parameters (ang, sx -/+ mean, sy - mean, mirror) as float
__global__ void __launch_bounds__(256)
avg_shift_kernel(const AvgMember* __restrict__ rec, const unsigned* __restrict__ order, const unsigned* __restrict__ start,
                 const unsigned* __restrict__ total, unsigned R, double2* __restrict__ mean, float2* __restrict__ shifts,
                 float4* __restrict__ params)
{
    const unsigned r = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (r >= R)
        return;
    const unsigned k0 = start[r], m = total[r];
    double ax = 0.0, ay = 0.0;
    for (unsigned k = lane; k < m; k += 32) {
        const AvgMember b = rec[order[k0 + k]];
        ax += b.mirror ? -(double)b.sx : (double)b.sx;
        ay += (double)b.sy;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ax += __shfl_xor_sync(0xffffffffu, ax, o);
        ay += __shfl_xor_sync(0xffffffffu, ay, o);
    }
    const double mx = m ? (double)(float)ax / (double)m : 0.0;
    const double my = m ? (double)(float)ay / (double)m : 0.0;
    if (lane == 0) {
        mean[r] = make_double2(mx, my);
        if (shifts)
            shifts[r] = make_float2((float)mx, (float)my);
    }
    if (params)
        for (unsigned k = lane; k < m; k += 32) {
            const AvgMember b = rec[order[k0 + k]];
            const double sx = b.mirror ? (double)b.sx + mx : (double)b.sx - mx;
            params[b.img] = make_float4(b.ang, (float)sx, (float)((double)b.sy - my), b.mirror ? 1.0f : 0.0f);
        }
}

struct AvgSumArgs {
    const float* imgs;
    const AvgMember* rec;
    const unsigned* order;
    const unsigned* start;
    const unsigned* total;
    const unsigned* pstart;
    float* partial;
    unsigned* err;
    unsigned P, R, D, G, piece, pitch, half;
    unsigned test_stall, wait_iters; // failure-path tests only (gpuisac_test_stall_ccf)
};

// the six pixels of the quadratic rule at one source point
struct Six {
    float f00, fp0, fm0, f0p, f0m, fpp; // offsets (0, 0), (+1, 0), (-1, 0), (0, +1), (0, -1), (+1, +1)
};

__device__ __forceinline__ Six six_at(const float* __restrict__ q, int ip, int im, int jp, int jm)
{
    return {q[0], q[ip], q[im], q[jp], q[jm], q[jp + ip]};
}

constexpr unsigned kSumTileX = 8, kSumTileY = 4; // a warp's pixels of the output

__device__ __forceinline__ f32x2 add2_down(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Adds one member's interpolated values to a thread's pixels of column ix: rows
// row0 + p step < limit, p < ROWS, two at a time in packed halves (float operations in the
// order of the restatement).
//   x + 2^23 rounded down is 2^23 + floor(x) for x in [0, 2^23): its low bits are
// the index and one subtraction gives the floor, where floorf and the conversion
// each take a quarter-rate instruction.  Any other x (negative, infinite, NaN)
// differs from 2^23 in its bits by more than D, as an unsigned number, so that one
// comparison finds the points with all neighbours inside; a pair with another
// point takes the general way.
template <int ROWS>
__device__ __forceinline__ void accumulate(f32x2 (&acc)[ROWS / 2], const float* __restrict__ src,
                                           const AvgMember& b, unsigned ix, unsigned row0, unsigned limit,
                                           unsigned step, unsigned D, unsigned pitch)
{
    const float h = (float)(D >> 1);
    const unsigned ixs = b.mirror ? (ix == 0 ? 0u : D - ix) : ix;
    const float x = __fsub_rn((float)ixs, __fadd_rn(h, b.sx));
    const float hy = __fadd_rn(h, b.sy);
    const float xc = __fmul_rn(x, b.c), xs = __fmul_rn(x, b.s);
    const f32x2 xc2 = pack_f32x2(xc, xc), xs2 = pack_f32x2(xs, xs), hy2 = pack_f32x2(hy, hy), h2 = pack_f32x2(h, h);
    const f32x2 two23 = pack_f32x2(8388608.0f, 8388608.0f), one = pack_f32x2(1.0f, 1.0f);
    const f32x2 half = pack_f32x2(0.5f, 0.5f), down = pack_f32x2((float)(2 * step), (float)(2 * step));
    f32x2 iy2 = pack_f32x2((float)row0, (float)(row0 + step));
    const unsigned first = 0x4B000001u; // the bits of 2^23 + 1: index 1
    const float* src1 = src + pitch + 1; // pixel (1, 1)
#pragma unroll
    for (int p = 0; p < ROWS / 2; p++) {
        const unsigned iy = row0 + 2u * (unsigned)p * step;
        if (iy >= limit)
            break;
        const f32x2 y = sub2(iy2, hy2);
        iy2 = add2(iy2, down);
        // (the products by themselves: a packed one would be contracted into the sum)
        const float2 yf = unpack_f32x2(y);
        const f32x2 ys = pack_f32x2(__fmul_rn(yf.x, b.s), __fmul_rn(yf.y, b.s));
        const f32x2 yc = pack_f32x2(__fmul_rn(yf.x, b.c), __fmul_rn(yf.y, b.c));
        const f32x2 xo = add2(sub2(xc2, ys), h2), yo = add2(add2(xs2, yc), h2);
        const f32x2 tx = add2_down(xo, two23), ty = add2_down(yo, two23);
        const float2 fx = unpack_f32x2(tx), fy = unpack_f32x2(ty);
        const unsigned ia = __float_as_uint(fx.x) - first, ib = __float_as_uint(fx.y) - first;
        const unsigned ja = __float_as_uint(fy.x) - first, jb = __float_as_uint(fy.y) - first;
        f32x2 dx = sub2(xo, sub2(tx, two23)), dy = sub2(yo, sub2(ty, two23));
        Six a, c;
        if (ia < D - 2u && ib < D - 2u && ja < D - 2u && jb < D - 2u) {
            a = six_at(src1 + (ja * pitch + ia), 1, -1, (int)pitch, -(int)pitch);
            c = six_at(src1 + (jb * pitch + ib), 1, -1, (int)pitch, -(int)pitch);
        } else {
            float2 dxs = unpack_f32x2(dx), dys = unpack_f32x2(dy);
            // a point outside [0, D)^2 is the pixel itself; neighbours wrap
            auto border = [&](unsigned i, unsigned j, unsigned iy_own, float& ddx, float& ddy) {
                if (i >= D || j >= D) {
                    i = ixs;
                    j = iy_own;
                    ddx = ddy = 0.0f;
                }
                const int Di = (int)D, wrap = (Di - 1) * (int)pitch;
                return six_at(src + (j * pitch + i), i + 1 == D ? 1 - Di : 1, i == 0 ? Di - 1 : -1,
                              j + 1 == D ? -wrap : (int)pitch, j == 0 ? wrap : -(int)pitch);
            };
            a = border(ia + 1u, ja + 1u, iy, dxs.x, dys.x);
            c = border(ib + 1u, jb + 1u, min(iy + step, D - 1), dxs.y, dys.y); // (a row past the last is not stored)
            dx = pack_f32x2(dxs.x, dxs.y), dy = pack_f32x2(dys.x, dys.y);
        }
        const f32x2 f00 = pack_f32x2(a.f00, c.f00);
        const f32x2 c1 = sub2(pack_f32x2(a.fp0, c.fp0), f00);
        const f32x2 c2 = mul2(add2(sub2(c1, f00), pack_f32x2(a.fm0, c.fm0)), half);
        const f32x2 c3 = sub2(pack_f32x2(a.f0p, c.f0p), f00);
        const f32x2 c4 = mul2(add2(sub2(c3, f00), pack_f32x2(a.f0m, c.f0m)), half);
        const f32x2 c5 = sub2(sub2(sub2(pack_f32x2(a.fpp, c.fpp), f00), c1), c3);
        const f32x2 u = fma2(dy, c5, fma2(sub2(dx, one), c2, c1));
        const f32x2 v = fma2(dy, fma2(sub2(dy, one), c4, c3), fma2(dx, u, f00));
        acc[p] = add2(acc[p], v);
    }
}

// grid: an upper bound on the pieces; CTA t >= pieces returns.  Warps
// ceil(D / 8) x G: warp (cb, g) has the tiles of four rows row0 + 4 (g + p G), p <
// ROWS, the first half of them (`half` output rows) of columns 8 cb .. 8 cb + 7, the
// second half of the columns half the image away (the outer columns have most of the
// border's pixels; a warp's share of a member is then about the others'), in passes of
// 2 half rows over the piece's members (one pass up to D = 128).  STAGED: the image
// in shared memory with row length `pitch`.
// What bounds it: issue and shared loads, six a pixel (without the border's branch
// 238 us instead of 274 for 20,000 members of side 76, without any interpolation 83).
// A warp's 8 x 4 pixels meet shared banks two deep at any angle where 32 of one row
// met them 2.5 deep, and 4 deep when the row length is a multiple of 32.  Before (a
// warp's pixels along rows, one at a time, floorf, pieces of P / (4 waves) members):
// 20,000 of side 76 in 200 groups 295 us, now 275; 4,000 of 64 in 40 89 -> 64; 3,000
// of 128 in 20 252 -> 141; 900 of 48 in 11 23 -> 12; 500 of 200 in 5 (read from global
// memory) 304 -> 83.  Not kept: three CTAs of 10 warps an SM (64 registers, spills) 284,
// four 299.
template <bool STAGED, int ROWS, int THREADS, int CTAS>
__global__ void __launch_bounds__(THREADS, CTAS)
avg_sum_kernel(AvgSumArgs a)
{
    extern __shared__ __align__(16) float sbuf[];
    __shared__ uint64_t bars[2];
    // the piece's members (read one by one as their copies are issued, the warp that
    // issues kept the others waiting at the end of each member)
    __shared__ AvgMember mrec[STAGED ? kMaxPiece : 1];
    const unsigned t = blockIdx.x, R = a.R, D = a.D, G = a.G;
    const unsigned n_pieces = a.pstart[R];
    if (t >= n_pieces)
        return;
    // the group whose pieces hold t: the last r with pstart[r] <= t
    unsigned lo = 0, hi = R; // pstart[lo] <= t < pstart[hi]
    while (hi - lo > 1) {
        const unsigned mid = (lo + hi) >> 1;
        if (a.pstart[mid] <= t)
            lo = mid;
        else
            hi = mid;
    }
    const unsigned r = lo;
    const unsigned k0 = a.start[r] + (t - a.pstart[r]) * a.piece;
    const unsigned k1 = min(a.start[r] + a.total[r], k0 + a.piece);
    const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const unsigned blocks = (D + kSumTileX - 1) / kSumTileX, cb = warp / G;
    const unsigned ix = cb * kSumTileX + lane % kSumTileX, iy0 = (warp % G) * kSumTileY + lane / kSumTileX;
    const unsigned ix2 = (cb + blocks / 2) % blocks * kSumTileX + lane % kSumTileX; // the second half's column
    const unsigned step = kSumTileY * G;
    const size_t npix = (size_t)D * D, nbuf = (size_t)D * a.pitch;
    const uint32_t bytes = (uint32_t)(npix * sizeof(float));
    const uint32_t wlim = wait_tries(a.wait_iters);
    auto issue = [&](unsigned k, unsigned buf) { // by warp 0
        if (a.test_stall)
            return; // failure-path test: no copy, a wait that runs out
        const unsigned img_of = mrec[k - k0].img;
        fence_proxy_async(); // the buffer's readers are done
        if (lane == 0)
            mbar_expect_tx(&bars[buf], img_of < a.P ? bytes : 0);
        __syncwarp();
        if (GPUISAC_IN_BOUNDS(kChkAvgImg, img_of, a.P)) {
            const float* img = a.imgs + (size_t)img_of * npix;
            float* dst = sbuf + buf * nbuf;
            if (a.pitch == D) {
                if (lane == 0)
                    bulk_g2s(dst, img, bytes, &bars[buf]);
            } else {
                for (unsigned y = lane; y < D; y += 32)
                    bulk_g2s(dst + y * a.pitch, img + (size_t)y * D, D * (uint32_t)sizeof(float), &bars[buf]);
            }
        }
    };
    if (STAGED) {
        if (tid == 0) {
            mbar_init(&bars[0], 1);
            mbar_init(&bars[1], 1);
            mbar_fence_init();
        }
        for (unsigned k = k0 + tid; k < k1; k += blockDim.x)
            mrec[k - k0] = a.rec[a.order[k]];
        __syncthreads();
    }
    unsigned u = 0; // members consumed: use u of buffer u & 1 completes phase (u >> 1) & 1
    // (columns beyond the last are not stored)
    auto add = [&](f32x2(&acc)[2][ROWS / 4], const float* src, const AvgMember& b, unsigned row0, unsigned pitch) {
        accumulate<ROWS / 2>(acc[0], src, b, min(ix, D - 1), row0 + iy0, min(row0 + a.half, D), step, D, pitch);
        accumulate<ROWS / 2>(acc[1], src, b, min(ix2, D - 1), row0 + a.half + iy0, D, step, D, pitch);
    };
    for (unsigned row0 = 0; row0 < D; row0 += 2 * a.half) {
        f32x2 acc[2][ROWS / 4];
#pragma unroll
        for (int p = 0; p < ROWS / 4; p++)
            acc[0][p] = acc[1][p] = 0;
        if (STAGED) {
            if (warp == 0) {
                issue(k0, u & 1u);
                if (k0 + 1 < k1)
                    issue(k0 + 1, (u + 1) & 1u);
            }
            for (unsigned k = k0; k < k1; k++, u++) {
                const unsigned buf = u & 1u;
                const bool ok = mbar_wait(&bars[buf], (u >> 1) & 1u, wlim);
                if (ok)
                    add(acc, sbuf + buf * nbuf, mrec[k - k0], row0, a.pitch);
                if (__syncthreads_or(!ok)) {
                    if (tid == 0) {
                        atomicAdd(a.err + kErrWait, 1u);
                        // the copies still in flight land before the CTA leaves
                        if (!ok && !a.test_stall)
                            mbar_wait(&bars[buf], (u >> 1) & 1u, wlim);
                        if (k + 1 < k1 && !a.test_stall)
                            mbar_wait(&bars[buf ^ 1u], ((u + 1) >> 1) & 1u, wlim);
                    }
                    return;
                }
                if (warp == 0 && k + 2 < k1)
                    issue(k + 2, buf);
            }
        } else {
            for (unsigned k = k0; k < k1; k++) {
                const AvgMember b = a.rec[a.order[k]];
                if (GPUISAC_IN_BOUNDS(kChkAvgImg, b.img, a.P))
                    add(acc, a.imgs + (size_t)b.img * npix, b, row0, D);
            }
        }
        float* out = a.partial + (size_t)t * npix;
#pragma unroll
        for (int p = 0; p < ROWS; p++) {
            const int hf = p / (ROWS / 2), ph = p % (ROWS / 2);
            const unsigned iy = row0 + hf * a.half + iy0 + (unsigned)ph * step, col = hf ? ix2 : ix;
            const float2 v = unpack_f32x2(acc[hf][ph / 2]);
            if (col < D && iy < (hf ? D : min(row0 + a.half, D)) &&
                GPUISAC_IN_BOUNDS(kChkAvgPartial, (size_t)t * npix + (size_t)iy * D + col, (size_t)n_pieces * npix))
                out[(size_t)iy * D + col] = ph % 2 ? v.y : v.x;
        }
    }
}

struct AvgFinishArgs {
    const float* partial;
    const unsigned* pstart;
    const unsigned* total;
    const double2* mean;
    const float2* tw; // e^(2 pi i j / D), j = 0..D-1
    float2* spec;     // [groups of the launch][D][H] half spectra
    float* avg;
    unsigned R, D;
    unsigned r0, tiles; // first group of the launch, CTAs per group
    float fl, ff;
    int center;
};

// ---- averages from their pieces, filtered and moved ----
// Per group: the sum of its pieces times float(1/members); then, when
// filtering or centring, the real DFT over rows (x) then columns (y), the
// spectrum times the filter 0.5 (tanh(k (r + fl)) - tanh(k (r - fl))),
// k = pi / (2 ff fl), r = |(kx, ky)| / D (ky > D/2 taken as ky - D; a step at fl
// when ff = 0), and the phase exp(-2 pi i (kx dx + ky dy) / D) with (dx, dy) =
// -mean shift, then the inverse DFT over columns and the real inverse over rows
// (the imaginary parts of the kx = 0 and D/2 terms dropped), divided by D^2.
//
// Any side up to 256, so the transforms are plain sums, in three kernels: rows
// (a CTA per group and 2 kFinTile rows), columns with filter and inverse columns
// (per group and 2 kFinCols columns), inverse rows (as the first).  Each sum is
// folded: terms j and D - j share a twiddle (their sum meets the cosine, their
// difference the sine), and so do results k and D - k of a column or an inverse
// row (they differ in the sine part's sign): half the products of the real passes,
// a quarter of the complex ones.  A thread has one k (or pair of results) and
// kFinTile rows or kFinCols columns, whose folded values it reads as float4 at one
// address per warp (two where a tile ends).
// What bounds it: latency; 200 groups of side 76 are 1,000 CTAs of three warps a
// kernel.  Pieces, rows, columns, inverse rows 18 + 11 + 24 + 11 us there and 9 + 9 +
// 17 + 9 for 20 groups of side 128, against 128 and 332 with one CTA per group and
// unfolded sums; the error against FP64 went from 4.1e-7 to 2.5e-7.
constexpr unsigned kFinTile = 8;  // rows per thread
constexpr unsigned kFinCols = 4;  // columns per thread
constexpr unsigned kFinRows = 2 * kFinTile;
constexpr unsigned kFinColumns = 2 * kFinCols;
constexpr unsigned kFinPitch = kFinRows + 4;       // of the folded rows: stores along x meet 4 banks deep, not 16
constexpr unsigned kFinColPitch = kFinColumns + 1; // of the columns' spectra: stores along ky without conflicts
constexpr size_t kFinSpecBytes = 64u << 20;        // half spectra held at once (in L2)
constexpr unsigned kFinThreads = 288; // covers 2 (kMaxDim / 2 + 1) in whole warps

// Each group's pieces summed in order, times float(1/members), into the averages
// (0 without members): a thread per pixel, eight pieces' loads in flight, the sum's
// rounding errors kept (Knuth's two-sum) and added at the end, so that the number of
// pieces costs no precision; a sum that overflowed or holds a NaN stays as it is.
// (Inside the row pass, a thread's pixels one after another, the two kernels' 18 us for
// 20 groups of side 128 with 19 pieces each were 63.)
__global__ void __launch_bounds__(256)
avg_mean_kernel(AvgFinishArgs a)
{
    const unsigned r = blockIdx.x / a.tiles, m = a.total[r];
    const size_t npix = (size_t)a.D * a.D, q = (size_t)(blockIdx.x % a.tiles) * 256 + threadIdx.x;
    if (q >= npix || !GPUISAC_IN_BOUNDS(kChkAvgOut, (size_t)r * npix + q, (size_t)a.R * npix))
        return;
    float s = 0.0f, lost = 0.0f;
    const unsigned p1 = a.pstart[r + 1];
    for (unsigned p = a.pstart[r]; p < p1; p += 8) {
        float v[8];
#pragma unroll
        for (unsigned i = 0; i < 8; i++)
            v[i] = p + i < p1 ? a.partial[(size_t)(p + i) * npix + q] : 0.0f;
#pragma unroll
        for (unsigned i = 0; i < 8; i++) {
            const float t = __fadd_rn(s, v[i]), w = __fsub_rn(t, s);
            lost += __fadd_rn(__fsub_rn(s, __fsub_rn(t, w)), __fsub_rn(v[i], w));
            s = t;
        }
    }
    s = isfinite(s) ? s + lost : s;
    a.avg[(size_t)r * npix + q] = m ? s * __double2float_rn(1.0 / (double)m) : 0.0f;
}

// spec[y][kx] = sum_x img[y][x] e^(-2 pi i kx x / D): CTA r tiles + t is the launch's
// group r, row tile t.  Shared memory: tw[D], then per x = 0..K the rows' folded sums
// and differences (x = 0: the values at 0 and at D / 2).
__global__ void __launch_bounds__(kFinThreads)
avg_rows_kernel(AvgFinishArgs a)
{
    extern __shared__ __align__(16) float2 fsm[];
    const unsigned rl = blockIdx.x / a.tiles, tile0 = blockIdx.x % a.tiles, r = a.r0 + rl;
    const unsigned D = a.D, H = D / 2 + 1, K = (D - 1) / 2, tid = threadIdx.x;
    if (a.total[r] == 0)
        return;
    const unsigned y0 = tile0 * kFinRows, rows = min(kFinRows, D - y0);
    const size_t npix = (size_t)D * D;
    float2* tw = fsm;                                             // [D | 1]
    float* es = reinterpret_cast<float*>(fsm + ((D + 1) & ~1u));  // [K + 1][kFinPitch]
    float* os = es + (K + 1) * kFinPitch;
    const float* img = a.avg + (size_t)r * npix;
    for (unsigned j = tid; j < D; j += blockDim.x)
        tw[j] = a.tw[j];
    for (unsigned e = tid; e < kFinRows * (K + 1); e += blockDim.x) {
        const unsigned yy = e / (K + 1), x = e % (K + 1);
        float2 v = make_float2(0.0f, 0.0f);
        if (yy < rows) {
            const size_t row = (size_t)(y0 + yy) * D;
            v = make_float2(img[row + x], img[row + (x > 0 ? D - x : D / 2)]);
            if (x == 0 && D % 2 != 0)
                v.y = 0.0f;
        }
        es[x * kFinPitch + yy] = x > 0 ? v.x + v.y : v.x;
        os[x * kFinPitch + yy] = x > 0 ? v.x - v.y : v.y;
    }
    __syncthreads();
    const unsigned tile = tid / H, k = tid % H;
    if (tile >= kFinRows / kFinTile)
        return;
    float re[kFinTile], im[kFinTile];
    const float4* e4 = reinterpret_cast<const float4*>(es) + tile * (kFinTile / 4);
    const float4* o4 = reinterpret_cast<const float4*>(os) + tile * (kFinTile / 4);
#pragma unroll
    for (unsigned i = 0; i < kFinTile; i++)
        re[i] = im[i] = 0.0f;
    unsigned j = k;
    for (unsigned x = 1; x <= K; x++) {
        const float2 w = tw[j];
        e4 += kFinPitch / 4, o4 += kFinPitch / 4;
#pragma unroll
        for (unsigned q = 0; q < kFinTile / 4; q++) {
            const float4 e = e4[q], o = o4[q];
            re[4 * q] = fmaf(e.x, w.x, re[4 * q]), im[4 * q] = fmaf(-o.x, w.y, im[4 * q]);
            re[4 * q + 1] = fmaf(e.y, w.x, re[4 * q + 1]), im[4 * q + 1] = fmaf(-o.y, w.y, im[4 * q + 1]);
            re[4 * q + 2] = fmaf(e.z, w.x, re[4 * q + 2]), im[4 * q + 2] = fmaf(-o.z, w.y, im[4 * q + 2]);
            re[4 * q + 3] = fmaf(e.w, w.x, re[4 * q + 3]), im[4 * q + 3] = fmaf(-o.w, w.y, im[4 * q + 3]);
        }
        j += k;
        j = j >= D ? j - D : j;
    }
    float2* out = a.spec + (size_t)rl * D * H;
#pragma unroll
    for (unsigned i = 0; i < kFinTile; i++) {
        const unsigned yy = tile * kFinTile + i;
        if (yy < rows) {
            const float nyq = os[yy]; // 0 on an odd side
            out[(size_t)(y0 + yy) * H + k] = make_float2(re[i] + es[yy] + ((k & 1u) ? -nyq : nyq), im[i]);
        }
    }
}

// A thread's results k and D - k of kFinCols columns of complex values, folded
// in smem as fold[j][column] = (sum.re, sum.im, difference.re, difference.im) for
// j = 1..K and (v[0], v[D / 2]) at j = 0: lo[c] = sum_j v[j] e^(-2 pi i k j / D),
// hi[c] the same at D - k
__device__ __forceinline__ void dft_columns(const float4* __restrict__ fold, const float2* __restrict__ tw, unsigned k,
                                            unsigned D, float2 (&lo)[kFinCols], float2 (&hi)[kFinCols])
{
    const unsigned K = (D - 1) / 2;
    float ar[kFinCols], ai[kFinCols], br[kFinCols], bi[kFinCols]; // cosine and sine parts
#pragma unroll
    for (unsigned c = 0; c < kFinCols; c++)
        ar[c] = ai[c] = br[c] = bi[c] = 0.0f;
    unsigned j = k;
    const float4* f = fold;
    for (unsigned y = 1; y <= K; y++) {
        const float2 w = tw[j];
        f += kFinColumns;
#pragma unroll
        for (unsigned c = 0; c < kFinCols; c++) {
            const float4 v = f[c];
            ar[c] = fmaf(v.x, w.x, ar[c]);
            ai[c] = fmaf(v.y, w.x, ai[c]);
            br[c] = fmaf(v.w, w.y, br[c]);
            bi[c] = fmaf(v.z, w.y, bi[c]);
        }
        j += k;
        j = j >= D ? j - D : j;
    }
#pragma unroll
    for (unsigned c = 0; c < kFinCols; c++) {
        const float4 v = fold[c];
        const float cr = ar[c] + v.x + ((k & 1u) ? -v.z : v.z), ci = ai[c] + v.y + ((k & 1u) ? -v.w : v.w);
        lo[c] = make_float2(cr + br[c], ci - bi[c]);
        hi[c] = make_float2(cr - br[c], ci + bi[c]);
    }
}

// The column pass in place on spec: forward sums over y, filter and phase,
// inverse sums over ky (the forward ones with results k and D - k exchanged).
// CTA r tiles + t is the launch's group r, column tile t; shared memory: tw[D], the
// folded columns, the columns' spectra.
__global__ void __launch_bounds__(kFinThreads)
avg_cols_kernel(AvgFinishArgs a)
{
    extern __shared__ __align__(16) float2 fsm[];
    const unsigned rl = blockIdx.x / a.tiles, tile0 = blockIdx.x % a.tiles, r = a.r0 + rl;
    const unsigned D = a.D, H = D / 2 + 1, K = (D - 1) / 2, tid = threadIdx.x;
    if (a.total[r] == 0)
        return;
    const unsigned x0 = tile0 * kFinColumns, cols = min(kFinColumns, H - x0);
    float2* tw = fsm;
    float4* fold = reinterpret_cast<float4*>(fsm + ((D + 1) & ~1u)); // [K + 1][kFinColumns]
    float2* g = reinterpret_cast<float2*>(fold + (K + 1) * kFinColumns); // [D][kFinColPitch]
    float2* spec = a.spec + (size_t)rl * D * H;
    auto fold_of = [&](float2 v1, float2 v2, unsigned y) {
        return y > 0 ? make_float4(v1.x + v2.x, v1.y + v2.y, v1.x - v2.x, v1.y - v2.y)
                     : make_float4(v1.x, v1.y, v2.x, v2.y);
    };
    auto partner = [&](unsigned y) { return y > 0 ? D - y : D / 2; }; // (D / 2: even sides only)
    for (unsigned j = tid; j < D; j += blockDim.x)
        tw[j] = a.tw[j];
    const float2 zero = make_float2(0.0f, 0.0f);
    for (unsigned e = tid; e < kFinColumns * (K + 1); e += blockDim.x) {
        const unsigned y = e / kFinColumns, c = e % kFinColumns;
        const bool in = c < cols, has2 = in && (y > 0 || D % 2 == 0);
        fold[e] = fold_of(in ? spec[(size_t)y * H + x0 + c] : zero,
                          has2 ? spec[(size_t)partner(y) * H + x0 + c] : zero, y);
    }
    __syncthreads();
    const unsigned tile = tid / H, k = tid % H;
    const bool work = tile < kFinColumns / kFinCols;
    const unsigned k2 = k == 0 ? 0 : D - k; // k's partner (itself at 0 and D / 2)
    float2 lo[kFinCols], hi[kFinCols];
    if (work) {
        // The phase exp(-2 pi i (kx dx + ky dy) / D) is sincospi(kx px + ky py),
        // px = -2 dx / D rounded to float once per group.
        const double2 mn = a.mean[r];
        const float px = a.center ? (float)(2.0 * mn.x / (double)D) : 0.0f;
        const float py = a.center ? (float)(2.0 * mn.y / (double)D) : 0.0f;
        const float kf = a.ff > 0.0f ? (float)(kPi / (2.0 * (double)a.ff * (double)a.fl)) : 0.0f;
        dft_columns(fold + tile * kFinCols, tw, k, D, lo, hi);
#pragma unroll
        for (unsigned c = 0; c < kFinCols; c++) {
            const unsigned kx = x0 + tile * kFinCols + c;
            // the filter is the same at ky and D - ky
            float hf = 1.0f;
            if (a.fl > 0.0f) {
                const float fx = (float)kx / (float)D, fy = (float)k / (float)D;
                const float rr = sqrtf(fx * fx + fy * fy);
                hf = a.ff > 0.0f ? 0.5f * (tanhf(kf * (rr + a.fl)) - tanhf(kf * (rr - a.fl)))
                                 : (rr < a.fl ? 1.0f : (rr == a.fl ? 0.5f : 0.0f));
            }
            auto finish_term = [&](float2 v, int kys) {
                float ps = 0.0f, pc = 1.0f;
                if (a.center)
                    sincospif(fmaf((float)kx, px, (float)kys * py), &ps, &pc);
                return make_float2((v.x * pc - v.y * ps) * hf, (v.x * ps + v.y * pc) * hf);
            };
            g[k * kFinColPitch + tile * kFinCols + c] = finish_term(lo[c], (int)k);
            if (k2 != k)
                g[k2 * kFinColPitch + tile * kFinCols + c] = finish_term(hi[c], -(int)k);
        }
    }
    __syncthreads();
    for (unsigned e = tid; e < kFinColumns * (K + 1); e += blockDim.x) {
        const unsigned y = e / kFinColumns, c = e % kFinColumns;
        fold[e] = fold_of(g[y * kFinColPitch + c], y > 0 || D % 2 == 0 ? g[partner(y) * kFinColPitch + c] : zero, y);
    }
    __syncthreads();
    if (!work)
        return;
    dft_columns(fold + tile * kFinCols, tw, k, D, lo, hi);
#pragma unroll
    for (unsigned c = 0; c < kFinCols; c++) {
        const unsigned cc = tile * kFinCols + c;
        if (cc < cols) {
            spec[(size_t)k * H + x0 + cc] = hi[c];
            if (k2 != k)
                spec[(size_t)k2 * H + x0 + cc] = lo[c];
        }
    }
}

// inverse rows, half spectrum to real: CTA r tiles + t is the launch's group r, row
// tile t.  Shared memory: tw[D], then per kx = 0..K the rows' real and imaginary
// parts (kx = 0: the real parts at 0 and at D / 2).
__global__ void __launch_bounds__(kFinThreads)
avg_inverse_kernel(AvgFinishArgs a)
{
    extern __shared__ __align__(16) float2 fsm[];
    const unsigned rl = blockIdx.x / a.tiles, tile0 = blockIdx.x % a.tiles, r = a.r0 + rl;
    const unsigned D = a.D, H = D / 2 + 1, K = (D - 1) / 2, tid = threadIdx.x;
    const unsigned y0 = tile0 * kFinRows, rows = min(kFinRows, D - y0);
    const size_t npix = (size_t)D * D;
    float* out = a.avg + (size_t)r * npix;
    if (a.total[r] == 0)
        return;
    float2* tw = fsm;
    float* es = reinterpret_cast<float*>(fsm + ((D + 1) & ~1u));
    float* os = es + (K + 1) * kFinPitch;
    const float2* spec = a.spec + (size_t)rl * D * H;
    for (unsigned j = tid; j < D; j += blockDim.x)
        tw[j] = a.tw[j];
    for (unsigned e = tid; e < kFinRows * (K + 1); e += blockDim.x) {
        const unsigned yy = e / (K + 1), kx = e % (K + 1);
        float2 v = make_float2(0.0f, 0.0f);
        if (yy < rows) {
            const float2* row = spec + (size_t)(y0 + yy) * H;
            v = row[kx];
            if (kx == 0)
                v.y = D % 2 == 0 ? row[D / 2].x : 0.0f;
        }
        es[kx * kFinPitch + yy] = v.x;
        os[kx * kFinPitch + yy] = v.y;
    }
    __syncthreads();
    const unsigned tile = tid / H, x = tid % H;
    if (tile >= kFinRows / kFinTile)
        return;
    float sc[kFinTile], ss[kFinTile];
    const float4* e4 = reinterpret_cast<const float4*>(es) + tile * (kFinTile / 4);
    const float4* o4 = reinterpret_cast<const float4*>(os) + tile * (kFinTile / 4);
#pragma unroll
    for (unsigned i = 0; i < kFinTile; i++)
        sc[i] = ss[i] = 0.0f;
    unsigned j = x;
    for (unsigned kx = 1; kx <= K; kx++) {
        const float2 w = tw[j];
        e4 += kFinPitch / 4, o4 += kFinPitch / 4;
#pragma unroll
        for (unsigned q = 0; q < kFinTile / 4; q++) {
            const float4 e = e4[q], o = o4[q];
            sc[4 * q] = fmaf(e.x, w.x, sc[4 * q]), ss[4 * q] = fmaf(o.x, w.y, ss[4 * q]);
            sc[4 * q + 1] = fmaf(e.y, w.x, sc[4 * q + 1]), ss[4 * q + 1] = fmaf(o.y, w.y, ss[4 * q + 1]);
            sc[4 * q + 2] = fmaf(e.z, w.x, sc[4 * q + 2]), ss[4 * q + 2] = fmaf(o.z, w.y, ss[4 * q + 2]);
            sc[4 * q + 3] = fmaf(e.w, w.x, sc[4 * q + 3]), ss[4 * q + 3] = fmaf(o.w, w.y, ss[4 * q + 3]);
        }
        j += x;
        j = j >= D ? j - D : j;
    }
    const float scale = 1.0f / (float)npix;
#pragma unroll
    for (unsigned i = 0; i < kFinTile; i++) {
        const unsigned yy = tile * kFinTile + i;
        if (yy >= rows)
            break;
        const float nyq = os[yy], base = es[yy] + ((x & 1u) ? -nyq : nyq);
        const size_t q = (size_t)(y0 + yy) * D;
        if (GPUISAC_IN_BOUNDS(kChkAvgOut, (size_t)r * npix + q + D - 1, (size_t)a.R * npix)) {
            out[q + x] = (base + 2.0f * (sc[i] - ss[i])) * scale;
            if (x > 0 && D - x != x)
                out[q + D - x] = (base + 2.0f * (sc[i] + ss[i])) * scale;
        }
    }
}

template <typename T>
struct Buf {
    T* p = nullptr;
    size_t n = 0;
    cudaError_t ensure(size_t count)
    {
        if (count <= n)
            return cudaSuccess;
        if (p)
            cudaFree(p);
        p = nullptr;
        n = 0;
        cudaError_t e = cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T));
        if (e == cudaSuccess)
            n = count;
        return e;
    }
};

struct AvgState {
    std::mutex mu;
    int dev = -1;
    Buf<unsigned> cnt, total, start, pstart, err;
    Buf<AvgMember> rec;
    Buf<unsigned> order;
    Buf<double2> mean;
    Buf<float> partial;
    Buf<float2> scratch, tw;
    std::vector<float2> h_tw;
    unsigned tw_dim = 0;
    unsigned* h_err = nullptr; // pinned
} g_avg;

int fail(int code, const char* msg)
{
    record_error(code, msg);
    return code;
}

#define AV_CK(expr)                                                                                    \
    do {                                                                                               \
        cudaError_t e_ = (expr);                                                                       \
        if (e_ != cudaSuccess) {                                                                       \
            char m_[384];                                                                              \
            snprintf(m_, sizeof(m_), "%s (%s) in the class averages", cudaGetErrorString(e_), #expr); \
            return fail(1, m_);                                                                        \
        }                                                                                              \
    } while (0)

// The sum kernel: images up to side 80 by CTAs of ceil(D / 8) warps with 20 rows a
// thread, two to an SM at side 76 (96 registers); larger ones with 16 rows a thread and two row groups (one
// pass) up to side 128, one group above.
constexpr unsigned kSumSmall = 80;
unsigned sum_groups(unsigned D) { return D <= kSumSmall || D > 128 ? 1 : 2; }

void release(AvgState& w)
{
    if (w.dev < 0)
        return;
    int cur = 0;
    cudaGetDevice(&cur);
    cudaSetDevice(w.dev);
    cudaFree(w.cnt.p), cudaFree(w.total.p), cudaFree(w.start.p), cudaFree(w.pstart.p), cudaFree(w.err.p);
    cudaFree(w.rec.p), cudaFree(w.order.p), cudaFree(w.mean.p), cudaFree(w.partial.p), cudaFree(w.scratch.p), cudaFree(w.tw.p);
    cudaSetDevice(cur);
    w.cnt = {}, w.total = {}, w.start = {}, w.pstart = {}, w.err = {}, w.rec = {}, w.order = {}, w.mean = {}, w.partial = {};
    w.scratch = {}, w.tw = {};
    w.tw_dim = 0;
}

} // namespace

GPUISAC_CHECKED_READER(checked_read_averages)

void averages_clear()
{
    std::lock_guard<std::mutex> lk(g_avg.mu);
    release(g_avg);
    g_avg.dev = -1;
    if (g_avg.h_err)
        cudaFreeHost(g_avg.h_err);
    g_avg.h_err = nullptr;
}

} // namespace gpuisac

using namespace gpuisac;

extern "C" int gpuisac_class_averages(const float* imgs, unsigned int n_img, unsigned int img_dim, const float* peaks,
                                      unsigned long long peak_pitch, const int* belongsto, unsigned int n_class,
                                      float fl, float ff, int center, float* averages, float* params, int* members,
                                      float* shifts, void* stream_)
{
    const gpuisac::NvtxRange nvtx_range("gpuisac:class_averages");
    if (!imgs || !peaks || !belongsto || !averages)
        return fail(2, "class_averages: NULL imgs, peaks, belongsto or averages");
    if (n_img == 0 || n_class == 0)
        return fail(2, "class_averages: needs n_img >= 1 and n_class >= 1");
    if (img_dim < 2 || img_dim > kMaxDim)
        return fail(2, "class_averages: img_dim outside 2..256");
    if (peak_pitch == 0)
        peak_pitch = n_img;
    if (peak_pitch < n_img)
        return fail(2, "class_averages: peak_pitch smaller than n_img");
    if ((uintptr_t)peaks % 16 != 0)
        return fail(2, "class_averages: peaks not 16-byte aligned");
    if (!(fl <= 0.5f) || !(ff >= 0.0f && ff <= 0.5f))
        return fail(2, "class_averages: needs fl <= 0.5 and 0 <= ff <= 0.5");
    if ((params && (uintptr_t)params % 16 != 0) || (shifts && (uintptr_t)shifts % 8 != 0))
        return fail(2, "class_averages: params not 16-byte or shifts not 8-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream_);
    std::lock_guard<std::mutex> lk(g_avg.mu);
    AvgState& w = g_avg;
    int dev = 0;
    AV_CK(cudaGetDevice(&dev));
    if (w.dev != dev) { // buffers of another device are not reused
        release(w);
        w.dev = dev;
    }
    const unsigned D = img_dim, R = n_class, P = n_img;
    const size_t npix = (size_t)D * D;
    const unsigned n_chunks = (P + kAvgChunk - 1) / kAvgChunk;
    // member images staged by bulk copies: whole rows of 16-byte multiples
    const bool staged = D % 2 == 0 && D <= kStagedMaxDim && (uintptr_t)imgs % 16 == 0;
    void (*sum_kernel)(AvgSumArgs) =
        D <= kSumSmall ? (staged ? avg_sum_kernel<true, 20, 320, 2> : avg_sum_kernel<false, 20, 320, 2>)
                       : (staged ? avg_sum_kernel<true, 16, 1024, 1> : avg_sum_kernel<false, 16, 1024, 1>);
    // a row length that is a multiple of 16 floats puts a tile's rows on the same
    // banks: such an image is staged with 4 more per row, row by row
    const unsigned pitch = staged && D % 16 == 0 ? D + 4 : D;
    const unsigned G = sum_groups(D), sum_threads = (D + kSumTileX - 1) / kSumTileX * G * 32;
    // output rows of a half pass: pairs of tiles, as few as cover the image
    const unsigned sum_rows = D <= kSumSmall ? 20 : 16, sum_tiles = (D + kSumTileY - 1) / kSumTileY;
    const unsigned half = std::min(sum_rows / 2, (sum_tiles + 4 * G - 1) / (4 * G) * 2) * kSumTileY * G;
    const size_t sum_smem = staged ? 2 * sizeof(float) * D * pitch : 0;
    int sms = 0, per_sm = 0;
    AV_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (sum_smem + kMaxPiece * sizeof(AvgMember) + 64 > 48 * 1024) // (the static arrays count)
        AV_CK(cudaFuncSetAttribute(sum_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sum_smem));
    AV_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sum_kernel, (int)sum_threads, sum_smem));
    // Members of a piece: whole waves of resident CTAs if the groups are of equal
    // size (what the assignment makes; with others only the last wave is less full), a
    // wave's time taken as its members and two more for the start; pieces of fewer than
    // 8 only where their partial images stay few, the longest of equals (the fewest
    // partial images).  A piece's members are added one after another in FP32, so it
    // has no more of them than additions follow one another with quarter waves of
    // `quarter` members and a plain sum of their pieces: 20,000 in 200 groups of side 76
    // 17 members, 50,000 in 200 42.  Root mean square error against FP64 of the largest
    // average 1.65e-8 and 1.99e-8 (without that bound, 34 and 84 members, in the same
    // time 2.10e-8 and 2.68e-8; in runs of 17 and 42 with plain sums 1.83e-8, 2.14e-8).
    const unsigned resident = (unsigned)std::max(1, sms * std::max(per_sm, 1)), group = (P + R - 1) / R;
    const unsigned least = P / kMinPiece + R <= 4 * resident ? kMinPiece : 8u;
    const unsigned quarter = std::min(kMaxPiece, std::max(8u, (P + 4 * resident - 1) / (4 * resident)));
    const unsigned most = std::min(kMaxPiece, quarter + (group - 1) / quarter);
    unsigned piece = least;
    unsigned long long best = ~0ull;
    for (unsigned c = least; c <= most; c++) {
        const unsigned long long n = (unsigned long long)R * ((group + c - 1) / c);
        const unsigned long long cost = (n + resident - 1) / resident * (std::min(c, group) + 2);
        if (cost <= best)
            best = cost, piece = c;
    }
    const size_t pieces_cap = (size_t)P / piece + R + 1;
    const bool spectra = fl > 0.0f || center;
    const unsigned H = D / 2 + 1, K = (D - 1) / 2;
    const unsigned fin_groups =
        (unsigned)std::min<size_t>(R, std::max<size_t>(1, kFinSpecBytes / ((size_t)D * H * sizeof(float2))));

    AV_CK(w.cnt.ensure((size_t)n_chunks * R));
    AV_CK(w.total.ensure(R));
    AV_CK(w.start.ensure(R));
    AV_CK(w.pstart.ensure((size_t)R + 1));
    AV_CK(w.err.ensure(kErrWords));
    AV_CK(w.rec.ensure(P));
    AV_CK(w.order.ensure(P));
    AV_CK(w.mean.ensure(R));
    AV_CK(w.partial.ensure(pieces_cap * npix));
    if (spectra)
        AV_CK(w.scratch.ensure((size_t)fin_groups * D * H));
    if (!w.h_err)
        AV_CK(cudaMallocHost(&w.h_err, kErrWords * sizeof(unsigned)));
    if (w.tw_dim != D) {
        // (read until the stream is synchronised below: kept in the state, copied on
        // the caller's stream)
        w.tw_dim = 0;
        w.h_tw.resize(D);
        for (unsigned j = 0; j < D; j++)
            w.h_tw[j] = make_float2((float)cos(2.0 * kPi * j / D), (float)sin(2.0 * kPi * j / D));
        AV_CK(w.tw.ensure(D));
        AV_CK(cudaMemcpyAsync(w.tw.p, w.h_tw.data(), D * sizeof(float2), cudaMemcpyHostToDevice, st));
        w.tw_dim = D;
    }

    AV_CK(cudaMemsetAsync(w.cnt.p, 0, (size_t)n_chunks * R * sizeof(unsigned), st));
    AV_CK(cudaMemsetAsync(w.err.p, 0, kErrWords * sizeof(unsigned), st));
    AV_CK(cudaMemsetAsync(w.err.p + kErrBadFirst, 0xff, sizeof(unsigned), st));
    AV_CK(cudaMemsetAsync(w.err.p + kErrEmptyFirst, 0xff, sizeof(unsigned), st));
    avg_count_kernel<<<n_chunks, 256, 0, st>>>(belongsto, P, R, w.cnt.p, w.err.p);
    avg_chunk_scan_kernel<<<(R + 255) / 256, 256, 0, st>>>(w.cnt.p, n_chunks, R, w.total.p);
    avg_group_scan_kernel<<<1, 1024, 0, st>>>(w.total.p, R, piece, w.start.p, w.pstart.p, members, w.err.p);
    const size_t scat_smem = R <= kSmemGroups ? (size_t)R * sizeof(unsigned) : 0;
    if (scat_smem > 48 * 1024)
        AV_CK(cudaFuncSetAttribute(avg_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)scat_smem));
    avg_convert_kernel<<<(P + 255) / 256, 256, 0, st>>>(belongsto, P, R, reinterpret_cast<const float4*>(peaks),
                                                        peak_pitch, w.rec.p);
    avg_scatter_kernel<<<n_chunks, 32, scat_smem, st>>>(belongsto, P, R, w.cnt.p, w.start.p, w.order.p);
    avg_shift_kernel<<<(R + 7) / 8, 256, 0, st>>>(w.rec.p, w.order.p, w.start.p, w.total.p, R, w.mean.p,
                                                  reinterpret_cast<float2*>(shifts), reinterpret_cast<float4*>(params));
    AvgSumArgs sa{imgs, w.rec.p, w.order.p, w.start.p, w.total.p, w.pstart.p, w.partial.p, w.err.p, P, R, D, G, piece,
                  pitch, half, 0, 0};
    ccf_test_settings(sa.test_stall, sa.wait_iters);
    sum_kernel<<<(unsigned)pieces_cap, sum_threads, sum_smem, st>>>(sa);
    AvgFinishArgs fa{w.partial.p, w.pstart.p, w.total.p, w.mean.p, w.tw.p, w.scratch.p, averages, R, D, 0, 0, fl, ff,
                     center};
    unsigned fin_launches = 1;
    fa.tiles = (unsigned)((npix + 255) / 256);
    avg_mean_kernel<<<R * fa.tiles, 256, 0, st>>>(fa);
    const unsigned fin_threads = (2 * H + 31) / 32 * 32;
    const size_t tw_bytes = ((D + 1) & ~1u) * sizeof(float2);
    const size_t row_smem = tw_bytes + 2 * sizeof(float) * (K + 1) * kFinPitch;
    const size_t col_smem = tw_bytes + sizeof(float4) * (K + 1) * kFinColumns + sizeof(float2) * D * kFinColPitch;
    const unsigned row_tiles = (D + kFinRows - 1) / kFinRows, col_tiles = (H + kFinColumns - 1) / kFinColumns;
    for (unsigned r0 = 0; spectra && r0 < R; r0 += fin_groups) {
        const unsigned n = std::min(fin_groups, R - r0);
        fa.r0 = r0;
        fa.tiles = row_tiles;
        avg_rows_kernel<<<n * row_tiles, fin_threads, row_smem, st>>>(fa);
        fa.tiles = col_tiles;
        avg_cols_kernel<<<n * col_tiles, fin_threads, col_smem, st>>>(fa);
        fa.tiles = row_tiles;
        avg_inverse_kernel<<<n * row_tiles, fin_threads, row_smem, st>>>(fa);
        fin_launches += 3;
    }
    g_kernel_launches.fetch_add(7 + fin_launches, std::memory_order_relaxed);
    AV_CK(cudaGetLastError());
    AV_CK(cudaMemcpyAsync(w.h_err, w.err.p, kErrWords * sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    AV_CK(cudaStreamSynchronize(st));
    char msg[256];
    if (w.h_err[kErrBad]) {
        snprintf(msg, sizeof(msg), "class_averages: %u belongsto entries outside [0, %u), the first at particle %u",
                 w.h_err[kErrBad], R, w.h_err[kErrBadFirst]);
        return fail(2, msg);
    }
    if (w.h_err[kErrWait])
        return fail(1, "class_averages: an image copy timed out (bounded wait ran out)");
    if (w.h_err[kErrEmpty]) {
        snprintf(msg, sizeof(msg), "class_averages: %u groups have no members, the first is group %u",
                 w.h_err[kErrEmpty], w.h_err[kErrEmptyFirst]);
        return fail(2, msg);
    }
    return 0;
}
