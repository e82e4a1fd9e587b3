// ring512.cu -- the multi-reference alignment with 512 samples per ring.
//
// The reference's GPU driver fixes the ring length at 256
// (bin/sp_isac2_gpu.py:113); its library takes the length from
// cfg->ring_len, and Numrinit (bin/sp_isac_alignment.py:713-747) gives a
// maximum ring length of 512 for a last ring of 41..81 (61 rings at 128^2).
// These kernels run the same semantics -- the reference's sample positions,
// texture filtering, normalisation (cuda/gpu_aln_noref.cu:1221-1354), ring
// weights (r+1) and CCF of both mirrors (:1483-1537), first-maximum scan and
// 7-point parabola (:1667-1794) -- at L = 512, in FP32 on the CUDA cores.
//
// Layouts: a spectra row (image x shift) is [ring][256 slots] float2 in the
// basis of the 256-sample kernels (slot k = 1..255 holds F[k], slot 0 holds
// (F[0], F[256]); subjects (Re+Im, Re-Im), references (r+1)(Re+Im, Re-Im)).
// A 512-point FFT is two 256-point FFTs of 16-thread groups (even and odd
// samples) and one radix-2 step.
//
// Work: spectra, one CTA of 512 threads per row.  CCF, two kernels per chunk of
// particles: the ring-summed contraction as a register-tiled product (rows =
// particle x shift against references, per slot) that writes the four ring
// sums of every pair and slot (4 KB a pair) to device memory, then a warp per
// pair and shift for the inverse FFT and the peak search.
#include <cuda_runtime.h>

#include <algorithm>

#include "ccf_device.cuh"
#include "gpuisac_kernels.h"

namespace gpuisac {
namespace {

constexpr int kL = kRingLen512;  // samples per ring
constexpr int kS = kSlots512;    // spectrum slots per ring
constexpr int kPair = 544;       // float2 per ring-pair region: two rings' samples (512), or two FFT workspaces (2 x 272)

// One CTA of 512 threads per row: thread tid samples angle tid of every ring,
// two rings' samples side by side as the complex input of one 512-point FFT;
// 32 groups of 16 threads take the ring pairs.  One CTA fills an SM's shared
// memory (143 KB at 61 rings), so its 16 warps are all that hides the texture
// latency (8 warps, with the offsets read from memory, the samples of a pair
// in separate planes and the spectrum re-read for the unpacking: 308 ns per
// row of 61 rings, now 101).  The sums of the mean and deviation are added in
// a fixed order (thread t < 256: ring by ring, angle t then t + 256).
template <bool kTex>
__global__ void __launch_bounds__(512, 1)
polar_spectra512_kernel(StackDesc st, const float2* __restrict__ dirs, const float2* __restrict__ tw512,
                        unsigned ring_num, const int2* __restrict__ shift_int, unsigned n_shift,
                        const float2* __restrict__ base, unsigned img0, unsigned n_img, int is_ref,
                        float2* __restrict__ out, const unsigned long long* __restrict__ tex_objs)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* polar = reinterpret_cast<float2*>(smem_raw); // [pair][kPair]: samples (ring a, ring b), then workspaces
    const unsigned n_pairs = (ring_num + 1) / 2;
    float2* tw = polar + (size_t)n_pairs * kPair;          // [256] e^(-2 pi i e / 512)
    float2* twl = tw + 256;                                // [16][kTwRow] e^(-2 pi i l j / 256)
    double* red = reinterpret_cast<double*>(twl + 16 * kTwRow); // 2 x 8 warps + 2

    const unsigned row = blockIdx.x;
    const unsigned img_local = row / n_shift;
    const unsigned s = row - img_local * n_shift;
    if (img_local >= n_img)
        return;
    const unsigned img = img0 + img_local;
    const int tid = threadIdx.x;
    const int g = tid >> 4, l = tid & 15;
    if (tid < 256) {
        tw[tid] = tw512[tid];
        twl[g * kTwRow + l] = tw512[2 * ((g * l) & 255)];
    }

    // sampling positions as the 256-sample kernel computes them
    const int2 sh = shift_int[s];
    const float* bx = base ? &base[img].x : nullptr;
    const float* by = base ? &base[img].y : nullptr;
    const TexPlacement place = tex_place(st, img);
    const float yoff = (float)(place.local * st.dim);
    const float2 cnt = make_float2(centre_coord(st.dim, sh.x, bx), yoff + centre_coord(st.dim, sh.y, by));
    const cudaTextureObject_t tobj = kTex ? (cudaTextureObject_t)__ldg(tex_objs + place.tex_id) : 0;
    const float2 dir = __ldg(&dirs[tid]);
    const RingScale scale(ring_num);
    auto sample = [&](float radius) -> float {
        const float2 p = __fadd2_rn(cnt, scale.offset(dir, radius));
        return kTex ? tex2D<float>(tobj, p.x, p.y) : tex_sample(st, place, p.x, p.y);
    };
    const unsigned n_full = ring_num >> 1;
#pragma unroll 8
    for (unsigned pr = 0; pr < n_full; pr++) {
        const float w = (float)(2 * pr + 1);
        const float va = sample(w), vb = sample(w + 1.f);
        polar[pr * kPair + tid] = make_float2(va, vb);
    }
    if (ring_num & 1u)
        polar[n_full * kPair + tid] = make_float2(sample((float)ring_num), 0.f);
    __syncthreads();
    if (tid < 256) {
        float s1 = 0.f, s2 = 0.f;
        auto add = [&](float w, float v) {
            s1 += w * v;
            s2 += w * v * v;
        };
#pragma unroll 4
        for (unsigned pr = 0; pr < n_full; pr++) {
            const float2 v0 = polar[pr * kPair + tid], v1 = polar[pr * kPair + tid + 256];
            const float w = (float)(2 * pr + 1);
            add(w, v0.x);
            add(w, v1.x);
            add(w + 1.f, v0.y);
            add(w + 1.f, v1.y);
        }
        if (ring_num & 1u) {
            add((float)ring_num, polar[n_full * kPair + tid].x);
            add((float)ring_num, polar[n_full * kPair + tid + 256].x);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            s1 += __shfl_xor_sync(0xffffffffu, s1, off);
            s2 += __shfl_xor_sync(0xffffffffu, s2, off);
        }
        if ((tid & 31) == 0) {
            red[tid >> 5] = s1;
            red[8 + (tid >> 5)] = s2;
        }
    }
    __syncthreads();
    if (tid == 0) {
        double a = 0.0, q = 0.0;
        for (int w = 0; w < 8; w++) {
            a += red[w];
            q += red[8 + w];
        }
        // avg = sum (r+1) A_r / (L sum (r+1)); the same for the squares
        const double nn = 0.5 * (double)ring_num * (double)(ring_num + 1) * (double)kL;
        const double avg = a / nn, msq = q / nn;
        const double sd = sqrt(fabs(msq - avg * avg));
        float* redf = reinterpret_cast<float*>(red + 16);
        redf[0] = (float)avg;
        redf[1] = (float)(1.0 / (sd + 0.0000001));
    }
    __syncthreads();
    const float avg_f = reinterpret_cast<const float*>(red + 16)[0];
    const float inv_f = reinterpret_cast<const float*>(red + 16)[1];

    // two rings per complex 512-point FFT: z = ring a + i ring b
    const unsigned gmask = 0xffffu << (tid & 16);
    const int partner = (16 - l) & 15;
    float2* out_row = out + (size_t)row * ring_num * kS;
    for (unsigned pr = g; pr < n_pairs; pr += 32) {
        const unsigned ra = 2 * pr, rb = 2 * pr + 1;
        const bool has_b = rb < ring_num;
        float2* ws = polar + pr * kPair;
        float2 xe[16], xo[16];
#pragma unroll
        for (int m = 0; m < 16; m++) {
            const float4 v = reinterpret_cast<const float4*>(ws)[l + 16 * m]; // samples 2 (l + 16 m) and the next
            xe[m] = make_float2((v.x - avg_f) * inv_f, has_b ? (v.y - avg_f) * inv_f : 0.f);
            xo[m] = make_float2((v.z - avg_f) * inv_f, has_b ? (v.w - avg_f) * inv_f : 0.f);
        }
        __syncwarp(gmask); // the pair's samples are read before its region turns workspace
        fft256_group_twl<-1, false>(xe, ws, twl + l * kTwRow, gmask);
        fft256_group_twl<-1, false>(xo, ws, twl + l * kTwRow, gmask);
        // Z[k] = E[k] + w^k O[k], Z[k + 256] = E[k] - w^k O[k]
#pragma unroll
        for (int k2 = 0; k2 < 16; k2++) {
            const float2 e = xe[perm16(k2)], o = cmul(xo[perm16(k2)], tw[l + 16 * k2]);
            xe[perm16(k2)] = cadd(e, o);
            xo[perm16(k2)] = csub(e, o);
        }
        const float wa = (float)(ra + 1), wb = (float)(rb + 1);
        // slots k = l + 16 i: Z[512 - k] is the minus half's entry 256 - k --
        // entry 15 - i of lane 16 - l (lane 0: its own entry 16 - i)
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int k = l + 16 * i;
            const float2 z = xe[perm16(i)];
            const float2 zs = xo[perm16(15 - i)];
            float2 zc = make_float2(__shfl_sync(gmask, zs.x, partner, 16), __shfl_sync(gmask, zs.y, partner, 16));
            if (l == 0)
                zc = xo[perm16(i == 0 ? 0 : 16 - i)]; // (slot 0: Z[256])
            float2 fa = make_float2(0.5f * (z.x + zc.x), 0.5f * (z.y - zc.y));
            float2 fb = make_float2(0.5f * (z.y + zc.y), -0.5f * (z.x - zc.x));
            if (i == 0 && l == 0) { // slot 0 carries (F[0], F[256]); both are real
                fa = make_float2(z.x, zc.x);
                fb = make_float2(z.y, zc.y);
            }
            float2 oa = make_float2(fa.x + fa.y, fa.x - fa.y), ob = make_float2(fb.x + fb.y, fb.x - fb.y);
            if (is_ref) {
                oa = make_float2(wa * oa.x, wa * oa.y);
                ob = make_float2(wb * ob.x, wb * ob.y);
            }
            [[maybe_unused]] const size_t n_out = (size_t)n_img * n_shift * ring_num * kS;
            [[maybe_unused]] const size_t at = (size_t)row * ring_num * kS + ra * kS + k;
            if (GPUISAC_IN_BOUNDS(kChkR512Out, at, n_out))
                out_row[ra * kS + k] = oa;
            if (has_b && GPUISAC_IN_BOUNDS(kChkR512Out, at + kS, n_out))
                out_row[rb * kS + k] = ob;
        }
    }
}

// ---- contraction ----
// For every slot k: sums over the rings of rows (particle x shift, (a, b))
// against references ((u, v), ring weight folded in).  CTA: 32 slots x (8 kRs
// rows) x (4 kQs references), kRs kQs = 8 warps; a lane owns one slot, a warp
// an 8 x 4 tile of pairs: 128 accumulators for 12 float2 operands per ring.
// The operands of kRc rings at a time come to shared memory by cp.async, three
// stages deep.  Sums run ring by ring in order.
//
// What bounds it: FP32 FMA issue (62.5k FMA a pair at 61 rings; the FMA pipe is
// active 60 % of the cycles, issue 56 %, two warps a scheduler, one packed FMA
// per two cycles) beside shared memory at 12 x 8 bytes per 128 FMAs and thread.
// The row is 125 KB at 61 rings, too large to keep a reference and a shift group
// on the SM with the pairs' spectra as the 256-sample kernel does; one CTA per (particle, reference), re-reading every shift row for each
// reference with four accumulators a thread, was bound by the latency of those
// reads (issue 13 %).  Contraction, FFT and search of 300 x 60 pairs, 61
// rings, 25 shifts: 13.4 -> 2.15 ms; 100 x 200, 81 shifts: 41.0 -> 7.2 ms.
// Scalar FMAs instead of packed pairs 2.31; 16 warps with 4 x 4 tiles 2.30
// scalar, 2.45 packed; 12 warps 2.44; four stages, or one CTA per tile: 2.3.
// kQs: 4, 8 or 16 references per CTA, so that few references don't run mostly
// padding (3 references, 35 rings, 40 particles, 49 shifts: 0.20 -> 0.05 ms).
constexpr int kCr = 8, kCq = 4; // rows and references per warp
constexpr int kRc = 4;          // rings per stage
constexpr int kStages = 3;
constexpr int kSlotTile = 32;

template <int kQs>
struct Tile512 {
    static constexpr int kRs = 8 / kQs;
    static constexpr int kRows = kCr * kRs, kRefs = kCq * kQs;
    static constexpr int kStageElems = (kRows + kRefs) * kRc * kSlotTile; // float2
    static constexpr size_t kSmem = (size_t)kStages * kStageElems * sizeof(float2);
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool in)
{
    const uint32_t n = in ? 16u : 0u; // 0: zero-fill
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(n) : "memory");
}

// The CTAs are persistent: the stages run on from one tile (row tile,
// reference tile, slot tile; slots fastest, so that the CTAs of a moment share
// their rows in L2) to the next, the next tile's first operands in flight
// while this one's sums are written.
template <int kQs>
__global__ void __launch_bounds__(256, 1)
ccf_sums512_kernel(const float2* __restrict__ sbj_sp, const float2* __restrict__ ref_sp, unsigned ring_num,
                   unsigned n_shift, unsigned n_ref, unsigned n_rows, unsigned q_tiles, unsigned n_tiles,
                   float4* __restrict__ z)
{
    using T = Tile512<kQs>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* const stage0 = reinterpret_cast<float2*>(smem_raw); // [stage][row or ref][ring of the stage][32 slots]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned n_steps = (ring_num + kRc - 1) / kRc;
    auto decode = [&](unsigned tile, unsigned& k0, unsigned& q0, unsigned& r0) {
        constexpr unsigned kTiles = kS / kSlotTile;
        const unsigned rest = tile / kTiles, rt = rest / q_tiles;
        k0 = (tile - rest * kTiles) * kSlotTile;
        q0 = (rest - rt * q_tiles) * T::kRefs;
        r0 = rt * T::kRows;
    };

    // the next stage to load: step l_step of tile l_tile into buffer l_buf
    unsigned l_tile = blockIdx.x, l_step = 0, l_buf = 0, lk0, lq0, lr0;
    decode(l_tile, lk0, lq0, lr0);
    auto load_next = [&]() {
        if (l_tile < n_tiles) {
            float2* const sb = stage0 + l_buf * T::kStageElems;
            // 16 bytes = 2 slots: 16 pieces per (row or ref, ring)
            constexpr int kPieces = (T::kRows + T::kRefs) * kRc * (kSlotTile / 2);
            static_assert(kPieces % 256 == 0 && kRc == 4, "piece indexing");
#pragma unroll
            for (int i = 0; i < kPieces / 256; i++) {
                const int c = tid + 256 * i;
                const int piece = c & 15, rr = (c >> 4) & (kRc - 1), e = c >> 6;
                const unsigned ring = l_step * kRc + rr;
                const bool is_row = e < T::kRows;
                const unsigned at = is_row ? lr0 + e : lq0 + (e - T::kRows);
                const bool in = ring < ring_num && at < (is_row ? n_rows : n_ref) &&
                                GPUISAC_IN_BOUNDS(kChkR512Row, at, is_row ? n_rows : n_ref);
                const float2* src = (is_row ? sbj_sp : ref_sp);
                if (in)
                    src += ((size_t)at * ring_num + ring) * kS + lk0 + 2 * piece;
                cp_async16(sb + (e * kRc + rr) * kSlotTile + 2 * piece, src, in);
            }
            l_buf = l_buf + 1 == kStages ? 0 : l_buf + 1;
            if (++l_step == n_steps) {
                l_step = 0;
                l_tile += gridDim.x;
                decode(l_tile, lk0, lq0, lr0);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int st = 0; st < kStages - 1; st++)
        load_next();

    const int wr = warp % T::kRs, wq = warp / T::kRs;
    unsigned buf = 0;
    for (unsigned tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        f32x2 acc[kCr][kCq][2]; // (sum u a, sum u b), (sum v a, sum v b)
#pragma unroll
        for (int i = 0; i < kCr; i++)
#pragma unroll
            for (int q = 0; q < kCq; q++)
                acc[i][q][0] = acc[i][q][1] = 0;
        for (unsigned step = 0; step < n_steps; step++) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
            __syncthreads(); // this stage has landed; everyone is done with the one loaded next
            load_next();
            const f32x2* const sb = reinterpret_cast<const f32x2*>(stage0) + buf * T::kStageElems + lane;
            buf = buf + 1 == kStages ? 0 : buf + 1;
            const f32x2* const rows = sb + (wr * kCr) * kRc * kSlotTile;
            const f32x2* const refs = sb + (T::kRows + wq * kCq) * kRc * kSlotTile;
#pragma unroll 1 // (unrolled by 2 or 4: 2.20)
            for (int rr = 0; rr < kRc; rr++) {
                f32x2 a[kCr], u[kCq], v[kCq];
#pragma unroll
                for (int i = 0; i < kCr; i++)
                    a[i] = rows[(i * kRc + rr) * kSlotTile];
#pragma unroll
                for (int q = 0; q < kCq; q++)
                    splat_both(refs[(q * kRc + rr) * kSlotTile], u[q], v[q]);
                // (rings past the count are zero on both sides: an accumulator
                // that starts at +0 is never -0, so adding 0 leaves it as it was)
#pragma unroll
                for (int i = 0; i < kCr; i++)
#pragma unroll
                    for (int q = 0; q < kCq; q++) {
                        fma_f32x2(acc[i][q][0], u[q], a[i]);
                        fma_f32x2(acc[i][q][1], v[q], a[i]);
                    }
            }
        }
        unsigned k0, q0, r0;
        decode(tile, k0, q0, r0);
#pragma unroll
        for (int i = 0; i < kCr; i++) {
            const unsigned r = r0 + wr * kCr + i;
            if (r >= n_rows)
                break;
            const unsigned p = r / n_shift, s = r - p * n_shift;
#pragma unroll
            for (int q = 0; q < kCq; q++) {
                const unsigned qq = q0 + wq * kCq + q;
                const float2 ua = unpack_f32x2(acc[i][q][0]), va = unpack_f32x2(acc[i][q][1]);
                if (qq < n_ref)
                    z[(((size_t)p * n_ref + qq) * n_shift + s) * kS + k0 + lane] =
                        make_float4(ua.x, ua.y, va.y, va.x);
            }
        }
    }
}

// ---- inverse FFT + peak search ----
// One CTA per (particle, reference); its warps take the shifts in turn, each
// shift's 512-point inverse FFT as two 256-point ones: half-warp 0 the even
// outputs from Z[k] + Z[k + 256], half-warp 1 the odd ones from
// (Z[k] - Z[k + 256]) e^(2 pi i k / 512).  Bound by issue (two transforms and
// a search per 4 KB read).
constexpr int kFftWarps = 8;

__global__ void __launch_bounds__(32 * kFftWarps, 3)
zfft_peak512_kernel(const float4* __restrict__ z, const float2* __restrict__ tw512, unsigned n_shift, unsigned n_ref,
                    unsigned n_part, unsigned p_first, unsigned p_total, unsigned q_first, unsigned q_total,
                    const float2* __restrict__ shifts_f, const float2* __restrict__ base, float* __restrict__ d_out,
                    float4* __restrict__ peak_out)
{
    __shared__ float2 wsp[2 * kFftWarps][kPairStride];
    __shared__ float2 twl[16 * kTwRow]; // e^(+2 pi i l j / 256)
    __shared__ float2 twc[256];         // e^(+2 pi i k / 512)
    __shared__ PeakSlot slots[kFftWarps];

    const unsigned item = blockIdx.x;
    const unsigned p = item / n_ref, q = item - p * n_ref;
    if (p >= n_part)
        return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    {
        const float2 t = tw512[tid], u = tw512[2 * (((tid >> 4) * (tid & 15)) & 255)];
        twc[tid] = make_float2(t.x, -t.y);
        twl[(tid >> 4) * kTwRow + (tid & 15)] = make_float2(u.x, u.y * -1.f);
    }
    static_assert(32 * kFftWarps == 256, "one thread per twiddle");
    __syncthreads();
    const int half = lane >> 4, l = lane & 15;
    const unsigned gmask = 0xffffu << (lane & 16);
    float2* const ws = wsp[2 * warp + half];
    // running best of the shifts this warp searches (lanes 0..6 keep the 7
    // samples around it)
    float bv = -3.40282e+038f, nb = 0.f;
    unsigned bh = 0, bt = 0;
    for (unsigned s = warp; s < n_shift; s += kFftWarps) {
        const float4* zp = z + ((size_t)item * n_shift + s) * kS;
        float2 x[16];
#pragma unroll
        for (int m = 0; m < 16; m++) {
            const int k = l + 16 * m;
            // Z[k] is the first half of slot k, Z[512 - k] the second; slot 0
            // carried (F[0], F[256]): recover the two real products
            float2 z0, z1;
            if (m == 0 && l == 0) {
                const float4 e = __ldcs(zp);
                const float p1 = 0.25f * (e.x + e.y + e.z + e.w);
                const float p2 = 0.25f * (e.x - e.y + e.z - e.w);
                z0 = make_float2(p1, p1);
                z1 = make_float2(p2, p2);
            } else {
                z0 = __ldg(reinterpret_cast<const float2*>(zp + k));
                z1 = __ldg(reinterpret_cast<const float2*>(zp + kS - k) + 1);
            }
            x[m] = half ? cmul(csub(z0, z1), twc[k]) : cadd(z0, z1);
        }
        fft256_group_twl<+1>(x, ws, twl + l * kTwRow, gmask);
        // x[perm16(k2)] = c[2 (l + 16 k2) + half] = (normal, mirrored)
        // correlation: each mirror's maximum first, the index only when it
        // can beat the running best
        float vm[2] = {x[perm16(0)].x, x[perm16(0)].y};
#pragma unroll
        for (int k2 = 1; k2 < 16; k2++) {
            vm[0] = fmaxf(vm[0], x[perm16(k2)].x);
            vm[1] = fmaxf(vm[1], x[perm16(k2)].y);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            vm[0] = fmaxf(vm[0], __shfl_xor_sync(0xffffffffu, vm[0], off));
            vm[1] = fmaxf(vm[1], __shfl_xor_sync(0xffffffffu, vm[1], off));
        }
        // at equal maxima the normal one: its scan index is lower
        const bool mir = vm[1] > vm[0] || vm[0] != vm[0];
        const float v = mir ? vm[1] : vm[0];
        const unsigned hc = mir ? n_shift + s : s;
        if (v >= bv) { // (the same on every lane; false for NaN)
            unsigned t = 0xffffffffu;
#pragma unroll
            for (int k2 = 15; k2 >= 0; k2--)
                if ((mir ? x[perm16(k2)].y : x[perm16(k2)].x) == v)
                    t = 2 * (l + 16 * k2) + half;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
                t = min(t, __shfl_xor_sync(0xffffffffu, t, off));
            if (better(v, hc, t, bv, bh, bt)) {
                bv = v;
                bh = hc;
                bt = t;
                float* const wf = reinterpret_cast<float*>(wsp[2 * warp]); // 512 of the warp's 1,088 floats
                __syncwarp();
#pragma unroll
                for (int k2 = 0; k2 < 16; k2++)
                    wf[2 * (l + 16 * k2) + half] = mir ? x[perm16(k2)].y : x[perm16(k2)].x;
                __syncwarp();
                if (lane < 7)
                    nb = wf[(t + (unsigned)lane - 3u) & (kL - 1)];
                __syncwarp();
            }
        }
    }
    // merge the warps' bests and write the outputs
    const unsigned n_warps = min((unsigned)kFftWarps, n_shift);
    if ((unsigned)warp < n_warps) {
        if (lane == 0) {
            slots[warp].v = bv;
            slots[warp].h = bh;
            slots[warp].t = bt;
        }
        if (lane < 7)
            slots[warp].nb[lane] = nb;
    }
    __syncthreads();
    if (tid == 0) {
        unsigned best = 0;
        for (unsigned w = 1; w < n_warps; w++)
            if (better(slots[w].v, slots[w].h, slots[w].t, slots[best].v, slots[best].h, slots[best].t))
                best = w;
        const PeakSlot& ps = slots[best];
        const bool mirror = ps.h >= n_shift;
        const unsigned sidx = mirror ? ps.h - n_shift : ps.h;
        const unsigned pg = p_first + p;
        const float angle = peak_angle(ps.nb, ps.t, mirror, kL);
        const float bxv = base ? base[pg].x : 0.f;
        const float byv = base ? base[pg].y : 0.f;
        const float2 sf = shifts_f[sidx];
        const size_t o = (size_t)(q_first + q) * p_total + pg;
        if (GPUISAC_IN_BOUNDS(kChkR512Res, o, (size_t)q_total * p_total)) {
            d_out[o] = ps.v;
            peak_out[o] = make_float4(angle, bxv + sf.x, byv + sf.y, mirror ? 1.f : 0.f);
        }
    }
}

size_t spectra512_smem(unsigned ring_num)
{
    return (size_t)((ring_num + 1) / 2) * kPair * sizeof(float2) + (256 + 16 * kTwRow) * sizeof(float2) +
           24 * sizeof(double);
}

} // namespace

GPUISAC_CHECKED_READER(checked_read_ring512)

cudaError_t launch_polar_spectra512(const StackDesc& st, const float2* dirs, const float2* tw512, unsigned ring_num,
                                    const int2* shift_int, unsigned n_shift, const float2* base, unsigned img0,
                                    unsigned n_img, int is_ref, float2* out, cudaStream_t stream,
                                    const unsigned long long* tex_objs)
{
    if (n_img == 0 || n_shift == 0)
        return cudaSuccess;
    if (ring_num == 0 || ring_num > kMaxRingNum)
        return cudaErrorInvalidValue;
    auto* const kernel = tex_objs ? polar_spectra512_kernel<true> : polar_spectra512_kernel<false>;
    cudaError_t e = opt_in_smem_k(kernel, spectra512_smem(kMaxRingNum));
    if (e != cudaSuccess)
        return e;
    const size_t rows = (size_t)n_img * n_shift;
    if (rows > 0x7FFFFFFFull)
        return cudaErrorInvalidValue;
    kernel<<<(unsigned)rows, 512, spectra512_smem(ring_num), stream>>>(st, dirs, tw512, ring_num, shift_int, n_shift,
                                                                       base, img0, n_img, is_ref, out, tex_objs);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError();
}

template <int kQs>
static cudaError_t launch_sums512(const float2* sbj_sp, const float2* ref_sp, unsigned ring_num, unsigned n_shift,
                                  unsigned n_ref, unsigned n_rows, float4* z, cudaStream_t stream)
{
    using T = Tile512<kQs>;
    cudaError_t e = opt_in_smem_k(ccf_sums512_kernel<kQs>, T::kSmem);
    if (e != cudaSuccess)
        return e;
    const unsigned q_tiles = (n_ref + T::kRefs - 1) / T::kRefs, r_tiles = (n_rows + T::kRows - 1) / T::kRows;
    const size_t tiles = (size_t)q_tiles * r_tiles * (kS / kSlotTile);
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return e;
    if (tiles > 0x7FFFFFFFull)
        return cudaErrorInvalidValue; // (8 GB of ring sums hold fewer)
    ccf_sums512_kernel<kQs><<<(unsigned)std::min<size_t>(tiles, (size_t)std::max(sms, 1)), 256, T::kSmem, stream>>>(
        sbj_sp, ref_sp, ring_num, n_shift, n_ref, n_rows, q_tiles, (unsigned)tiles, z);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError();
}

cudaError_t launch_ccf_peak512(const float2* sbj_sp, const float2* ref_sp, const float2* tw512, unsigned ring_num,
                               unsigned n_shift, unsigned n_ref, unsigned n_part, unsigned p_first, unsigned p_total,
                               unsigned q_first, unsigned q_total, const float2* shifts_f, const float2* base,
                               float4* z, float* d_out, float4* peak_out, cudaStream_t stream)
{
    if (n_part == 0 || n_ref == 0)
        return cudaSuccess;
    if (ring_num == 0 || ring_num > kMaxRingNum || n_shift == 0)
        return cudaErrorInvalidValue;
    const size_t items = (size_t)n_part * n_ref;
    if (items > 0x7FFFFFFFull || (size_t)n_part * n_shift > 0x7FFFFFFFull)
        return cudaErrorInvalidValue;
    // references per CTA: a narrow tile for few references, else 16
    const unsigned rows = n_part * n_shift;
    cudaError_t e = n_ref <= 4   ? launch_sums512<1>(sbj_sp, ref_sp, ring_num, n_shift, n_ref, rows, z, stream)
                    : n_ref <= 8 ? launch_sums512<2>(sbj_sp, ref_sp, ring_num, n_shift, n_ref, rows, z, stream)
                                 : launch_sums512<4>(sbj_sp, ref_sp, ring_num, n_shift, n_ref, rows, z, stream);
    if (e != cudaSuccess)
        return e;
    zfft_peak512_kernel<<<(unsigned)items, 32 * kFftWarps, 0, stream>>>(z, tw512, n_shift, n_ref, n_part, p_first,
                                                                        p_total, q_first, q_total, shifts_f, base,
                                                                        d_out, peak_out);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError();
}

} // namespace gpuisac
