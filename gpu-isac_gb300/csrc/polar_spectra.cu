// polar_spectra.cu -- polar resampling, per-image normalisation and per-ring
// real FFT of images (one CTA per image x shift), written straight in the
// basis the CCF contraction consumes.
//
// Reference semantics: cu_resample_to_polar (cuda/gpu_aln_noref.cu:1221-1354)
// followed by the in-place R2C cuFFT of every ring (:2121-2125).
//
// Output, per (image, shift) row, [ring][slot] float2:
//   slot k = 1..127 holds F[k]; slot 0 holds (F[0], F[128]) (both real);
//   subjects store (Re+Im, Re-Im)            of that pair of numbers,
//   references store (r+1) * (Re+Im, Re-Im)  (the ring weight folded in).
// With refs (u, v) and subjects (a, b) the four sums sum_r u a, u b, v b, v a
// are exactly Re/Im of Z[k] = O[k] + i M[k] and of Z[256-k], the spectrum
// whose inverse FFT gives the normal (real part) and mirrored (imaginary
// part) correlation at once.
#include <algorithm>
#include <map>
#include <mutex>
#include <utility>

#include "gpuisac_device.cuh"
#include "gpuisac_kernels.h"

namespace gpuisac {

std::atomic<unsigned long long> g_kernel_launches{0};

namespace {
std::mutex g_optin_mu;
std::map<std::pair<int, const void*>, int> g_optin; // (device, kernel) -> bytes opted in
} // namespace

cudaError_t opt_in_smem(const void* kernel, int bytes)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return e;
    std::lock_guard<std::mutex> lk(g_optin_mu);
    auto it = g_optin.find({dev, kernel});
    if (it != g_optin.end() && it->second >= bytes)
        return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess)
        g_optin[{dev, kernel}] = bytes;
    return e;
}

int smem_optin_max()
{
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return v;
}

// split (x, y) into BF16 hi = rn(x), rn(y) and lo = rn(x - hi) (x - hi is exact
// in FP32), each pair packed with x in the low half
__device__ __forceinline__ void bf16_split2(float x, float y, uint32_t& hi, uint32_t& lo)
{
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(y), "f"(x));
    const float dx = x - __uint_as_float(hi << 16), dy = y - __uint_as_float(hi & 0xFFFF0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(dy), "f"(dx));
}

constexpr bool kSpectraPacked = false; // scalar radix-4 sums: fewer live registers

// One CTA of 256 threads per row.  Sampling: thread tid takes angle tid of every
// ring; two rings' samples sit side by side in shared memory as the complex
// input of one FFT (one 8-byte store and load per pair of samples).  FFT: 16
// groups of 16 threads take the ring pairs in turn; the two real spectra are
// unpacked by shuffle (slot k needs Z[256 - k], which lane 16 - l holds).
//
// What bounds it: latency and the shared-memory pipe, not DRAM (76^2, 35 rings:
// 36 KB written per row).  The texture unit's own floor is 8,960 samples at 4
// a cycle, 2,240 of the ~5,400 cycles an SM spends per row.  Measured (GB300,
// kernel launch, 73,500 rows of 35 rings / 24,300 of 61): 28.0 / 66.2 ns per
// row with the offsets read from a template in memory (its L2 fetch before
// every texture fetch), the twiddles through a 256-entry table (2.8-way bank
// conflicts) and the spectrum written back and re-read for the unpacking;
// 17.5 / 32.5 ns with the offsets computed, a padded twiddle row per lane,
// samples stored in pairs and the unpacking by shuffle.  Sampling loops
// unrolled by 2, 3, 6 or 8 pairs: 18.2, 17.9, 18.2, 17.4 (61 rings: 35.0,
// 32.9, 31.4, 33.6); 4 CTAs per SM with 64 registers: 18.9.
//
// kOperand: the spectra go to shared memory and leave as BF16 hi/lo
// tensor-core operands (OperandLayout) instead of FP32 rows.  kTex: the stack
// has textures (the texture unit samples), else its emulation.
template <bool kOperand, bool kTex>
__device__ __forceinline__ void
polar_spectra_body(const StackDesc& st, const float2* __restrict__ dirs, const float2* __restrict__ twiddle,
                   unsigned ring_num, const int2* __restrict__ shift_int, unsigned n_shift,
                   const float2* __restrict__ base, unsigned img0, unsigned n_img, int is_ref,
                   float2* __restrict__ out, const unsigned* __restrict__ img_list,
                   const unsigned long long* __restrict__ tex_objs, const OperandLayout& opnd, unsigned row)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // ring pair p's samples (ring 2p, ring 2p + 1) at polar[p * kPairStride +
    // angle]; once a pair is in registers its region is the FFT workspace
    float2* polar = reinterpret_cast<float2*>(smem_raw);
    const unsigned n_pairs = (ring_num + 1) / 2;
    float2* tw = polar + n_pairs * kPairStride;              // [16][kTwRow] per FFT lane
    double* red = reinterpret_cast<double*>(tw + 16 * kTwRow); // 2 x 8 warps + 2

    const unsigned img_local = row / n_shift;
    const unsigned s = row - img_local * n_shift;
    if (img_local >= n_img)
        return;
    // output row i holds image img0 + i, or img_list[i] when a list is given
    const unsigned img = img_list ? img_list[img_local] : img0 + img_local;
    const int tid = threadIdx.x;
    const int g = tid >> 4; // FFT group 0..15
    const int l = tid & 15;

    tw[g * kTwRow + l] = twiddle[(g * l) & (kRingLen - 1)]; // lane g's forward twiddles, row g

    // ---- sampling positions exactly as the reference computes them ----
    const int2 sh = shift_int[s];
    const float* bx = base ? &base[img].x : nullptr;
    const float* by = base ? &base[img].y : nullptr;
    const TexPlacement place = tex_place(st, img);
    const float yoff = (float)(place.local * st.dim);
    const float2 cnt = make_float2(centre_coord(st.dim, sh.x, bx), yoff + centre_coord(st.dim, sh.y, by));
    const cudaTextureObject_t tobj = kTex ? (cudaTextureObject_t)__ldg(tex_objs + place.tex_id) : 0;
    const float2 dir = GPUISAC_IN_BOUNDS(kChkSpectraTmpl, tid, kRingLen) ? __ldg(&dirs[tid]) : make_float2(0.f, 0.f);
    const RingScale scale(ring_num);
    auto sample = [&](float radius) -> float {
        const float2 p = __fadd2_rn(cnt, scale.offset(dir, radius));
        return kTex ? tex2D<float>(tobj, p.x, p.y) : tex_sample(st, place, p.x, p.y);
    };

    // FP32 ring-weighted partial sums, reduced in FP32 across each warp, feed
    // the image mean / deviation (the eight warp sums are added in FP64)
    float s1 = 0.f, s2 = 0.f;
    auto add = [&](float w, float v) {
        s1 += w * v;
        s2 += w * v * v;
    };
    const unsigned n_full = ring_num >> 1;
#pragma unroll 4
    for (unsigned pr = 0; pr < n_full; pr++) {
        const float w = (float)(2 * pr + 1);
        const float va = sample(w), vb = sample(w + 1.f);
        polar[pr * kPairStride + tid] = make_float2(va, vb);
        add(w, va);
        add(w + 1.f, vb);
    }
    if (ring_num & 1u) {
        const float va = sample((float)ring_num);
        polar[n_full * kPairStride + tid] = make_float2(va, 0.f);
        add((float)ring_num, va);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        s1 += __shfl_xor_sync(0xffffffffu, s1, off);
        s2 += __shfl_xor_sync(0xffffffffu, s2, off);
    }
    const double d1 = s1, d2 = s2;
    const int warp = tid >> 5, lane = tid & 31;
    if (lane == 0) {
        red[warp] = d1;
        red[8 + warp] = d2;
    }
    __syncthreads();
    if (tid == 0) {
        double a = 0.0, q = 0.0;
        for (int w = 0; w < 8; w++) {
            a += red[w];
            q += red[8 + w];
        }
        // avg = sum (r+1) A_r / (L sum (r+1)); same for the squares (noref.cu:1314-1337)
        double nn = 0.5 * (double)ring_num * (double)(ring_num + 1) * (double)kRingLen;
        double avg = a / nn, msq = q / nn;
        double sd = sqrt(fabs(msq - avg * avg));
        // stored as the floats every thread uses (one conversion, not 256)
        float* redf = reinterpret_cast<float*>(red + 16);
        redf[0] = (float)avg;
        redf[1] = (float)(1.0 / (sd + 0.0000001));
    }
    __syncthreads();
    const float avg_f = reinterpret_cast<const float*>(red + 16)[0];
    const float inv_f = reinterpret_cast<const float*>(red + 16)[1];

    // ---- per-ring FFT, two rings per complex 256-point FFT ----
    const unsigned gmask = 0xffffu << (tid & 16);
    const int partner = (16 - l) & 15;
    float2* out_row = out + (size_t)row * ring_num * kSlots;
    for (unsigned pr = g; pr < n_pairs; pr += 16) {
        const unsigned ra = 2 * pr, rb = 2 * pr + 1;
        const bool has_b = rb < ring_num;
        float2* gws = polar + pr * kPairStride;
        float2 x[16];
#pragma unroll
        for (int m = 0; m < 16; m++) {
            const float2 v = gws[l + 16 * m];
            x[m] = make_float2((v.x - avg_f) * inv_f, has_b ? (v.y - avg_f) * inv_f : 0.f);
        }
        __syncwarp(gmask); // the pair's samples are read before its region turns workspace
        fft256_group_twl<-1, kSpectraPacked>(x, gws, tw + l * kTwRow, gmask);
        // x[perm16(k2)] = Z[l + 16 k2]: unpack the two real spectra into slots
        // k = l + 16 i (i = 0..7); Z[256 - k] is entry 15 - i of lane 16 - l
        // (lane 0: its own entry 16 - i)
        const float wa = (float)(ra + 1), wb = (float)(rb + 1);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float2 z = x[perm16(i)];
            const float2 zs = x[perm16(15 - i)];
            float2 zc = make_float2(__shfl_sync(gmask, zs.x, partner, 16), __shfl_sync(gmask, zs.y, partner, 16));
            if (l == 0)
                zc = x[perm16(i == 0 ? 8 : 16 - i)]; // (slot 0: Z[128])
            // F_a = (Z[k] + conj Z[256-k]) / 2 ; F_b = (Z[k] - conj Z[256-k]) / (2i)
            float2 fa = make_float2(0.5f * (z.x + zc.x), 0.5f * (z.y - zc.y));
            float2 fb = make_float2(0.5f * (z.y + zc.y), -0.5f * (z.x - zc.x));
            if (i == 0 && l == 0) {
                // slot 0 carries (F[0], F[128]); both are real
                fa = make_float2(z.x, zc.x);
                fb = make_float2(z.y, zc.y);
            }
            const int k = l + 16 * i;
            float2 oa = make_float2(fa.x + fa.y, fa.x - fa.y), ob = make_float2(fb.x + fb.y, fb.x - fb.y);
            if (is_ref) {
                oa = make_float2(wa * oa.x, wa * oa.y);
                ob = make_float2(wb * ob.x, wb * ob.y);
            }
            if (kOperand) {
                // the pair's region takes its two rings' spectra: ring ra at
                // [0, 128), ring rb at [128, 256) (zero for a missing ring)
                gws[k] = oa;
                gws[kSlots + k] = has_b ? ob : make_float2(0.f, 0.f);
            } else {
                [[maybe_unused]] const size_t n_out = (size_t)n_img * n_shift * ring_num * kSlots;
                [[maybe_unused]] const size_t at = (size_t)row * ring_num * kSlots + ra * kSlots + k;
                if (GPUISAC_IN_BOUNDS(kChkSpectraOut, at, n_out))
                    out_row[ra * kSlots + k] = oa;
                if (has_b && GPUISAC_IN_BOUNDS(kChkSpectraOut, at + kSlots, n_out))
                    out_row[rb * kSlots + k] = ob;
            }
        }
    }
    if (!kOperand)
        return;
    __syncthreads();
    // ---- write-out as BF16 hi/lo operand rows ----
    // One (slot, K group, a or b) per thread, a and b on neighbouring lanes: a
    // store instruction then touches 16 lines of 32 bytes each instead of 32
    // lines twice, which is what bounds this phase (slots lie 10 to 20 KB apart):
    // 32.3 -> 25.5 ns per row of 35 rings, 56.0 -> 44.1 of 61 (5 CTAs per SM
    // instead of 4: 26.1, 47.2).
    const unsigned tile = is_ref ? img_local / opnd.block : img_local * opnd.n_blocks + s / opnd.block;
    const unsigned orow = 2 * (is_ref ? img_local % opnd.block : s % opnd.block); // a / u; +1: b / v
    unsigned char* tb = opnd.base + (size_t)tile * opnd.tile_bytes() + (orow >> 3) * 128 + (orow & 7) * 16;
    const size_t sb = opnd.slot_bytes(), hb = (size_t)opnd.kg * opnd.rg * 128, kb = (size_t)opnd.rg * 128;
    const float* spec = reinterpret_cast<const float*>(polar);
    for (unsigned it = tid; it < 2 * kSlots * opnd.kg; it += 256) {
        const unsigned c = it & 1u, k = (it >> 1) & (kSlots - 1), kgi = it >> 8;
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float v[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const unsigned r = 8 * kgi + 2 * j + h;
                v[h] = r < ring_num ? spec[2 * ((r >> 1) * kPairStride + (r & 1) * kSlots + k) + c] : 0.f;
            }
            bf16_split2(v[0], v[1], hi[j], lo[j]);
        }
        unsigned char* p = tb + k * sb + kgi * kb + 16 * c;
        [[maybe_unused]] const size_t n_tiles =
            is_ref ? (n_img + opnd.block - 1) / opnd.block : (size_t)n_img * opnd.n_blocks;
        if (!GPUISAC_IN_BOUNDS(kChkOperandOut, (size_t)(p - opnd.base) + hb + 15, n_tiles * opnd.tile_bytes()))
            continue;
        *reinterpret_cast<uint4*>(p) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(p + hb) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
}

template <bool kTex>
__global__ void __launch_bounds__(256, 5)
polar_spectra_kernel(StackDesc st, const float2* __restrict__ dirs, const float2* __restrict__ twiddle,
                     unsigned ring_num, const int2* __restrict__ shift_int, unsigned n_shift,
                     const float2* __restrict__ base, unsigned img0, unsigned n_img, int is_ref,
                     float2* __restrict__ out, const unsigned* __restrict__ img_list,
                     const unsigned long long* __restrict__ tex_objs)
{
    polar_spectra_body<false, kTex>(st, dirs, twiddle, ring_num, shift_int, n_shift, base, img0, n_img, is_ref, out,
                                    img_list, tex_objs, OperandLayout(), blockIdx.x);
}

// The same rows for a table of jobs (SpectraJobs), one CTA per row, the row
// count read from device memory so that a recorded launch (grid = the
// capacity) serves any table the buffers hold.  A row's job: the lookup entry
// of its block of kJobLutRows rows (the job holding the block's first row),
// then forward over the jobs that start inside the block.
template <bool kTex>
__global__ void __launch_bounds__(256, 5)
polar_spectra_jobs_kernel(const SpectraJob* __restrict__ jobs, const unsigned* __restrict__ hdr,
                          const unsigned* __restrict__ lut, const float2* __restrict__ dirs,
                          const float2* __restrict__ twiddle, unsigned ring_num)
{
    const unsigned row = blockIdx.x;
    if (row >= hdr[2])
        return;
    const unsigned last = hdr[0] + hdr[1] - 1;
    unsigned j = lut[hdr[3] + row / kJobLutRows];
    while (j < last && jobs[j + 1].row_begin <= row)
        j++;
    const SpectraJob& jb = jobs[j];
    polar_spectra_body<false, kTex>(jb.st, dirs, twiddle, ring_num, jb.shift_int, jb.n_shift, jb.base, jb.img0,
                                    jb.n_img, jb.is_ref, jb.out, nullptr, jb.tex_objs, OperandLayout(),
                                    row - jb.row_begin);
}

template <bool kTex>
__global__ void __launch_bounds__(256, 4)
polar_operands_kernel(StackDesc st, const float2* __restrict__ dirs, const float2* __restrict__ twiddle,
                      unsigned ring_num, const int2* __restrict__ shift_int, unsigned n_shift,
                      const float2* __restrict__ base, unsigned img0, unsigned n_img, int is_ref,
                      OperandLayout opnd, const unsigned long long* __restrict__ tex_objs)
{
    polar_spectra_body<true, kTex>(st, dirs, twiddle, ring_num, shift_int, n_shift, base, img0, n_img, is_ref,
                                   nullptr, nullptr, tex_objs, opnd, blockIdx.x);
}

GPUISAC_CHECKED_READER(checked_read_spectra)

cudaError_t launch_polar_spectra(const StackDesc& st, const float2* dirs, const float2* twiddle,
                                 unsigned ring_num, const int2* shift_int, unsigned n_shift,
                                 const float2* base, unsigned img0, unsigned n_img, int is_ref,
                                 float2* out, cudaStream_t stream, const unsigned* img_list,
                                 const unsigned long long* tex_objs)
{
    if (n_img == 0 || n_shift == 0)
        return cudaSuccess;
    size_t smem = polar_spectra_smem_bytes(ring_num);
    auto* const kernel = tex_objs ? polar_spectra_kernel<true> : polar_spectra_kernel<false>;
    cudaError_t e = opt_in_smem_k(kernel, polar_spectra_smem_bytes(kMaxRingNum));
    if (e != cudaSuccess)
        return e;
    unsigned rows = n_img * n_shift;
    kernel<<<rows, 256, smem, stream>>>(st, dirs, twiddle, ring_num, shift_int, n_shift, base,
                                                       img0, n_img, is_ref, out, img_list, tex_objs);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError();
}

cudaError_t launch_polar_spectra_jobs(const SpectraJob* jobs, const unsigned* hdr, const unsigned* lut,
                                      const float2* dirs, const float2* twiddle, unsigned ring_num, unsigned grid,
                                      cudaStream_t stream, bool textures)
{
    if (grid == 0)
        return cudaSuccess;
    auto* const kernel = textures ? polar_spectra_jobs_kernel<true> : polar_spectra_jobs_kernel<false>;
    cudaError_t e = opt_in_smem_k(kernel, polar_spectra_smem_bytes(kMaxRingNum));
    if (e != cudaSuccess)
        return e;
    kernel<<<grid, 256, polar_spectra_smem_bytes(ring_num), stream>>>(jobs, hdr, lut, dirs, twiddle, ring_num);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError();
}

cudaError_t launch_polar_operands(const StackDesc& st, const float2* dirs, const float2* twiddle,
                                  unsigned ring_num, const int2* shift_int, unsigned n_shift,
                                  const float2* base, unsigned img0, unsigned n_img, int is_ref,
                                  const OperandLayout& opnd, cudaStream_t stream,
                                  const unsigned long long* tex_objs)
{
    if (n_img == 0 || n_shift == 0)
        return cudaSuccess;
    if (!opnd.base || opnd.block == 0 || opnd.kg * 8 < ring_num || (is_ref && n_shift != 1) ||
        opnd.rg * 8 < 2 * opnd.block || (!is_ref && opnd.block * opnd.n_blocks < n_shift))
        return cudaErrorInvalidValue;
    size_t smem = polar_spectra_smem_bytes(ring_num);
    auto* const kernel = tex_objs ? polar_operands_kernel<true> : polar_operands_kernel<false>;
    cudaError_t e = opt_in_smem_k(kernel, polar_spectra_smem_bytes(kMaxRingNum));
    if (e != cudaSuccess)
        return e;
    unsigned rows = n_img * n_shift;
    kernel<<<rows, 256, smem, stream>>>(st, dirs, twiddle, ring_num, shift_int, n_shift, base, img0, n_img, is_ref,
                                        opnd, tex_objs);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError();
}

} // namespace gpuisac
