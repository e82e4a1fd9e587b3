// assign.cu -- equal-size assignment of particles to groups on the peak matrix
// d[ref][particle] the multi-reference alignment writes: the step ISAC runs
// right after the alignment (bin/sp_isac2_gpu.py:1114-1136, through EMAN2's
// Util::assign_groups on the host, after d has been copied off the GPU).
//
// The host algorithm takes (reference, particle) pairs in descending peak
// order (equal peaks: smaller pair index ref*nima + particle first) and puts a
// particle into the pair's group while the group has room: maxasi = nima/nref
// places, except the group that closes last, which also takes the
// nima % nref particles left over.  With a strict order on the pairs, that
// greedy result is the unique stable assignment of the ranking with capacity
// maxasi per group (no particle and group outside it prefer each other to
// their partners), which deferred acceptance finds in parallel:
//   round:  every unplaced particle proposes to its best group among those
//           whose threshold its pair beats (a scan of its column of d); every
//           group that received proposals keeps its maxasi best pairs, its
//           threshold becomes the maxasi-th best pair key, and the rest are
//           unplaced again;
//   end:    when a round turns nobody away (every round and what follows run in one
//           cooperative grid, up to 1,024 rounds a launch, or, where the steps are long,
//           each step as a launch of its own).  Every group then holds maxasi
//           particles; the one with the lowest threshold is the group the host
//           algorithm closes last, and the leftover particles join it.
// The result also comes out as the host function's list: each group's members
// in descending pair order, group after group, the leftovers in descending
// order of their pair with the last group, then that group's index.
//
// Pair keys are 64-bit: the peak's float bits mapped to an unsigned order
// (-0 taken as +0) above 0xFFFFFFFF - (ref*nima + particle), so that a larger
// key is an earlier pair; key 0 means "open" for a group threshold.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstdio>
#include <mutex>

#include "../../include/gpu_aln_pack.h"
#include "gpuisac_kernels.h"
#include "host_geometry.h"

namespace gpuisac {
namespace {

constexpr unsigned kThreads = 256;   // 8 warps: a group's selection, 32 particles x 8 row slices, ...
constexpr unsigned kRows = 8;        // row slices of d per particle in the proposal scan
// groups up to this many candidates select by counting in shared memory, others by
// digits: c^2 / 256 steps against two or three passes over c and 256 counters (20,000
// particles in 20 groups: 582 us in all when 1,024 candidates still counted, 181 now)
constexpr unsigned kSmallSel = 128;
constexpr unsigned kSparseDiv = 8;   // a round with at most nima / 8 particles to place uses the list form
// CTAs of the cooperative grid per SM: two meet faster (20,000 particles x 200 groups:
// 222 us against 238), four read the peaks of many particles faster (100,000 x 500: 614
// against 792)
constexpr unsigned kCtasPerSm = 2, kCtasPerSmWide = 4;
constexpr unsigned kWideTiles = 8; // tiles of 32 particles per SM from which on four
constexpr unsigned kMaxRounds = 1024; // per launch (a launch goes on where the last one stopped)
// tries of a grid barrier's wait, 0.23 us each.  At the first meeting of a launch CTAs
// may not have started (another stream's kernels hold their SMs): 15 seconds.  From then
// on all run, and no step of a call that takes this form lasts more than milliseconds:
// one second, as the other kernels' waits.
constexpr unsigned kStartTries = 1u << 26, kWaitTries = 1u << 22;
constexpr unsigned kErrNaN = 1u, kErrInternal = 2u, kErrWait = 4u;

// kScNext: particles turned away; kScTotal: bucketed members of a round;
// kScRounds: rounds done; kScBar: arrivals at the grid barrier
enum { kScNext = 0, kScErr, kScLast, kScLeft, kScTotal, kScRounds, kScBar = 32, kScCount };
constexpr unsigned kScWords = 32; // 64-bit words they take (the barrier's line apart, and nothing else on theirs)

__device__ __forceinline__ uint64_t pair_key(float v, uint32_t l)
{
    uint32_t u = __float_as_uint(v == 0.0f ? 0.0f : v);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return ((uint64_t)u << 32) | (uint64_t)(0xFFFFFFFFu - l);
}

// One call's arrays.  Those the kernel writes are read by plain loads after a grid
// barrier (no read-only path).
struct Assign {
    const float* d;
    size_t pitch;
    unsigned nref, nima, maxasi, extra;
    bool first;  // nobody has proposed yet
    int* belongsto;
    int* out;    // the list, or NULL
    uint64_t *theta, *pkey, *bk;
    unsigned *cnt, *touched, *off, *fill, *bp, *list, *sc;
    unsigned char* redo;
    int* assign;
    unsigned start_tries, wait_tries;
    unsigned stall; // failure-path tests only (gpuisac_test_stall_ccf): every meeting waits for one arrival too many
};

// All CTAs of the (cooperative) grid meet: what each wrote before is seen by all
// after.  False when the wait ran out in any of them that this one heard of: the
// caller returns (every other wait of the launch runs out as well).
__device__ bool grid_meet(const Assign& a, unsigned& target)
{
    __shared__ bool s_ok;
    __syncthreads();
    target += gridDim.x;
    if (threadIdx.x == 0) {
        unsigned *bar = a.sc + kScBar, seen = 0, tries = 0;
        const unsigned want = target + a.stall, limit = target == gridDim.x ? a.start_tries : a.wait_tries;
        __threadfence();
        atomicAdd(bar, 1u);
        while (true) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
            if ((int)(seen - want) >= 0 || ++tries > limit)
                break;
            __nanosleep(20);
        }
        s_ok = (int)(seen - want) >= 0;
        if (!s_ok)
            atomicOr(a.sc + kScErr, kErrWait);
        __threadfence();
    }
    __syncthreads();
    return s_ok;
}

__device__ __forceinline__ void propose_to(const Assign& a, unsigned p, int bg, uint64_t best)
{
    a.assign[p] = bg;
    a.pkey[p] = best;
    if (bg >= 0) {
        atomicAdd(a.cnt + bg, 1u);
        a.touched[bg] = 1u;
    }
}

// Each unplaced particle's best pair among the groups whose threshold it
// beats.  Tile = 32 consecutive particles x kRows row slices; the lanes of a
// warp read one row of d for the tile's unplaced particles, so that a round
// with few of them touches only the 32-byte sectors they share; a tile with
// none is passed over.  all: every particle (the first round); otherwise
// redo[p] = 1 marks the particles turned away last round (cleared here).
__device__ void propose_scan(const Assign& a, bool all)
{
    __shared__ uint64_t s_key[kRows][32];
    __shared__ int s_grp[kRows][32];
    const unsigned x = threadIdx.x & 31u, y = threadIdx.x >> 5;
    for (unsigned tile = blockIdx.x; tile < (a.nima + 31) / 32; tile += gridDim.x) {
        const unsigned p = tile * 32 + x;
        const bool live = p < a.nima && (all || a.redo[p]);
        if (!__syncthreads_or(live))
            continue;
        if (live && !all && y == 0)
            a.redo[p] = 0;
        uint64_t best = 0;
        int bg = -1;
        bool nan = false;
        if (live) {
            const float* col = a.d + p;
#pragma unroll 4
            for (unsigned g = y; g < a.nref; g += kRows) {
                const float v = __ldg(col + (size_t)g * a.pitch);
                nan |= (v != v);
                const uint64_t k = pair_key(v, g * a.nima + p);
                if (k > best && k > a.theta[g]) {
                    best = k;
                    bg = (int)g;
                }
            }
        }
        if (nan)
            atomicOr(a.sc + kScErr, kErrNaN);
        s_key[y][x] = best;
        s_grp[y][x] = bg;
        __syncthreads();
        if (y == 0 && live) {
#pragma unroll
            for (unsigned r = 1; r < kRows; r++)
                if (s_key[r][x] > best) {
                    best = s_key[r][x];
                    bg = s_grp[r][x];
                }
            propose_to(a, p, bg, best);
        }
        __syncthreads();
    }
}

// The list form of the proposal scan, for rounds with few particles to
// place: one warp per particle of list[0..n), its lanes striding over the
// rows of the particle's column, the best pair found by a warp reduction.
__device__ void propose_listed(const Assign& a, unsigned n)
{
    const unsigned lane = threadIdx.x & 31;
    for (unsigned i = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); i < n; i += gridDim.x * (kThreads / 32)) {
        const unsigned p = a.list[i];
        uint64_t best = 0;
        int bg = -1;
        bool nan = false;
        const float* col = a.d + p;
#pragma unroll 4
        for (unsigned g = lane; g < a.nref; g += 32) {
            const float v = __ldg(col + (size_t)g * a.pitch);
            nan |= (v != v);
            const uint64_t k = pair_key(v, g * a.nima + p);
            if (k > best && k > a.theta[g]) {
                best = k;
                bg = (int)g;
            }
        }
#pragma unroll
        for (unsigned o = 16; o > 0; o >>= 1) {
            const uint64_t ok = __shfl_xor_sync(0xFFFFFFFFu, best, o);
            const int og = __shfl_xor_sync(0xFFFFFFFFu, bg, o);
            if (ok > best) {
                best = ok;
                bg = og;
            }
        }
        if (__any_sync(0xFFFFFFFFu, nan) && lane == 0)
            atomicOr(a.sc + kScErr, kErrNaN);
        if (lane == 0) {
            a.redo[p] = 0;
            propose_to(a, p, bg, best);
        }
    }
}

// The k-th largest of c distinct keys (1 <= k <= c), by a radix select over
// the 8-bit digits from the top, in one CTA; stops early once one key is left
// in the selected bucket.
__device__ uint64_t kth_largest(const uint64_t* keys, unsigned c, unsigned k)
{
    __shared__ unsigned hist[256];
    __shared__ uint64_t s_prefix, s_found;
    __shared__ unsigned s_k, s_single;
    uint64_t prefix = 0, mask = 0;
    unsigned kk = k;
    for (int shift = 56; shift >= 0; shift -= 8) {
        for (unsigned i = threadIdx.x; i < 256; i += blockDim.x)
            hist[i] = 0;
        __syncthreads();
        for (unsigned i = threadIdx.x; i < c; i += blockDim.x) {
            const uint64_t v = keys[i];
            if ((v & mask) == prefix)
                atomicAdd(&hist[(unsigned)(v >> shift) & 255u], 1u);
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            // lane l has bins 255 - 8 l down to 248 - 8 l; the bin that holds the kk-th
            // largest is in the first lane whose sum from the top reaches kk
            const unsigned top = 255u - 8u * threadIdx.x;
            unsigned own = 0;
#pragma unroll
            for (unsigned i = 0; i < 8; i++)
                own += hist[top - i];
            unsigned acc = own;
#pragma unroll
            for (unsigned o = 1; o < 32; o <<= 1) {
                const unsigned up = __shfl_up_sync(0xFFFFFFFFu, acc, o);
                if (threadIdx.x >= o)
                    acc += up;
            }
            if (acc >= kk && acc - own < kk) {
                acc -= own;
                unsigned b = top;
                while (acc + hist[b] < kk)
                    acc += hist[b--];
                s_prefix = prefix | ((uint64_t)b << shift);
                s_k = kk - acc;
                s_single = hist[b] == 1u;
            }
        }
        __syncthreads();
        prefix = s_prefix;
        mask |= 0xFFull << shift;
        kk = s_k;
        if (s_single) {
            for (unsigned i = threadIdx.x; i < c; i += blockDim.x) {
                const uint64_t v = keys[i];
                if ((v & mask) == prefix)
                    s_found = v;
            }
            __syncthreads();
            return s_found;
        }
        __syncthreads();
    }
    return prefix;
}

// The k-th largest of c <= kSmallSel distinct keys: the one with exactly
// k - 1 larger keys, counted against a copy in shared memory.
__device__ uint64_t kth_largest_small(const uint64_t* keys, unsigned c, unsigned k)
{
    __shared__ uint64_t s_keys[kSmallSel];
    __shared__ uint64_t s_found;
    for (unsigned i = threadIdx.x; i < c; i += blockDim.x)
        s_keys[i] = keys[i];
    __syncthreads();
    for (unsigned i = threadIdx.x; i < c; i += blockDim.x) {
        const uint64_t v = s_keys[i];
        unsigned larger = 0;
#pragma unroll 8
        for (unsigned j = 0; j < c; j++)
            larger += s_keys[j] > v;
        if (larger == k - 1)
            s_found = v;
    }
    __syncthreads();
    return s_found;
}

// One CTA per group: a group with proposals and at least maxasi members keeps
// its maxasi best, takes the maxasi-th best key as its threshold and turns
// the others away: marked in redo and appended to list (they propose again
// next round); kScNext counts them.
__device__ void select_best(const Assign& a, unsigned g)
{
    const unsigned t = a.touched[g], c = a.cnt[g];
    __syncthreads();
    if (!t)
        return;
    if (threadIdx.x == 0)
        a.touched[g] = 0;
    if (c < a.maxasi)
        return;
    const unsigned base = a.off[g];
    const uint64_t* bk = a.bk + base;
    const uint64_t kth = c <= kSmallSel ? kth_largest_small(bk, c, a.maxasi) : kth_largest(bk, c, a.maxasi);
    if (c > a.maxasi)
        for (unsigned i = threadIdx.x; i < c; i += kThreads)
            if (bk[i] < kth) {
                const unsigned p = a.bp[base + i];
                a.assign[p] = -1;
                a.redo[p] = 1;
                a.list[atomicAdd(a.sc + kScNext, 1u)] = p;
            }
    if (threadIdx.x == 0) {
        a.theta[g] = kth;
        a.cnt[g] = a.maxasi;
    }
}

// The group that closed last (lowest threshold), found by every CTA for itself;
// the first checks that every group holds maxasi members.
__device__ unsigned last_group(const Assign& a)
{
    __shared__ uint64_t s_key[kThreads];
    __shared__ unsigned s_grp[kThreads];
    uint64_t best = ~0ull;
    unsigned bg = 0;
    for (unsigned g = threadIdx.x; g < a.nref; g += kThreads) {
        const uint64_t t = a.theta[g];
        if (blockIdx.x == 0 && (a.cnt[g] != a.maxasi || t == 0))
            atomicOr(a.sc + kScErr, kErrInternal);
        if (t < best) {
            best = t;
            bg = g;
        }
    }
    s_key[threadIdx.x] = best;
    s_grp[threadIdx.x] = bg;
    __syncthreads();
    for (unsigned h = kThreads / 2; h > 0; h >>= 1) {
        if (threadIdx.x < h && s_key[threadIdx.x + h] < s_key[threadIdx.x]) {
            s_key[threadIdx.x] = s_key[threadIdx.x + h];
            s_grp[threadIdx.x] = s_grp[threadIdx.x + h];
        }
        __syncthreads();
    }
    return s_grp[0];
}

// Rank of each member within its group by counting the larger keys: chunk
// `chunk` places members chunk*256 .. +255 of group g (g = nref: the
// leftovers) at their rank.
__device__ void rank_chunk(const Assign& a, unsigned g, unsigned chunk)
{
    __shared__ ulonglong2 tile[kThreads / 2];
    const unsigned c = g < a.nref ? a.maxasi : a.extra;
    const unsigned base = g * a.maxasi, i = chunk * kThreads + threadIdx.x;
    const bool live = i < c;
    const uint64_t ki = live ? a.bk[base + i] : 0;
    unsigned r = 0;
    for (unsigned j0 = 0; j0 < c; j0 += kThreads) {
        __syncthreads();
        reinterpret_cast<uint64_t*>(tile)[threadIdx.x] = j0 + threadIdx.x < c ? a.bk[base + j0 + threadIdx.x] : 0;
        __syncthreads();
        const unsigned m = (min(kThreads, c - j0) + 1) / 2; // (a zero past the last is no larger key)
#pragma unroll 8
        for (unsigned j = 0; j < m; j++) {
            const ulonglong2 k = tile[j];
            r += k.x > ki;
            r += k.y > ki;
        }
    }
    if (live)
        a.out[base + r] = (int)a.bp[base + i];
}

// ---- the steps of a round, and of what follows the rounds; every CTA of the grid takes
// its share ----

// room for the members of the groups that received proposals, in any order
__device__ void make_room(const Assign& a)
{
    const unsigned t0 = blockIdx.x * kThreads + threadIdx.x, nt = gridDim.x * kThreads;
    for (unsigned g = t0; g < a.nref; g += nt)
        if (a.touched[g]) {
            a.off[g] = atomicAdd(a.sc + kScTotal, a.cnt[g]);
            a.fill[g] = 0;
        }
    if (t0 == 0) {
        a.sc[kScNext] = 0;
        a.sc[kScRounds]++;
    }
}

// their members, bucketed by group
__device__ void bucket_members(const Assign& a)
{
    const unsigned t0 = blockIdx.x * kThreads + threadIdx.x, nt = gridDim.x * kThreads;
    for (unsigned p = t0; p < a.nima; p += nt) {
        const int g = a.assign[p];
        if (g >= 0 && a.touched[g]) {
            const unsigned s = a.off[g] + atomicAdd(a.fill + g, 1u);
            a.bp[s] = p;
            a.bk[s] = a.pkey[p];
        }
    }
}

__device__ void select_groups(const Assign& a)
{
    if (blockIdx.x == 0 && threadIdx.x == 0)
        a.sc[kScTotal] = 0;
    for (unsigned g = blockIdx.x; g < a.nref; g += gridDim.x)
        select_best(a, g);
}

// belongsto; a leftover particle joins the last group (its pair key with that
// group ranks it among the leftovers) and is tagged with group index nref
__device__ void join_groups(const Assign& a)
{
    const unsigned t0 = blockIdx.x * kThreads + threadIdx.x, nt = gridDim.x * kThreads;
    const unsigned last = last_group(a);
    if (t0 == 0)
        a.sc[kScLast] = last;
    for (unsigned g = t0; g <= a.nref; g += nt)
        a.fill[g] = 0;
    for (unsigned p = t0; p < a.nima; p += nt) {
        int g = a.assign[p];
        if (g < 0) {
            a.pkey[p] = pair_key(a.d[(size_t)last * a.pitch + p], last * a.nima + p);
            a.assign[p] = (int)a.nref;
            atomicAdd(a.sc + kScLeft, 1u);
            g = (int)last;
        }
        if (a.belongsto)
            a.belongsto[p] = g;
    }
}

// members bucketed by final group: group g at g*maxasi, the leftovers at
// nref*maxasi
__device__ void bucket_final(const Assign& a)
{
    const unsigned t0 = blockIdx.x * kThreads + threadIdx.x, nt = gridDim.x * kThreads;
    for (unsigned p = t0; p < a.nima; p += nt) {
        const unsigned g = (unsigned)a.assign[p];
        const unsigned cap = g < a.nref ? a.maxasi : a.extra;
        const unsigned j = g <= a.nref ? atomicAdd(a.fill + g, 1u) : cap;
        if (j >= cap) {
            atomicOr(a.sc + kScErr, kErrInternal);
            continue;
        }
        const unsigned s = g * a.maxasi + j;
        a.bp[s] = p;
        a.bk[s] = a.pkey[p];
    }
}

__device__ void rank_members(const Assign& a)
{
    const unsigned chunks = (a.maxasi + kThreads - 1) / kThreads, chunks_left = (a.extra + kThreads - 1) / kThreads;
    const unsigned long long items = (unsigned long long)a.nref * chunks + chunks_left;
    for (unsigned long long i = blockIdx.x; i < items; i += gridDim.x) {
        const unsigned g = (unsigned)min(i / chunks, (unsigned long long)a.nref);
        rank_chunk(a, g, (unsigned)(i - (unsigned long long)g * chunks));
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        a.out[(size_t)a.nref * a.maxasi + a.extra] = (int)a.sc[kScLast];
}

// The rounds and what follows them, in one cooperative grid that meets between
// steps.  What bounds it: the meetings (four a round) and the steps' dependent
// loads.  As four kernels a round with a read of the count after each, launches and
// reads were most of the time: 20,000 particles x 200 groups (9 rounds) 376 us, now
// 233; 3,000 x 76 (7) 274 -> 135; 300 x 7 (4) 179 -> 82; 100,000 x 500 (10) 661 ->
// 579.  The count read after every third or fourth such round: 311 to 362 us.
__global__ void __launch_bounds__(kThreads)
assign_kernel(Assign a)
{
    unsigned target = 0;
    for (unsigned round = 0;; round++) {
        const bool all = a.first && round == 0;
        // (changed next after the meeting that follows the proposals)
        const unsigned n = all ? a.nima : __ldcg(a.sc + kScNext);
        if (n == 0)
            break;
        if (round == kMaxRounds)
            return;
        if (!all && n <= a.nima / kSparseDiv)
            propose_listed(a, n);
        else
            propose_scan(a, all);
        if (!grid_meet(a, target) || (__ldcg(a.sc + kScErr) & kErrNaN))
            return;
        make_room(a);
        if (!grid_meet(a, target))
            return;
        bucket_members(a);
        if (!grid_meet(a, target))
            return;
        select_groups(a);
        if (!grid_meet(a, target))
            return;
    }
    join_groups(a);
    if (!a.out || !grid_meet(a, target))
        return;
    bucket_final(a);
    if (!grid_meet(a, target) || (__ldcg(a.sc + kScErr) & kErrInternal))
        return;
    rank_members(a);
}

// The same steps a launch each, with a read of the count after every round: a step
// then has as many CTAs as it has work for, with the registers of its own code, where
// the cooperative grid's two to four CTAs an SM (all steps' registers, every CTA in
// every meeting) take many groups and tiles one after another.
enum { kStepScan, kStepListed, kStepRoom, kStepBucket, kStepSelect, kStepJoin, kStepFinal, kStepRank };

template <int STEP>
__global__ void __launch_bounds__(kThreads)
assign_step_kernel(Assign a, unsigned n)
{
    if constexpr (STEP == kStepScan)
        propose_scan(a, a.first);
    else if constexpr (STEP == kStepListed)
        propose_listed(a, n);
    else if constexpr (STEP == kStepRoom)
        make_room(a);
    else if constexpr (STEP == kStepBucket)
        bucket_members(a);
    else if constexpr (STEP == kStepSelect)
        select_groups(a);
    else if constexpr (STEP == kStepJoin)
        join_groups(a);
    else if constexpr (STEP == kStepFinal)
        bucket_final(a);
    else if (!(__ldcg(a.sc + kScErr) & kErrInternal))
        rank_members(a);
}

// Whether the steps run as launches of their own.  Long reads: many pairs, or many
// particles.  Many groups: a selection per group, unless the rounds place few
// particles each, and a scan of all of them per tile, the more so when the
// cooperative grid's CTAs have a second tile each.  us in all, cooperative grid / own
// launches (random peaks, particles x groups):
//   300,000 x 200   792 /   805    500,000 x 200 1,534 / 1,434  1,000,000 x 1,000 4,807 / 3,213
//   300,000 x 100   836 /   882  1,000,000 x 100 3,507 / 3,227    600,000 x 50    2,581 / 2,468
//    10,000 x 2,000 776 /   798     13,000 x 2,000   926 / 790     20,000 x 3,000 1,706 / 991
//     9,000 x 3,000 1,074 / 1,173   11,750 x 2,500 1,626 / 1,010   40,000 x 40,000 35,457 / 27,163
//     6,000 x 6,000 2,376 / 2,467   12,000 x 6,000 3,167 / 2,417
//    50,000 x 1,000 673 /   755    100,000 x 1,000   937 / 876
bool steps_apart(unsigned nref, unsigned nima, unsigned sms)
{
    const unsigned long long pairs = (unsigned long long)nref * nima;
    const bool second_tile = nima > 32 * kCtasPerSm * sms;
    return nima > 400000u || pairs > 80000000ull || (nref > 1000u && pairs > 36000000ull) ||
           (nref >= 2000u && second_tile && pairs > 22000000ull);
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

struct AssignState {
    std::mutex mu;
    Buf<uint64_t> zeroed; // sc, theta, cnt, touched, redo: what a call starts from zero
    Buf<uint64_t> pkey, bk;
    Buf<unsigned> off, fill, bp, list;
    Buf<int> assign;
    Buf<float> d_host_copy;
    Buf<int> ids_host_copy;
    unsigned* h_sc = nullptr; // pinned
} g_asg;

int fail(int code, const char* msg)
{
    record_error(code, msg);
    return code;
}

#define A_CK(expr)                                                                                    \
    do {                                                                                              \
        cudaError_t e_ = (expr);                                                                      \
        if (e_ != cudaSuccess) {                                                                      \
            char m_[384];                                                                             \
            snprintf(m_, sizeof(m_), "%s (%s) in the group assignment", cudaGetErrorString(e_), #expr); \
            return fail(1, m_);                                                                       \
        }                                                                                             \
    } while (0)

int check_args(const float* d, unsigned long long pitch, unsigned nref, unsigned nima)
{
    if (!d)
        return fail(2, "assign_groups: d is NULL");
    if (nref == 0 || nima < nref)
        return fail(2, "assign_groups: needs 1 <= nref <= nima");
    if ((unsigned long long)nref * nima > 0xFFFFFFFFull)
        return fail(2, "assign_groups: nref * nima must stay below 2^32");
    if (pitch < nima)
        return fail(2, "assign_groups: d_pitch smaller than nima");
    // (the list ranks members by comparing all of a group with all: 40 s at that size)
    if ((nima / nref + kThreads - 1) / kThreads > 65535u)
        return fail(2, "assign_groups: groups of more than 16,776,960 particles");
    return 0;
}

int assign_locked(const float* d, size_t pitch, unsigned nref, unsigned nima, int* belongsto, int* id_list_long,
                  unsigned* rounds_out, cudaStream_t st)
{
    AssignState& w = g_asg;
    const unsigned maxasi = nima / nref, extra = nima % nref;
    const size_t zero_words = kScWords + 2 * (size_t)nref + ((size_t)nima + 7) / 8;
    A_CK(w.zeroed.ensure(zero_words));
    unsigned* const sc = reinterpret_cast<unsigned*>(w.zeroed.p);
    uint64_t* const theta = w.zeroed.p + kScWords;
    unsigned *const cnt = reinterpret_cast<unsigned*>(theta + nref), *const touched = cnt + nref;
    unsigned char* const redo = reinterpret_cast<unsigned char*>(theta + 2 * (size_t)nref);
    A_CK(w.off.ensure(nref));
    A_CK(w.fill.ensure(nref + 1));
    A_CK(w.assign.ensure(nima));
    A_CK(w.pkey.ensure(nima));
    A_CK(w.bp.ensure(nima));
    A_CK(w.bk.ensure(nima));
    A_CK(w.list.ensure(nima));
    if (!w.h_sc)
        A_CK(cudaHostAlloc(&w.h_sc, kScCount * sizeof(unsigned), cudaHostAllocDefault));

    A_CK(cudaMemsetAsync(w.zeroed.p, 0, zero_words * sizeof(uint64_t), st));

    int dev = 0, sms = 0, per_sm = 0;
    A_CK(cudaGetDevice(&dev));
    A_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    A_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, assign_kernel, (int)kThreads, 0));
    const unsigned tiles = (nima + 31) / 32;
    const unsigned want = tiles >= kWideTiles * (unsigned)sms ? kCtasPerSmWide : kCtasPerSm;
    // no more CTAs than the widest step has work for
    const unsigned grid = std::min((unsigned)sms * std::min((unsigned)std::max(per_sm, 1), want), std::max(tiles, nref));
    Assign a{d, pitch, nref, nima, maxasi, extra, true, belongsto, id_list_long, theta, w.pkey.p, w.bk.p,
             cnt, touched, w.off.p, w.fill.p, w.bp.p, w.list.p, sc, redo, w.assign.p, kStartTries, kWaitTries, 0};
    unsigned test_stall = 0, test_tries = 0;
    ccf_test_settings(test_stall, test_tries);
    if (test_stall)
        a.stall = 1, a.start_tries = a.wait_tries = test_tries;
    const unsigned long long max_rounds = (unsigned long long)nref * nima + 1;
    unsigned rounds = 0, turned = nima;
    const bool apart = steps_apart(nref, nima, (unsigned)sms);
    auto step = [&](auto kernel, unsigned ctas, unsigned n) {
        kernel<<<std::max(ctas, 1u), kThreads, 0, st>>>(a, n);
        g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    };
    const unsigned per_particle = (nima + kThreads - 1) / kThreads;
    for (;;) {
        if (apart) {
            if (!a.first && turned <= nima / kSparseDiv)
                step(assign_step_kernel<kStepListed>, (turned + 7) / 8, turned);
            else
                step(assign_step_kernel<kStepScan>, tiles, 0);
            step(assign_step_kernel<kStepRoom>, (nref + kThreads - 1) / kThreads, 0);
            step(assign_step_kernel<kStepBucket>, per_particle, 0);
            step(assign_step_kernel<kStepSelect>, nref, 0);
            A_CK(cudaGetLastError());
        } else {
            void* args[] = {&a};
            A_CK(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(assign_kernel), dim3(grid), dim3(kThreads),
                                             args, 0, st));
            g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
        }
        A_CK(cudaMemcpyAsync(w.h_sc, sc, kScCount * sizeof(unsigned), cudaMemcpyDeviceToHost, st));
        A_CK(cudaStreamSynchronize(st));
        rounds = w.h_sc[kScRounds];
        if (w.h_sc[kScErr] & kErrWait)
            return fail(1, "assign_groups: a grid barrier timed out (bounded wait ran out)");
        if (w.h_sc[kScErr] & kErrNaN)
            return fail(2, "assign_groups: d holds a NaN peak");
        turned = w.h_sc[kScNext];
        if (turned == 0)
            break;
        if (turned > nima || rounds >= max_rounds)
            return fail(1, "assign_groups: the proposal rounds did not settle (internal error)");
        a.first = false;
        if (!apart)
            A_CK(cudaMemsetAsync(sc + kScBar, 0, sizeof(unsigned), st));
    }
    if (apart) {
        step(assign_step_kernel<kStepJoin>, std::min(per_particle, 8u * (unsigned)sms), 0);
        if (id_list_long) {
            step(assign_step_kernel<kStepFinal>, per_particle, 0);
            step(assign_step_kernel<kStepRank>, nref * ((maxasi + kThreads - 1) / kThreads) + 1, 0);
        }
        A_CK(cudaGetLastError());
        A_CK(cudaMemcpyAsync(w.h_sc, sc, kScCount * sizeof(unsigned), cudaMemcpyDeviceToHost, st));
        A_CK(cudaStreamSynchronize(st));
    }
    if ((w.h_sc[kScErr] & kErrInternal) || w.h_sc[kScLeft] != extra)
        return fail(1, "assign_groups: inconsistent group sizes (internal error)");
    if (rounds_out)
        *rounds_out = rounds;
    return 0;
}

} // namespace

void assign_clear()
{
    std::lock_guard<std::mutex> lk(g_asg.mu);
    AssignState& w = g_asg;
    auto drop = [](auto& b) {
        if (b.p)
            cudaFree(b.p);
        b.p = nullptr;
        b.n = 0;
    };
    drop(w.zeroed), drop(w.pkey), drop(w.bk), drop(w.off), drop(w.fill);
    drop(w.bp), drop(w.list), drop(w.assign), drop(w.d_host_copy);
    drop(w.ids_host_copy);
    if (w.h_sc)
        cudaFreeHost(w.h_sc);
    w.h_sc = nullptr;
}

} // namespace gpuisac

using namespace gpuisac;

extern "C" int gpuisac_assign_groups_device(const float* d, unsigned long long d_pitch, unsigned int nref,
                                            unsigned int nima, int* belongsto, int* id_list_long,
                                            unsigned int* rounds, void* stream)
{
    const gpuisac::NvtxRange nvtx_range("gpuisac:assign_groups");
    if (d_pitch == 0)
        d_pitch = nima;
    int rc = check_args(d, d_pitch, nref, nima);
    if (rc)
        return rc;
    if (!belongsto && !id_list_long)
        return fail(2, "assign_groups: neither belongsto nor id_list_long given");
    std::lock_guard<std::mutex> lk(g_asg.mu);
    return assign_locked(d, (size_t)d_pitch, nref, nima, belongsto, id_list_long, rounds, (cudaStream_t)stream);
}

extern "C" int gpuisac_assign_groups(const float* d, unsigned int nref, unsigned int nima, int* id_list_long)
{
    int rc = check_args(d, nima, nref, nima);
    if (rc)
        return rc;
    if (!id_list_long)
        return fail(2, "assign_groups: id_list_long is NULL");
    std::lock_guard<std::mutex> lk(g_asg.mu);
    AssignState& w = g_asg;
    const size_t n = (size_t)nref * nima;
    A_CK(w.d_host_copy.ensure(n));
    A_CK(w.ids_host_copy.ensure((size_t)nima + 1));
    A_CK(cudaMemcpy(w.d_host_copy.p, d, n * sizeof(float), cudaMemcpyHostToDevice));
    rc = assign_locked(w.d_host_copy.p, nima, nref, nima, nullptr, w.ids_host_copy.p, nullptr, nullptr);
    if (rc)
        return rc;
    A_CK(cudaMemcpy(id_list_long, w.ids_host_copy.p, ((size_t)nima + 1) * sizeof(int), cudaMemcpyDeviceToHost));
    return 0;
}
