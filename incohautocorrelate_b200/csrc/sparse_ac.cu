// sparse_ac.cu -- (a) sparse photon pairs -> uint64 3D q-mesh.
//
// Replaces the device route of Detector::AutoCorrelateSparseList
// (IAC/Detector.cpp:1053-1181) and its kernel Autocor_sparseHL with helpers
// AddRotatedQToMesh / AddQToPositiveSS (IAC/kernel.cl:349-652), batched over
// many frames.
//
// Work decomposition.  A frame of n photons has n(n-1)/2 distinct pairs plus
// n self pairs.  Every unordered pair {i, j}, i != j, is (i, i + d mod n) for
// exactly one offset d = 1 .. floor(n/2) (d = n/2 only for i < n/2 when n is
// even).  The offsets are cut into chunks of L steps; an item is (photon i,
// chunk), a unit 32 consecutive items: a warp whose lanes hold one photon each
// and walk the L partners i + d, so the partner loads of a step are 512
// contiguous bytes and a step needs one load, no division and no ordering of
// its two photons.  Frames are laid end to end by cost (units x (L + overhead))
// and the warps of the launch take equal chunks of the batch's cost from one
// counter: no queue of tiles, no barrier between frames.  L comes from the batch's
// pair count, so that a single event still spreads over the GPU.
//
// Exactness.  All float operations are the reference's, in its order, as
// explicitly rounded intrinsics (no contraction into FMA); the value
// (double)v_lo * v_hi * Multiplicator is truncated to uint64 as the C cast
// does.  Swapping a pair's photons negates q exactly, and nearest binning of
// -q is the point reflection of that of q, which the half mesh folds back; the
// linear modes restore the reference's order q = k_lo - k_hi.  Self pairs add
// (uint64)(v*v*Mult) at q = 0, which the reference writes to half-mesh voxel
// (C, C, 0) without a mirror for every second-level interpolation mode; they
// are summed per warp and added with one atomic.
//
// The half mesh accumulates with 64-bit atomic adds in L2 (the 201^3 half mesh
// is 32.6 MB and stays L2-resident).  Writes whose voxel would fall outside the
// mesh (possible only for non-orthonormal rotations; the reference writes them
// out of bounds) are skipped and counted in the context's error block.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include <cooperative_groups.h>

#include "iac_internal.cuh"

namespace iac {

namespace cg = cooperative_groups;

// L2 cache policies (PTX createpolicy) for the pair kernel: the half mesh is
// kept resident while the photon stream passes through.
__device__ __forceinline__ uint64_t l2_policy_evict_last()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_first()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_policy_normal()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_unchanged.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void red_add_hint(unsigned long long *addr, unsigned long long v, uint64_t pol)
{
    asm volatile("red.global.add.L2::cache_hint.u64 [%0], %1, %2;" ::"l"(addr), "l"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ float4 ld_photon_hint(const float4 *p, uint64_t pol)
{
    float4 r;
    asm volatile("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
                 : "l"(p), "l"(pol));
    return r;
}

// ---------------------------------------------------------------------------
// the walk over a batch's pairs
// ---------------------------------------------------------------------------
constexpr uint32_t PAIR_STEPS_MAX = 32;   // steps of a unit (partners a lane walks) at most
constexpr uint32_t PAIR_UNIT_COST = 3;    // a unit's set-up in units of a step, for the shares
constexpr uint32_t PAIR_DIRECT = 256;     // frames a CTA plans by itself, without the planner's launch

// what the planner leaves for the walking kernels, before the table of frame starts
struct PlanHeader {
    unsigned long long cost;   // of the whole batch
    unsigned long long pairs;  // distinct pairs of the whole batch
    uint32_t steps;            // the batch's step limit
    uint32_t next;             // chunks of the batch taken so far
};

struct WalkArgs {
    const float4 *__restrict__ photons;
    const uint64_t *__restrict__ offsets;
    PlanHeader *head;                                   // written by the planner; null: planned by the CTA
    const unsigned long long *__restrict__ cost_off;    // nframes + 1
    uint32_t nframes;
    uint32_t steps_max;
};

__device__ __forceinline__ unsigned long long frame_pairs(uint32_t n)
{
    return n ? (unsigned long long)n * (n - 1) / 2 : 0ull;
}

// chunks and steps of a frame of n photons under the batch's step limit
struct FrameShape {
    uint32_t nc, L;
    unsigned long long units;
};
__device__ __forceinline__ FrameShape frame_shape(uint32_t n, uint32_t steps)
{
    // steps run two at a time, so L is even; of the two smallest chunk counts the
    // one with the less padding and set-up
    const uint32_t half = n >> 1;
    const uint32_t nc0 = max(1u, (half + steps - 1) / steps), nc1 = nc0 + 1;
    const uint32_t L0 = ((half + nc0 - 1) / nc0 + 1) & ~1u, L1 = ((half + nc1 - 1) / nc1 + 1) & ~1u;
    FrameShape s;
    const bool more = nc1 * (L1 + PAIR_UNIT_COST) < nc0 * (L0 + PAIR_UNIT_COST);
    s.nc = more ? nc1 : nc0;
    s.L = more ? L1 : L0;
    s.units = ((unsigned long long)n * s.nc + 31) / 32;
    return s;
}
__device__ __forceinline__ unsigned long long frame_cost(uint32_t n, uint32_t steps)
{
    const FrameShape s = frame_shape(n, steps);
    return s.units * (s.L + PAIR_UNIT_COST);
}
// the step limit that leaves every warp of the launch about two units or more
__device__ __forceinline__ uint32_t batch_steps(unsigned long long pairs, uint32_t warps, uint32_t steps_max)
{
    const unsigned long long s = pairs / (64ull * warps);
    return (uint32_t)max(1ull, min((unsigned long long)steps_max, s));
}

// ---------------------------------------------------------------------------
// planner: the exclusive prefix sum of the frames' costs (the first cluster),
// and per frame a flag for the pair kernel's fast path (the other CTAs, one warp
// per frame): the largest photon count if all photon values are integers in
// [1, 128], so that v_lo * v_hi * Mult (Mult an integer <= 1024) is at most 2^24
// and exact in FP32, FLAG_VALUES for other values, and 0 (no fast path) unless
// the k-vectors are finite and the rows of the rotation are short enough
// (row_limit2, a little over 1 for the mesh of a detector) that no pair within
// MaxQ can leave the mesh.
// Bound by reading the photons once: 61 us for 100 000 frames of 11 M photons
// (one CTA walking 98 frames per thread took 146 us, the check another 36).
// ---------------------------------------------------------------------------
constexpr int PLAN_THREADS = 1024;
constexpr int PLAN_CTAS = 8;  // CTAs of the scanning cluster (the portable cluster size)

__device__ __forceinline__ unsigned long long block_sum_u64(unsigned long long v, unsigned long long *warp_sums)
{
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();  // warp_sums may still be read
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = v;
    __syncthreads();
    unsigned long long t = 0;
    for (uint32_t w = 0; w < blockDim.x / 32; w++) t += warp_sums[w];
    return t;
}

constexpr uint32_t FLAG_VALUES = 129, FLAG_GENERAL = 255;  // 255 is stored as 0
// the photon's count, or what rules counts or the fast path out
__device__ __forceinline__ uint32_t fast_count(const float4 p)
{
    const bool count = p.w >= 1.0f && p.w <= 128.0f && p.w == truncf(p.w);
    const bool finite = fabsf(p.x) < INFINITY && fabsf(p.y) < INFINITY && fabsf(p.z) < INFINITY;
    return !finite ? FLAG_GENERAL : count ? (uint32_t)p.w : FLAG_VALUES;
}
__device__ __forceinline__ bool fast_row(const float *r, float row_limit2)
{
    return r[0] * r[0] + r[1] * r[1] + r[2] * r[2] <= row_limit2;  // false for a NaN
}

__global__ void __cluster_dims__(PLAN_CTAS, 1, 1) __launch_bounds__(PLAN_THREADS)
    sparse_plan_kernel(const uint64_t *__restrict__ off, uint32_t nframes, uint32_t steps_max, uint32_t warps,
                       unsigned long long *__restrict__ cost_off, PlanHeader *head, const float4 *__restrict__ ph,
                       const float *__restrict__ rot, float row_limit2, unsigned char *__restrict__ flags)
{
    __shared__ unsigned long long warp_sums[PLAN_THREADS / 32];
    __shared__ unsigned long long s_mine[2];  // this CTA's pairs and cost, read by the cluster
    const uint32_t tid = threadIdx.x;
    const int lane = tid & 31, w = tid >> 5;
    if (blockIdx.x >= PLAN_CTAS) {
        const uint32_t warp = (blockIdx.x - PLAN_CTAS) * (PLAN_THREADS / 32) + w;
        const uint32_t stride = (gridDim.x - PLAN_CTAS) * (PLAN_THREADS / 32);
        for (uint32_t f = warp; f < nframes; f += stride) {
            uint32_t m = lane >= 3 || fast_row(rot + 9 * (size_t)f + 3 * lane, row_limit2) ? 1u : FLAG_GENERAL;
            const uint64_t end = off[f + 1];
            for (uint64_t i = off[f] + lane; i < end; i += 128) {  // four loads in flight
                const float4 p0 = ph[i], p1 = ph[min(i + 32, end - 1)], p2 = ph[min(i + 64, end - 1)],
                             p3 = ph[min(i + 96, end - 1)];
                m = max(max(max(m, fast_count(p0)), max(fast_count(p1), fast_count(p2))), fast_count(p3));
            }
            m = __reduce_max_sync(0xffffffffu, m);
            if (lane == 0) flags[f] = m == FLAG_GENERAL ? 0 : (unsigned char)m;
        }
        return;
    }
    cg::cluster_group cl = cg::this_cluster();
    const uint32_t rank = cl.block_rank();
    const uint32_t f0 = (uint32_t)((uint64_t)nframes * rank / PLAN_CTAS),
                   f1 = (uint32_t)((uint64_t)nframes * (rank + 1) / PLAN_CTAS);
    unsigned long long v = 0;
    for (uint32_t f = f0 + tid; f < f1; f += PLAN_THREADS) v += frame_pairs((uint32_t)(off[f + 1] - off[f]));
    v = block_sum_u64(v, warp_sums);
    if (tid == 0) s_mine[0] = v;
    cl.sync();
    unsigned long long pairs = 0;
    for (int r = 0; r < PLAN_CTAS; r++) pairs += *cl.map_shared_rank(&s_mine[0], r);
    const uint32_t steps = batch_steps(pairs, warps, steps_max);
    v = 0;
    for (uint32_t f = f0 + tid; f < f1; f += PLAN_THREADS) v += frame_cost((uint32_t)(off[f + 1] - off[f]), steps);
    v = block_sum_u64(v, warp_sums);
    if (tid == 0) s_mine[1] = v;
    cl.sync();
    unsigned long long run = 0, cost = 0;
    for (uint32_t r = 0; r < PLAN_CTAS; r++) {
        const unsigned long long c = *cl.map_shared_rank(&s_mine[1], r);
        run += r < rank ? c : 0ull;
        cost += c;
    }
    cl.sync();  // no CTA leaves while its sums are read
    for (uint32_t c0 = f0; c0 < f1; c0 += PLAN_THREADS) {
        const uint32_t f = c0 + tid;
        const unsigned long long c = f < f1 ? frame_cost((uint32_t)(off[f + 1] - off[f]), steps) : 0ull;
        unsigned long long incl = c;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        __syncthreads();
        if (lane == 31) warp_sums[w] = incl;
        __syncthreads();
        unsigned long long before = 0, all = 0;
        for (int k = 0; k < PLAN_THREADS / 32; k++) {
            const unsigned long long s = warp_sums[k];
            before += k < w ? s : 0ull;
            all += s;
        }
        if (f < f1) cost_off[f] = run + before + incl - c;
        run += all;
    }
    if (rank == 0 && tid == 0) {
        cost_off[nframes] = cost;
        head->cost = cost;
        head->pairs = pairs;
        head->steps = steps;
        head->next = 0u;
    }
}

// a small batch planned by the CTA itself in shared memory (every thread of
// the block): s_off gets nframes + 1 starts; returns the header.  The sums and the
// scan take the whole block: by one warp, with 64-bit shared adds, 200 frames took
// 9 us longer.
__device__ __forceinline__ PlanHeader plan_direct(const WalkArgs &a, uint32_t warps, unsigned long long *s_off,
                                                  unsigned long long *warp_sums)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    PlanHeader h;
    h.next = 0u;
    if (a.nframes <= 32) {  // each warp by itself, one barrier
        const uint32_t n = lane < a.nframes ? (uint32_t)(a.offsets[lane + 1] - a.offsets[lane]) : 0u;
        h.pairs = frame_pairs(n);
        for (int o = 16; o; o >>= 1) h.pairs += __shfl_xor_sync(0xffffffffu, h.pairs, o);
        h.steps = batch_steps(h.pairs, warps, a.steps_max);
        unsigned long long incl = lane < a.nframes ? frame_cost(n, h.steps) : 0ull;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long u = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += u;
        }
        if (w == 0 && lane < a.nframes) s_off[lane + 1] = incl;
        if (tid == 0) s_off[0] = 0ull;
        __syncthreads();
        h.cost = __shfl_sync(0xffffffffu, incl, 31);
        return h;
    }
    unsigned long long pairs = 0;
    for (uint32_t f = tid; f < a.nframes; f += blockDim.x) {
        const uint32_t n = (uint32_t)(a.offsets[f + 1] - a.offsets[f]);
        s_off[f + 1] = n;
        pairs += frame_pairs(n);
    }
    h.pairs = block_sum_u64(pairs, warp_sums);
    h.steps = batch_steps(h.pairs, warps, a.steps_max);
    unsigned long long run = 0;
    for (uint32_t c0 = 0; c0 < a.nframes; c0 += blockDim.x) {
        const uint32_t f = c0 + tid;
        unsigned long long incl = f < a.nframes ? frame_cost((uint32_t)s_off[f + 1], h.steps) : 0ull;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long u = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += u;
        }
        __syncthreads();
        if (lane == 31) warp_sums[w] = incl;
        __syncthreads();
        unsigned long long before = 0, all = 0;
        for (uint32_t k = 0; k < blockDim.x / 32; k++) {
            const unsigned long long s = warp_sums[k];
            before += k < w ? s : 0ull;
            all += s;
        }
        if (f < a.nframes) s_off[f + 1] = run + before + incl;
        run += all;
    }
    if (tid == 0) s_off[0] = 0ull;
    __syncthreads();
    h.cost = run;
    return h;
}

// last frame f with off[f] <= x, by a whole warp (off[0] <= x < off[nframes])
__device__ __forceinline__ uint32_t warp_find_frame(const unsigned long long *off, uint32_t nframes,
                                                    unsigned long long x)
{
    uint32_t lo = 0, hi = nframes;  // off[lo] <= x < off[hi]
    const uint32_t lane = threadIdx.x & 31;
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t at = lo + lane * step;
        const unsigned below = __ballot_sync(0xffffffffu, at < hi && off[at] <= x);
        const uint32_t k = 31 - __clz(below);  // lane 0 is always below
        lo += k * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// The cost [x0, x1) that a CTA's warps take chunks of: the whole batch, from
// the counter in the header, or for a batch planned in the CTA an equal part of
// it, from a counter of the CTA.  Shares fixed beforehand left the slowest SM
// of a 100 000-frame batch 24 % behind the mean.  A CTA takes at most `most`
// chunks, twice its part of the batch, which bounds what it can add up.
struct Share {
    unsigned long long x0, x1;
    uint32_t chunk;  // cost a warp takes at a time
    uint32_t most;
};
// A chunk: about four a warp at least, whole units, few enough frame searches, and so
// many of the cost that its 32-bit counter holds them.
__host__ __device__ constexpr uint32_t chunk_cost(unsigned long long cost, uint32_t ctas, uint32_t threads, uint32_t steps)
{
    unsigned long long c = cost / ctas / (threads / 8);
    c = c > 128 ? 128 : c;
    c = c < steps + PAIR_UNIT_COST ? steps + PAIR_UNIT_COST : c;
    return (uint32_t)(c < (cost >> 31) ? cost >> 31 : c);
}
static_assert(chunk_cost(1ull << 16, 148, 1024, 2) == 5 && chunk_cost(1ull << 30, 148, 1024, 32) == 128 &&
                  chunk_cost(1ull << 40, 148, 1024, 32) == 512 && (1ull << 50) / chunk_cost(1ull << 50, 1, 32, 32) <= 1ull << 31,
              "the chunks of a batch fit the counter");
__device__ __forceinline__ Share cta_share(const PlanHeader &h, bool whole)
{
    Share s;
    s.x0 = whole ? 0ull : h.cost * blockIdx.x / gridDim.x;
    s.x1 = whole ? h.cost : h.cost * (blockIdx.x + 1) / gridDim.x;
    const unsigned long long part = h.cost / gridDim.x;
    s.chunk = chunk_cost(h.cost, gridDim.x, blockDim.x, h.steps);
    s.most = (uint32_t)min(0x7fffffffull, 2 * part / s.chunk + 64);
    return s;
}

// The warps of a CTA take chunks of its share in turn (next: its counter; taken:
// the CTA's own count in shared memory, zero before).  frame(f, base, n) is called (by all lanes) when a warp enters
// frame f, unit(i, c, active, nc, L) for each unit with the lane's photon i and
// chunk c (an inactive lane: i = 0).
template <class Frame, class Unit>
__device__ __forceinline__ void walk_share(const WalkArgs &a, const PlanHeader &h, const unsigned long long *off,
                                           const Share &sh, uint32_t *next, uint32_t *taken, Frame frame, Unit unit)
{
    const uint32_t lane = threadIdx.x & 31;
    uint32_t f = warp_find_frame(off, a.nframes, sh.x0);
    for (;;) {
        uint32_t at0 = 0xffffffffu;
        if (lane == 0 && atomicAdd(taken, 1u) < sh.most) at0 = atomicAdd(next, 1u);
        at0 = __shfl_sync(0xffffffffu, at0, 0);
        const unsigned long long start = sh.x0 + (unsigned long long)at0 * sh.chunk;
        if (at0 == 0xffffffffu || start >= sh.x1) return;
        const unsigned long long end = min(sh.x1, start + sh.chunk);
        {   // the frame of `start`, at or after the last one
            const uint32_t at = f + 1 + lane;
            const unsigned below = __ballot_sync(0xffffffffu, at <= a.nframes && off[min(at, a.nframes)] <= start);
            f += __popc(below);
            if (below == 0xffffffffu) f += warp_find_frame(off + f, a.nframes - f, start);
        }
        unsigned long long pos = off[f], skip = start - pos;  // skip: cost of the frame's units before `start`
        for (uint32_t g = f; pos < end && g < a.nframes; g++) {
            const uint64_t base = a.offsets[g];
            const uint32_t n = (uint32_t)(a.offsets[g + 1] - base);
            const FrameShape s = frame_shape(n, h.steps);
            const uint32_t cost = s.L + PAIR_UNIT_COST;
            unsigned long long u = skip ? (skip + cost - 1) / cost : 0ull;  // the units that start in the chunk
            skip = 0;
            unsigned long long last = s.units;
            if (pos + s.units * cost > end) last = (end - pos + cost - 1) / cost;
            if (u < last) {
                frame(g, base, n);
                const unsigned long long items = (unsigned long long)n * s.nc;
                for (; u < last; u++) {
                    const unsigned long long t = u * 32 + lane;
                    const bool active = t < items;
                    const uint32_t c = !active ? 0u : items < (1ull << 32) ? (uint32_t)t / n : (uint32_t)(t / n);
                    const uint32_t i = active ? (uint32_t)(t - (unsigned long long)c * n) : 0u;
                    unit(i, c, active, s.nc, s.L);
                }
            }
            pos += s.units * cost;
        }
    }
}

// the partners of photon i in chunk c: offsets d0 .. d0 + steps - 1
__device__ __forceinline__ void chunk_steps(uint32_t n, uint32_t i, uint32_t c, uint32_t L, bool active, uint32_t &d0,
                                            int &steps)
{
    const uint32_t half = n >> 1;
    const uint32_t dmax = (n & 1) ? half : half - (i >= half ? 1u : 0u);
    d0 = 1 + c * L;
    steps = active ? (int)min(L, dmax + 1 > d0 ? dmax + 1 - d0 : 0u) : 0;
}

// Half-width R of the shared-memory box of voxels around q = 0 (ss <= R,
// |fs - C| <= R, |ms - C| <= R) that each CTA of the pair kernel accumulates
// privately, by the batch's distinct pairs: none below BOX_PAIRS_SMALL,
// BOX_R_SMALL below BOX_PAIRS_LARGE, else BOX_R_MAX (BOX_R_HEAVY).  L2
// takes scattered adds at about 2e11 per second, one request each, whatever
// their width, so every add that stays in the box counts: in a 201^3 mesh of
// the rotated workload R = 22 keeps 32 % of them, R = 10 9 %.  100 000 frames
// (1.16e9 pairs): 5.01 ms at R = 16, 4.35 at 20, 4.21 at 22 (R = 23 leaves the
// photons too little L1: 4.18, but a short batch is slower).  The lines between
// the sizes: 1 000 frames (1.2e7 pairs) 149 us without a box, 139 at R = 10,
// 148 at 22; 3 000 frames 273, 251 and 229; 300 frames 103, 104 and 118.
constexpr int BOX_R_MAX = 22;    // 23 x 45 x 45 words: 186 KB
constexpr int BOX_R_SMALL = 10;
constexpr int BOX_R_HEAVY = 17;  // the most where the first level is linear
constexpr unsigned long long BOX_PAIRS_SMALL = 1000000ull, BOX_PAIRS_LARGE = 20000000ull;

struct SparseArgs {
    WalkArgs walk;
    const float *__restrict__ rot;
    unsigned long long *__restrict__ half;
    DeviceCounters *counters;
    int S, C, half_ss;
    uint32_t plane;  // S * S (the half mesh has fewer than 2^32 words for S <= 1621)
    float maxq2;  // largest float s with sqrtf(s) <= maxq: |q| > maxq  <=>  |q|^2 > maxq2
    float vpdq;   // (float)Voxel_per_dq
    float row_limit2;  // squared length of a rotation's rows up to which the fast path applies
    float neg_zero;  // -0.0f: fma(a, b, -0) is a * b rounded once, and never merges with an add
    double mult;
    uint32_t mult_u;                        // Multiplicator when it is an integer <= 1024, else 0
    const unsigned char *__restrict__ flags;  // per frame: largest count, 0: not the fast path (the planner's check)
    int check_here;   // no planner ran: the CTA checks its frames itself
    int fast_ok;      // MaxQ is finite
    int cache_hints;  // 1: mesh atomics evict-last, photon loads evict-first in L2; else no preference
    int box_max;      // half-width of the largest shared-memory box
    // set inside the kernel
    uint64_t mesh_policy, photon_policy;
    float box_lim;    // |rotated component| below this rounds into the box (box_r + 0.5; 0: no box)
    int center, box_center, box_plane;  // words of the mesh's and the box's centre, words of a box plane
    int box_r;        // half-width of the box around q = 0 (-1: none)
    uint32_t box_w;   // 2 * box_r + 1 (0: none)
    uint32_t box_base;  // shared-memory address of the box
};

// ---------------------------------------------------------------------------
// binning helpers (IAC/kernel.cl:349-448)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void mesh_add(const SparseArgs &a, uint32_t word, unsigned long long v)
{
    red_add_hint(&a.half[word], v, a.mesh_policy);
}

__device__ __forceinline__ uint32_t box_add32(const SparseArgs &a, uint32_t k, uint32_t v)
{
    uint32_t old;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(a.box_base + 4u * k), "r"(v) : "memory");
    return old;
}

// 2^32 times `up` at mesh word `word`, or at both words of a mirrored pair of
// the plane ss = 0
static __device__ __noinline__ void carry_out(unsigned long long *half, uint32_t word, uint32_t mirror, uint32_t up)
{
    atomicAdd(&half[word], (unsigned long long)up << 32);
    if (mirror != word) atomicAdd(&half[mirror], (unsigned long long)up << 32);
}

// one write outside the mesh, or a mirrored pair of them, added up over the lanes that
// are here first (3 000 frames with rotations stretched by 1.3: 482 us, 894 with each
// lane's own add to the one counter).  EACH, for the 64 corners of two linear levels, whose
// lanes part: 3.98 ms for 200 frames, 5.45 added up.
static __device__ __noinline__ void count_lost(DeviceCounters *counters, bool two)
{
    const unsigned here = __activemask();
    const uint32_t n = __reduce_add_sync(here, two ? 2u : 1u);
    if ((threadIdx.x & 31) == (unsigned)__ffs(here) - 1u) atomicAdd(&counters->out_of_mesh, (unsigned long long)n);
}

// v at the voxel (r0, r1, r2) relative to the mesh centre, r2 >= 0; a voxel of
// the plane r2 = 0 and its mirror (-r0, -r1) always receive the same value
// (q and -q of a pair), so this adds it to both: two adds at the centre itself.
// The box keeps the low 32 bits of its sums, and one of the two mirrored voxels
// of its plane 0, which the flush adds to both; what leaves the 32 bits (a
// carry, seen by the add that caused it, or a value past them) goes straight to
// the mesh.
template <bool EACH = false>
__device__ __forceinline__ void put_pair(const SparseArgs &a, int r0, int r1, int r2, unsigned long long v)
{
    const int fs = r0 + a.C, ms = r1 + a.C;
    const uint32_t word = (uint32_t)fs + (uint32_t)ms * (uint32_t)a.S + (uint32_t)r2 * a.plane;
    const uint32_t mirror = r2 == 0 ? (uint32_t)(a.C - r0) + (uint32_t)(a.C - r1) * (uint32_t)a.S : word;
    if ((uint32_t)fs >= (uint32_t)a.S || (uint32_t)ms >= (uint32_t)a.S || r2 >= a.half_ss) {
        if (EACH)
            atomicAdd(&a.counters->out_of_mesh, r2 == 0 ? 2ull : 1ull);
        else
            count_lost(a.counters, r2 == 0);
        return;
    }
    if (v == 0) return;
    if ((uint32_t)(r0 + a.box_r) < a.box_w && (uint32_t)(r1 + a.box_r) < a.box_w && r2 <= a.box_r) {
        const uint32_t k = ((uint32_t)r2 * a.box_w + (uint32_t)(r1 + a.box_r)) * a.box_w + (uint32_t)(r0 + a.box_r);
        const uint32_t old = box_add32(a, k, (uint32_t)v);
        uint32_t up = (uint32_t)(v >> 32) + (old + (uint32_t)v < old ? 1u : 0u);
        if (r2 == 0 && word == mirror) up *= 2;  // the flush counts the centre twice
        if (up) carry_out(a.half, word, mirror, up);
    } else {
        mesh_add(a, word, v);
        if (r2 == 0) mesh_add(a, mirror, v);
    }
}

// AddQToPositiveSS, IAC/kernel.cl:349-372 (q != 0 here; q = 0 is the self
// pair): ss > 0 as it is, ss < 0 at the point reflection, ss = 0 at both
template <bool EACH = false>
__device__ __forceinline__ void add_positive_ss(const SparseArgs &a, int fs, int ms, int ss,
                                                unsigned long long v)
{
    const bool neg = ss < 0;
    put_pair<EACH>(a, neg ? a.C - fs : fs - a.C, neg ? a.C - ms : ms - a.C, neg ? -ss : ss, v);
}

// Second-level nearest neighbour of AddRotatedQToMesh (IAC/kernel.cl:380-389)
// followed by AddQToPositiveSS: fs = C + round(q0), ms = C + round(q1),
// ss = round(q2).  (The reference adds the float centre to the rounded float,
// which is exact for every in-mesh index.)
__device__ __forceinline__ void add_nearest(const SparseArgs &a, float q0, float q1, float q2,
                                            unsigned long long v)
{
    add_positive_ss(a, a.C + round_away_rz_i(q0), a.C + round_away_rz_i(q1), round_away_rz_i(q2), v);
}

// AddRotatedQToMesh, IAC/kernel.cl:374-448
template <int I2, bool EACH = false>
__device__ __forceinline__ void add_rotated(const SparseArgs &a, double val, float q0, float q1,
                                            float q2)
{
    const float Cf = (float)a.C;
    if (I2 == 0) {
        const unsigned long long v = d2u64(dmul(val, a.mult));
        add_nearest(a, q0, q1, q2, v);
    } else {
        const float f0 = floorf(q0), f1 = floorf(q1), f2 = floorf(q2);
        const double sf = dsub(1.0, (double)fsub(q0, f0));
        const double sm = dsub(1.0, (double)fsub(q1, f1));
        const double sz = dsub(1.0, (double)fsub(q2, f2));
        const int fs = (int)fadd(Cf, f0), ms = (int)fadd(Cf, f1), ss = (int)f2;
        const double tm = dmul(val, a.mult);
        const double xf[2] = {sf, dsub(1.0, sf)}, yf[2] = {sm, dsub(1.0, sm)},
                     zf[2] = {sz, dsub(1.0, sz)};
#pragma unroll
        for (int cz = 0; cz < 2; cz++)
#pragma unroll
            for (int cy = 0; cy < 2; cy++)
#pragma unroll
                for (int cx = 0; cx < 2; cx++) {
                    const double w = dmul(dmul(xf[cx], yf[cy]), zf[cz]);
                    add_positive_ss<EACH>(a, fs + cx, ms + cy, ss + cz, d2u64(dmul(tm, w)));
                }
    }
}

// One distinct pair, the body of the reference's loop for i > ind
// (IAC/kernel.cl:493-649): any values, any interpolation.
template <int DMAP, int I1, int I2>
__device__ __forceinline__ void bin_pair(const SparseArgs &a, const float4 A, const float4 B,
                                         const float *R)
{
    float q0 = fsub(A.x, B.x), q1 = fsub(A.y, B.y), q2 = fsub(A.z, B.z);
    // sqrt(|q|^2) > MaxQ, decided on |q|^2 against the exact float threshold
    if (fadd(fadd(fmul(q0, q0), fmul(q1, q1)), fmul(q2, q2)) > a.maxq2) return;
    q0 = fmul(q0, a.vpdq);
    q1 = fmul(q1, a.vpdq);
    q2 = fmul(q2, a.vpdq);
    const int C = a.C;
    const float Cf = (float)C;
    if (I2 == 0 && (DMAP == 0 || I1 == 0)) {
        // nearest neighbour at the second level: value (ulong)(v_lo * v_hi * Mult)
        const unsigned long long v = d2u64(dmul(dmul((double)A.w, (double)B.w), a.mult));
        float t0 = q0, t1 = q1, t2 = q2;
        if (DMAP) {  // first-level nearest neighbour: back to the voxel centre
            // |q| <= MaxQ * Voxel_per_dq < 2^22 here (MaxQ test, host check)
            t0 = round_away_rz_f(q0);
            t1 = round_away_rz_f(q1);
            t2 = round_away_rz_f(q2);
        }
        add_nearest(a, rot_row(t0, t1, t2, R[0], R[1], R[2]), rot_row(t0, t1, t2, R[3], R[4], R[5]),
                    rot_row(t0, t1, t2, R[6], R[7], R[8]), v);
        return;
    }
    const double val = dmul((double)A.w, (double)B.w);
    if (DMAP) {
        if (I1 == 0) {
            const float r0 = round_away_rz_f(q0), r1 = round_away_rz_f(q1), r2 = round_away_rz_f(q2);
            add_rotated<I2>(a, val, rot_row(r0, r1, r2, R[0], R[1], R[2]),
                            rot_row(r0, r1, r2, R[3], R[4], R[5]),
                            rot_row(r0, r1, r2, R[6], R[7], R[8]));
        } else {
            const float f0 = floorf(q0), f1 = floorf(q1), f2 = floorf(q2);
            const double sf = dsub(1.0, (double)fsub(q0, f0));
            const double sm = dsub(1.0, (double)fsub(q1, f1));
            const double sz = dsub(1.0, (double)fsub(q2, f2));
            const int fs = (int)fadd(Cf, f0), ms = (int)fadd(Cf, f1), ss = (int)fadd(Cf, f2);
            const float base = (float)val;
            const double xf[2] = {sf, dsub(1.0, sf)}, yf[2] = {sm, dsub(1.0, sm)},
                         zf[2] = {sz, dsub(1.0, sz)};
#pragma unroll
            for (int cz = 0; cz < 2; cz++)
#pragma unroll
                for (int cy = 0; cy < 2; cy++)
#pragma unroll
                    for (int cx = 0; cx < 2; cx++) {
                        const float tv =
                            (float)dmul((double)base, dmul(dmul(xf[cx], yf[cy]), zf[cz]));
                        const float r0 = (float)((fs + cx) - C), r1 = (float)((ms + cy) - C),
                                    r2 = (float)((ss + cz) - C);
                        add_rotated<I2, I2 == 1>(a, (double)tv, rot_row(r0, r1, r2, R[0], R[1], R[2]),
                                                 rot_row(r0, r1, r2, R[3], R[4], R[5]),
                                                 rot_row(r0, r1, r2, R[6], R[7], R[8]));
                    }
        }
    } else {
        add_rotated<I2>(a, val, rot_row(q0, q1, q2, R[0], R[1], R[2]),
                        rot_row(q0, q1, q2, R[3], R[4], R[5]),
                        rot_row(q0, q1, q2, R[6], R[7], R[8]));
    }
}

// ---------------------------------------------------------------------------
// pair kernel
// ---------------------------------------------------------------------------
// One rotated pair of the fast path at its nearest voxel (add_nearest, for a q
// that is finite and inside the mesh): a negative slow component flips the sign
// of all three first, which is the reflection of a negative ss; the rounding is
// the sign-magnitude trunc(x + copysign(0.49999997, x)) of round_away_rz_i.
// What the box holds, and c: SUM_COUNTS sums of c, the product of the counts,
// which cannot leave 32 bits (the kernel checks the CTA's whole share), so its
// adds return nothing; SUM_SMALL the values c * Mult, below 2^32, with their
// carries as in put_pair; SUM_VALUES any values (c is the value).  The adds are
// predicated rather than branched around: nearly every warp has lanes on either
// side, and without branches the two pairs of a step overlap.
enum { SUM_COUNTS, SUM_SMALL, SUM_VALUES };
template <int SUM>
__device__ __forceinline__ void put_nearest(const SparseArgs &a, bool on, float x0, float x1, float x2,
                                            unsigned long long c)
{
    const bool box = fmaxf(fmaxf(fabsf(x0), fabsf(x1)), fabsf(x2)) < a.box_lim;
    const uint32_t sg = __float_as_uint(x2) & 0x80000000u;
    x0 = __uint_as_float(__float_as_uint(x0) ^ sg);
    x1 = __uint_as_float(__float_as_uint(x1) ^ sg);
    const int r0 = __float2int_rz(fadd(x0, copysignf(0.49999997f, x0)));
    const int r1 = __float2int_rz(fadd(x1, copysignf(0.49999997f, x1)));
    const int r2 = __float2int_rz(fadd(fabsf(x2), 0.49999997f));
    const uint32_t word = (uint32_t)(r0 + r1 * a.S + r2 * (int)a.plane + a.center);
    const uint32_t bat = a.box_base + 4u * (uint32_t)(r0 + r1 * (int)a.box_w + r2 * a.box_plane + a.box_center);
    const unsigned long long v = SUM == SUM_VALUES ? c : (unsigned long long)((uint32_t)c * a.mult_u);
    const int in_box = on && box, in_mesh = on && !box, mirrored = in_mesh && r2 == 0;
    if (SUM == SUM_COUNTS) {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %0, 0;\n\t@p red.shared.add.u32 [%1], %2;\n\t}" ::"r"(in_box),
                     "r"(bat), "r"((uint32_t)c)
                     : "memory");
    } else if (in_box) {
        uint32_t old;
        asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(bat), "r"((uint32_t)v) : "memory");
        uint32_t up = (uint32_t)(v >> 32) + (old + (uint32_t)v < old ? 1u : 0u);
        if (up) {
            if (r2 == 0 && word == (uint32_t)a.center) up *= 2;
            carry_out(a.half, word, r2 == 0 ? 2u * (uint32_t)a.center - word : word, up);
        }
    }
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %0, 0;\n\t@p red.global.add.L2::cache_hint.u64 [%1], %2, %3;\n\t}" ::"r"(
                     in_mesh),
                 "l"(&a.half[word]), "l"(v), "l"(a.mesh_policy)
                 : "memory");
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %0, 0;\n\t@p red.global.add.L2::cache_hint.u64 [%1], %2, %3;\n\t}" ::"r"(
                     mirrored),
                 "l"(&a.half[2u * (uint32_t)a.center - word]), "l"(v), "l"(a.mesh_policy)
                 : "memory");
}

template <int DMAP, int SUM>
__device__ __forceinline__ void nearest_unit(const SparseArgs &a, const float4 *__restrict__ P, uint32_t n, const float *R,
                                             uint32_t i, uint32_t d0, int steps)
{
    auto load = [&](uint32_t j) { return ld_photon_hint(P + j, a.photon_policy); };
    const float4 A = load(i);
    const float2 nz = make_float2(a.neg_zero, a.neg_zero);
    auto mul = [&](float2 x, float2 y) { return f2fma(x, y, nz); };
    auto dup = [](float x) { return make_float2(x, x); };
    uint32_t j = i + d0;
    if (j >= n) j -= n;
    auto step = [&](uint32_t x) { return x + 1 == n ? 0u : x + 1; };
    for (int k = 0; k < steps; k += 2) {
        const float4 B0 = load(j);
        j = step(j);
        const float4 B1 = load(j);
        j = step(j);
        float2 q0 = make_float2(fsub(A.x, B0.x), fsub(A.x, B1.x)), q1 = make_float2(fsub(A.y, B0.y), fsub(A.y, B1.y)),
               q2 = make_float2(fsub(A.z, B0.z), fsub(A.z, B1.z));
        // sqrt(|q|^2) > MaxQ, decided on |q|^2 against the exact float threshold
        const float2 s = f2add(f2add(mul(q0, q0), mul(q1, q1)), mul(q2, q2));
        q0 = mul(q0, dup(a.vpdq));
        q1 = mul(q1, dup(a.vpdq));
        q2 = mul(q2, dup(a.vpdq));
        if (DMAP) {  // first-level nearest neighbour: back to the voxel centre
            auto near = [](float2 x) {
                const float2 t = f2add(x, make_float2(copysignf(0.49999997f, x.x), copysignf(0.49999997f, x.y)));
                return make_float2(truncf(t.x), truncf(t.y));
            };
            q0 = near(q0);
            q1 = near(q1);
            q2 = near(q2);
        }
        auto row = [&](float r0, float r1, float r2) {
            return f2add(f2add(mul(q0, dup(r0)), mul(q1, dup(r1))), mul(q2, dup(r2)));
        };
        const float2 x0 = row(R[0], R[1], R[2]), x1 = row(R[3], R[4], R[5]), x2 = row(R[6], R[7], R[8]);
        // the double product of two counts is exact, as the float one is
        auto value = [&](float w) {
            return SUM == SUM_VALUES ? d2u64(dmul(dmul((double)A.w, (double)w), a.mult))
                                     : (unsigned long long)__float2uint_rz(fmul(A.w, w));
        };
        put_nearest<SUM>(a, s.x <= a.maxq2, x0.x, x1.x, x2.x, value(B0.w));
        put_nearest<SUM>(a, s.y <= a.maxq2 && k + 1 < steps, x0.y, x1.y, x2.y, value(B1.w));
    }
}

// Pairs of the fast path split over the eight voxels around their rotated q
// (add_rotated<1>).  The values stay below 2^24, so their floor is read from the
// low word of the double product rounded down to a multiple of one (an add of
// 2^52 toward zero) instead of a 64-bit conversion.  A pair whose eight voxels
// lie in the box adds there; of the others, neighbouring lanes exchange halves:
// both lanes add one pair's two voxels of a mesh row, adjacent words, with one
// instruction and then the other pair's, since L2 takes adjacent words of a
// request together (measured: 3.4e11 adds/s in pairs, 2.2e11 single).
template <int DMAP>
__device__ __forceinline__ void linear_unit(const SparseArgs &a, const float4 *__restrict__ P, uint32_t n, const float *R,
                                            uint32_t i, uint32_t d0, int steps, uint32_t L)
{
    const float4 A = ld_photon_hint(P + i, a.photon_policy);
    const int odd = threadIdx.x & 1;
    uint32_t j = i + d0;
    if (j >= n) j -= n;
    for (int k = 0; k < (int)L; k++) {  // all lanes: the exchange is warp-wide
        const float4 B = ld_photon_hint(P + j, a.photon_policy);
        const uint32_t flip = j < i ? 0x80000000u : 0u;  // q = k_lo - k_hi
        j = j + 1 == n ? 0u : j + 1;
        float q0 = fsub(A.x, B.x), q1 = fsub(A.y, B.y), q2 = fsub(A.z, B.z);
        bool on = k < steps && fadd(fadd(fmul(q0, q0), fmul(q1, q1)), fmul(q2, q2)) <= a.maxq2;
        auto scaled = [&](float q) {
            q = fmul(__uint_as_float(__float_as_uint(q) ^ flip), a.vpdq);
            return DMAP ? truncf(fadd(q, copysignf(0.49999997f, q))) : q;  // first level: the voxel centre
        };
        q0 = scaled(q0);
        q1 = scaled(q1);
        q2 = scaled(q2);
        const float x0 = rot_row(q0, q1, q2, R[0], R[1], R[2]), x1 = rot_row(q0, q1, q2, R[3], R[4], R[5]),
                    x2 = rot_row(q0, q1, q2, R[6], R[7], R[8]);
        const double val = (double)fmul(A.w, B.w);  // exact: counts <= 128
        const float m = fmaxf(fmaxf(fabsf(x0), fabsf(x1)), fabsf(x2));
        if (on && !(m < (float)a.C)) {  // a voxel outside the mesh
            add_rotated<1>(a, val, x0, x1, x2);
            on = false;
        }
        const float f0 = floorf(x0), f1 = floorf(x1), f2 = floorf(x2);
        const double sf = dsub(1.0, (double)fsub(x0, f0)), sm = dsub(1.0, (double)fsub(x1, f1)),
                     sz = dsub(1.0, (double)fsub(x2, f2));
        const double tm = dmul(val, a.mult);
        const double yf[2] = {sm, dsub(1.0, sm)}, zf[2] = {sz, dsub(1.0, sz)}, xf[2] = {sf, dsub(1.0, sf)};
        uint32_t v[4][2];  // [2 cz + cy][cx]
#pragma unroll
        for (int cy = 0; cy < 2; cy++)
#pragma unroll
            for (int cx = 0; cx < 2; cx++) {
                const double w = dmul(xf[cx], yf[cy]);
#pragma unroll
                for (int cz = 0; cz < 2; cz++)
                    v[2 * cz + cy][cx] = (uint32_t)__double2loint(__dadd_rz(dmul(tm, dmul(w, zf[cz])), 4503599627370496.0));
            }
        const int b0 = __float2int_rz(f0), b1 = __float2int_rz(f1), b2 = __float2int_rz(f2);
        // the word of corner (cx, cy, cz) is the centre's plus its offset, or minus
        // it for a negative slow index (the point reflection)
        const bool in_box = on && m < a.box_lim - 0.5f;  // box_r: every corner within it
        if (in_box) {
            const int bl = b0 + b1 * (int)a.box_w + b2 * a.box_plane, ml = b0 + b1 * a.S + b2 * (int)a.plane;
            uint32_t carry = 0;
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int cx = 0; cx < 2; cx++) {
                    const int off = bl + (r & 1) * (int)a.box_w + (r >> 1) * a.box_plane + cx;
                    const int at = a.box_center + (b2 + (r >> 1) < 0 ? -off : off);
                    const uint32_t old = box_add32(a, (uint32_t)at, v[r][cx]);
                    carry |= (old + v[r][cx] < old ? 1u : 0u) << (2 * r + cx);
                }
            while (carry) {
                const int b = __ffs(carry) - 1, r = b >> 1;
                carry &= carry - 1;
                const int off = ml + (r & 1) * a.S + (r >> 1) * (int)a.plane + (b & 1), s = b2 + (r >> 1);
                const uint32_t word = (uint32_t)(a.center + (s < 0 ? -off : off));
                const uint32_t mirror = s == 0 ? 2u * (uint32_t)a.center - word : word;
                carry_out(a.half, word, mirror, s == 0 && word == mirror ? 2u : 1u);
            }
        }
        const bool in_mesh = on && !in_box;
        if (__any_sync(0xffffffffu, in_mesh)) {
            const int ml = b0 + b1 * a.S + b2 * (int)a.plane;
            const int state = in_mesh ? b2 : -0x40000000;  // the partner's slow index, or nothing to add
            const int pml = __shfl_xor_sync(0xffffffffu, ml, 1), pstate = __shfl_xor_sync(0xffffffffu, state, 1);
            uint32_t own[4], got[4];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                own[r] = odd ? v[r][1] : v[r][0];
                got[r] = __shfl_xor_sync(0xffffffffu, odd ? v[r][0] : v[r][1], 1);
            }
#pragma unroll
            for (int turn = 0; turn < 2; turn++) {  // the even lane's pair, then the odd lane's
                const bool mine = turn == odd;
                const int base = (mine ? ml : pml) + odd, s0 = mine ? state : pstate;
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int off = base + (r & 1) * a.S + (r >> 1) * (int)a.plane, s = s0 + (r >> 1);
                    const uint32_t word = (uint32_t)(a.center + (s < 0 ? -off : off));
                    const uint32_t val32 = mine ? own[r] : got[r];
                    if (s > -0x20000000 && val32) {
                        mesh_add(a, word, val32);
                        if (s == 0) mesh_add(a, 2u * (uint32_t)a.center - word, val32);
                    }
                }
            }
        }
    }
}

// threads of a CTA at most: all that share a box at 64 registers (linear second level: 680 us for
// 3.6e7 pairs of a 129^3 mesh, 750 at 512 threads), fewer where 64 first-level corners each go on
constexpr int pair_threads(int dmap, int i1, int i2) { return dmap && i1 ? 512 : 1024; }

// One CTA per SM, whose warps take chunks of the batch (walk_share); its box of
// the voxels around q = 0 takes their adds in shared memory and goes to the half
// mesh once, at the end.  Bound by the L2 request rate of the adds outside the
// box and by issue slots, about evenly: 89 instructions per 32 pairs (164 with
// a thread per pair, its two loads and its index arithmetic), 100 000 frames
// 4.3 ms (5.8 with a work queue, a barrier per frame and R = 9), one event of
// 164 photons 10 us (three launches, 36 us), linear second level on 3.6e7 pairs
// of a 129^3 mesh 0.67 ms (1.5).
template <int DMAP, int I1, int I2>
__global__ void __launch_bounds__(pair_threads(DMAP, I1, I2), 1) sparse_pairs_kernel(SparseArgs a)
{
    constexpr bool FAST = DMAP == 0 || I1 == 0;
    __shared__ unsigned long long s_off[PAIR_DIRECT + 1];
    __shared__ unsigned long long s_sums[32];
    __shared__ uint32_t s_next, s_taken, s_worst[32];
    __shared__ uint32_t s_flags[PAIR_DIRECT];
    extern __shared__ uint32_t s_box[];  // (box_r + 1) x box_w x box_w low words, [ss][ms][fs]
    a.mesh_policy = a.cache_hints ? l2_policy_evict_last() : l2_policy_normal();
    a.photon_policy = a.cache_hints ? l2_policy_evict_first() : l2_policy_normal();
    const uint32_t nthr = blockDim.x;
    const int lane = threadIdx.x & 31;
    const unsigned long long *off = a.walk.head ? a.walk.cost_off : s_off;
    const PlanHeader h = a.walk.head ? *a.walk.head : plan_direct(a.walk, gridDim.x * (nthr / 32), s_off, s_sums);
    const Share share = cta_share(h, a.walk.head != nullptr);
    if (share.x0 >= share.x1) return;  // a CTA without work (uniform over the block)
    if (threadIdx.x == 0) s_next = s_taken = 0u;
    uint32_t worst = 0;  // the largest flag of the batch
    if (FAST && a.fast_ok && a.check_here) {  // the planner's check, for the frames of this CTA
        for (uint32_t f = threadIdx.x; f < a.walk.nframes; f += nthr) s_flags[f] = 1u;
        __syncthreads();
        for (uint32_t f = warp_find_frame(off, a.walk.nframes, share.x0); f < a.walk.nframes && off[f] < share.x1; f++) {
            const uint64_t b = a.walk.offsets[f], e = a.walk.offsets[f + 1];
            uint32_t m = threadIdx.x >= 3 || fast_row(a.rot + 9 * (size_t)f + 3 * threadIdx.x, a.row_limit2) ? 1u : FLAG_GENERAL;
            for (uint64_t i = b + threadIdx.x; i < e; i += nthr) m = max(m, fast_count(a.walk.photons[i]));
            if (m > 128u) atomicMax(&s_flags[f], m);
            worst = max(worst, m);
        }
    } else if (FAST && a.fast_ok) {
        const uint32_t words = a.walk.nframes / 16;
        const uint4 *fl = reinterpret_cast<const uint4 *>(a.flags);
        uint32_t most = 0, least = 0xffffffffu;  // of the bytes
        for (uint32_t k = threadIdx.x; k < words; k += nthr) {
            const uint4 x = fl[k];
            most = __vmaxu4(__vmaxu4(most, __vmaxu4(x.x, x.y)), __vmaxu4(x.z, x.w));
            least = __vminu4(__vminu4(least, __vminu4(x.x, x.y)), __vminu4(x.z, x.w));
        }
        for (uint32_t f = 16 * words + threadIdx.x; f < a.walk.nframes; f += nthr) {
            most = __vmaxu4(most, a.flags[f]);
            least = __vminu4(least, 0xffffff00u | a.flags[f]);
        }
        for (int k = 0; k < 32; k += 8) {
            worst = max(worst, (most >> k) & 255u);
            if (((least >> k) & 255u) == 0) worst = FLAG_GENERAL;
        }
    }
    worst = __reduce_max_sync(0xffffffffu, worst);
    if (lane == 0) s_worst[threadIdx.x >> 5] = worst;
    // the box pays where its voxels collect many adds per CTA: its flush costs
    // one coalesced mesh add per voxel
    a.box_r = h.pairs < BOX_PAIRS_SMALL ? -1 : h.pairs < BOX_PAIRS_LARGE ? min(a.box_max, BOX_R_SMALL) : a.box_max;
    a.box_w = a.box_r >= 0 ? 2u * a.box_r + 1u : 0u;
    a.box_plane = (int)(a.box_w * a.box_w);
    a.box_center = a.box_r >= 0 ? a.box_r + a.box_r * (int)a.box_w : 0;
    a.box_lim = a.box_r >= 0 ? (float)a.box_r + 0.5f : 0.0f;
    a.center = a.C + a.C * a.S;
    a.box_base = (uint32_t)__cvta_generic_to_shared(s_box);
    const uint32_t box_n = (uint32_t)(a.box_r + 1) * a.box_w * a.box_w;
    for (uint32_t k = threadIdx.x; k < box_n; k += nthr) s_box[k] = 0u;
    __syncthreads();
    for (uint32_t w = 0; w < nthr / 32; w++) worst = max(worst, s_worst[w]);
    // 32 pairs per unit of cost; a chunk's last unit may reach past it
    const bool counts = FAST && I2 == 0 && a.fast_ok && a.mult_u && worst <= 128u &&
                        (unsigned long long)share.most * (share.chunk + h.steps + PAIR_UNIT_COST) * 32 * (worst * worst) <
                            (1ull << 32);

    float R[9];
    const float4 *__restrict__ P = nullptr;
    uint32_t n = 0;
    uint32_t flag = FLAG_GENERAL;
    unsigned long long self = 0;  // self pairs (q = 0) of this lane
    walk_share(
        a.walk, h, off, share, a.walk.head ? &a.walk.head->next : &s_next, &s_taken,
        [&](uint32_t f, uint64_t base, uint32_t nf) {
            P = a.walk.photons + base;
            n = nf;
            if (FAST && a.fast_ok) {
                flag = a.check_here ? s_flags[f] : a.flags[f];
                if (flag == 0) flag = FLAG_GENERAL;
                if (flag <= 128u && !a.mult_u) flag = FLAG_VALUES;
            }
#pragma unroll
            for (int k = 0; k < 9; k++) R[k] = a.rot[9 * (size_t)f + k];
        },
        [&](uint32_t i, uint32_t c, bool active, uint32_t nc, uint32_t L) {
            uint32_t d0;
            int steps;
            chunk_steps(n, i, c, L, active, d0, steps);
            if (active && c == 0) {
                const double v = (double)P[i].w;
                self += d2u64(dmul(dmul(v, v), a.mult));
            }
            if (FAST && I2 && flag <= 128u) {
                linear_unit<DMAP>(a, P, n, R, i, d0, steps, L);
            } else if (FAST && !I2 && counts) {
                nearest_unit<DMAP, SUM_COUNTS>(a, P, n, R, i, d0, steps);
            } else if (FAST && !I2 && flag <= 128u) {
                nearest_unit<DMAP, SUM_SMALL>(a, P, n, R, i, d0, steps);
            } else if (FAST && !I2 && flag == FLAG_VALUES) {
                nearest_unit<DMAP, SUM_VALUES>(a, P, n, R, i, d0, steps);
            } else {
                uint32_t j = i + d0;
                if (j >= n) j -= n;
                for (int k = 0; k < steps; k++) {
                    bin_pair<DMAP, I1, I2>(a, P[min(i, j)], P[max(i, j)], R);
                    if (++j == n) j = 0;
                }
            }
        });
    for (int o = 16; o; o >>= 1) self += __shfl_xor_sync(0xffffffffu, self, o);
    if (lane == 0 && self) mesh_add(a, (uint32_t)a.C + (uint32_t)a.C * (uint32_t)a.S, self);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < box_n; k += nthr) {
        const unsigned long long v = counts ? (unsigned long long)s_box[k] * a.mult_u : s_box[k];
        if (v == 0) continue;
        const uint32_t ss = k / (a.box_w * a.box_w), r = k - ss * (a.box_w * a.box_w);
        const uint32_t ms = (uint32_t)(a.C - a.box_r) + r / a.box_w;
        const uint32_t fs = (uint32_t)(a.C - a.box_r) + r % a.box_w;
        const uint32_t word = fs + ms * (uint32_t)a.S + ss * a.plane;
        mesh_add(a, word, v);
        if (ss == 0) mesh_add(a, 2u * (uint32_t)a.center - word, v);
    }
}

// ---------------------------------------------------------------------------
// fold: full[fs, ms, ss + C] += half; full[2C - fs, 2C - ms, C - ss] += half
// for ss > 0 (IAC/Detector.cpp:1147-1170).  Every full-mesh voxel receives
// exactly one half-mesh voxel, so plain read-modify-write suffices.
// ---------------------------------------------------------------------------
__global__ void sparse_fold_kernel(const unsigned long long *__restrict__ half, uint32_t S,
                                   unsigned long long *__restrict__ full)
{
    const uint32_t C = (S - 1) / 2;
    const uint64_t plane = (uint64_t)S * S;
    const uint64_t total = plane * ((S + 1) / 2);
    for (uint64_t h = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; h < total;
         h += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t ss = (uint32_t)(h / plane);
        const uint32_t rem = (uint32_t)(h - (uint64_t)ss * plane);
        const uint32_t ms = rem / S, fs = rem - ms * S;
        const unsigned long long v = half[h];
        if (v == 0) continue;
        full[fs + (uint64_t)ms * S + (uint64_t)(ss + C) * plane] += v;
        if (ss != 0) full[(2 * C - fs) + (uint64_t)(2 * C - ms) * S + (uint64_t)(C - ss) * plane] += v;
    }
}

// ---------------------------------------------------------------------------
// AC_UW of sparse photon lists: both routes of Calculate_AC_UW_Mapped
// (IAC/AC1D.cpp:248-379).  The reference picks a route per frame: with fewer
// than 0.75 % of the detector's pixels hit ((float)n / (float)pixels < 0.0075f,
// :251-253) it loops on the host over k >= j (:254-293); otherwise it launches
// AutoCorr_sparseHL_AAV (IAC/kernel.cl:863-950, host side :295-379).
//
// Device route: every ordered pair of a frame, self pairs included, adds
// (uint64)(v_a * v_b * Mult) at bin floor(|q|/dq + 0.5) (nearest) or splits
// it over floor(|q|/dq) and the next bin (linear).  The two orders of a
// distinct pair give the same |q| and value, so each distinct pair adds twice
// its value.  Bins are taken modulo VecSize, which is what the reference's
// sub-histogram layout and index-modulo fold (IAC/AC1D.cpp:366-375) do to bins
// at or beyond VecSize.
//
// Host route: every unordered pair k >= j adds the float 2*(v_j*v_k)
// (nearest), or 2*((v_j*v_k)*(1-Sep)) and 2*((v_j*v_k)*Sep) (linear), to a
// double histogram of Size bins; the factor 2 also doubles the self pair.
// These floats are whole numbers for photon counts (nearest): those are summed
// in uint64, exactly, so the double totals equal the reference's sequential
// double sums bit for bit.  Fractions from counts (linear) are multiples of
// fix_top 2^-23 past the first bins, because |q| / dq has 24 bits and some of them
// go to the bin; those are summed in these units, exactly too: 32-bit shared adds
// are native, while a double add in shared memory is a loop of compare-and-swaps.
// Adding and taking off fix_top tells whether a value is one.  The rest is summed
// with double atomics, whose order differs from the reference's loop by rounding
// only, as are all fractions when the histograms leave no room for the
// fixed-point one.
//
// The histograms live in shared memory for the whole launch.  The walk over the
// batch and its planner are the pair kernel's: a warp's lanes take consecutive
// photons i and step through partners two at a time, the squared distances in
// f32x2, |q| / dq by the two-word reciprocal; the order of a pair's photons
// changes neither |q| nor the value.  A unit belongs to one frame, so the route
// branch is uniform across the warp.  Issue-bound (84 %, 117 instructions a pair):
// 20 000 frames (2.2e8 pairs, 2048 bins) 1578 -> 884 us linear, 979 -> 590 nearest;
// with double adds the linear walk took 1100.  Device route, 2 000 frames of 230
// photons, 950 bins: 455 -> 288 us linear, 347 -> 239 nearest.
// ---------------------------------------------------------------------------
// b % n without the division when b < n (bins past the histogram are rare)
__device__ __forceinline__ uint32_t wrap_bin(uint32_t b, uint32_t n)
{
    if (b >= n) b %= n;
    return b;
}

struct AC1DArgs {
    WalkArgs walk;
    DeviceCounters *counters;
    double mult;
    float maxq, dqdx;
    Divisor by_dq;
    float neg_zero;
    uint32_t vecsize;   // device-route bins (VecSize)
    uint32_t size;      // host-route bins (Shape.Size; 0 when no frame takes the host route)
    int divide;         // dq is too large or small for by_dq
    int fixed;          // the fixed-point histogram has room
    float fix_top;      // its values are below this, in units of fix_top 2^-23
    uint32_t fix_mask;  // the units' fraction bits
    float det_pixels;   // (float) detector pixel count, for the route choice
    int route;          // -1: the reference's choice per frame, 0: host route, 1: device route
    unsigned long long *dev_out;  // vecsize words
    unsigned long long *int_out;  // size words: host-route whole-number values
    double *frac_out;             // size doubles: host-route other values
};

// shared-memory histograms of one CTA: 64-bit counters as split 32-bit words
// (shared_add_u64_split), host-route fractions in units of fix_top 2^-23 or as doubles
struct AC1DHist {
    uint32_t *dev_lo, *dev_hi;  // vecsize words each
    unsigned long long *whole;  // size split words, then size doubles
    uint32_t *fix_lo, *fix_hi;  // size words each (if fixed)
};

__device__ __forceinline__ uint32_t shared_add32(uint32_t at, uint32_t v)
{
    uint32_t old;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(at), "r"(v) : "memory");
    return old;
}
// host-route value v (>= 0) into a bin of the whole-number histogram (split words)
// and the doubles behind it
__device__ __forceinline__ void host_route_add(unsigned long long *whole, uint32_t size, DeviceCounters *counters,
                                               uint32_t bin, float v)
{
    if (bin >= size) {  // only for inconsistent MaxQ / dq; the reference writes out of bounds
        atomicAdd(&counters->out_of_mesh, 1ull);
        return;
    }
    if (v == 0.0f) return;
    uint32_t *lo = reinterpret_cast<uint32_t *>(whole), *hi = lo + size;
    double *frac = reinterpret_cast<double *>(whole + size);
    if (v > 0.0f && v < 8388608.0f) {  // the usual case, without conversion-unit instructions
        const float t = __fadd_rz(v, 8388608.0f);  // 2^23 + floor(v)
        if (fsub(t, 8388608.0f) == v)
            shared_add_u64_split(lo, hi, bin, (unsigned long long)(uint32_t)(__float_as_int(t) - TWO23_BITS));
        else
            atomicAdd(&frac[bin], (double)v);
        return;
    }
    if (v >= 8388608.0f && v < 4294967296.0f)  // a whole number of 32 bits
        shared_add_u64_split(lo, hi, bin, (unsigned long long)__float2uint_rz(v));
    else if (v == truncf(v) && v < 1.8e19f)
        shared_add_u64_split(lo, hi, bin, (unsigned long long)__float2ull_rz(v));
    else
        atomicAdd(&frac[bin], (double)v);
}
// twice floor(x) of a device-route value into bin
__device__ __forceinline__ void device_route_add(const AC1DArgs &b, const AC1DHist &h, uint32_t bin, double x)
{
    const unsigned long long w = d2u64(x);
    if (w) shared_add_u64_split(h.dev_lo, h.dev_hi, wrap_bin(bin, b.vecsize), 2ull * w);
}

// 20 000 frames, linear, by threads x CTAs per SM, before the device route's walk took
// registers of it: 512 x 2 857 us (884 now), 512 x 3 823, 768 x 2 817, 1024 x 1 855; 200
// frames 39, 57, 47 and 52: a short batch pays for each CTA.
constexpr int AC1D_THREADS = 512, AC1D_PER_SM = 2;
// batches planned by the CTAs themselves: 1000 frames 79 us, with the planner's launch 87
constexpr uint32_t AC1D_DIRECT = 1024;
template <int INTERP>
__global__ void __launch_bounds__(2 * AC1D_THREADS, 1) ac1d_sparse_kernel(const AC1DArgs a)
{
    __shared__ unsigned long long s_off[AC1D_DIRECT + 1];
    __shared__ unsigned long long s_sums[32];
    __shared__ uint32_t s_next, s_taken;
    extern __shared__ unsigned long long hist[];
    AC1DHist h;
    h.dev_lo = reinterpret_cast<uint32_t *>(hist);
    h.dev_hi = h.dev_lo + a.vecsize;
    h.whole = hist + a.vecsize;
    h.fix_lo = reinterpret_cast<uint32_t *>(hist + a.vecsize + 2 * a.size);
    h.fix_hi = h.fix_lo + a.size;
    const uint32_t nthr = blockDim.x;
    const unsigned long long *off = a.walk.head ? a.walk.cost_off : s_off;
    const PlanHeader head = a.walk.head ? *a.walk.head : plan_direct(a.walk, gridDim.x * (nthr / 32), s_off, s_sums);
    const Share share = cta_share(head, a.walk.head != nullptr);
    if (share.x0 >= share.x1) return;  // a CTA without work (uniform over the block)
    if (threadIdx.x == 0) s_next = s_taken = 0u;
    const uint32_t words = a.vecsize + (a.fixed ? 3 : 2) * a.size;
    for (uint32_t i = threadIdx.x; i < words; i += nthr) hist[i] = 0;  // 0 bits = +0.0
    __syncthreads();
    const uint32_t whole = (uint32_t)__cvta_generic_to_shared(h.whole), 
                   // without room every pair adds 0, at a word that exists
                   fixed = a.fixed ? (uint32_t)__cvta_generic_to_shared(h.fix_lo) : whole;
    const uint32_t dev = (uint32_t)__cvta_generic_to_shared(h.dev_lo);
    const uint32_t dev_bins = a.vecsize - INTERP;  // a pair's first bin below this: no bin wraps
    const uint32_t fix_bins = a.fixed ? a.size - 1 : 0u;  // a pair's first bin below this: both exist
    const float2 nz = make_float2(a.neg_zero, a.neg_zero);
    const float4 *__restrict__ P = nullptr;
    uint32_t n = 0;
    bool host = false;
    unsigned long long self_int = 0, self_dev = 0;  // this lane's self pairs: q = 0, bin 0
    walk_share(
        a.walk, head, off, share, a.walk.head ? &a.walk.head->next : &s_next, &s_taken,
        [&](uint32_t, uint64_t base, uint32_t nf) {
            P = a.walk.photons + base;
            n = nf;
            // SHLsizeQuot < 0.0075f (IAC/AC1D.cpp:251-253), in the reference's float arithmetic
            host = a.route == 0 || (a.route < 0 && __fdiv_rn(__uint2float_rn(n), a.det_pixels) < 0.0075f);
        },
        [&](uint32_t i, uint32_t c, bool active, uint32_t, uint32_t L) {
            uint32_t d0;
            int steps;
            chunk_steps(n, i, c, L, active, d0, steps);
            const float4 A = P[i];
            if (active && c == 0) {  // linear: bin 0 gets all of it, bin 1 nothing
                if (host) {
                    const float v = fmul(2.0f, fmul(A.w, A.w));
                    if (v == truncf(v) && v < 1.8e19f)
                        self_int += __float2ull_rz(v);
                    else
                        host_route_add(h.whole, a.size, a.counters, 0, v);
                } else {
                    const double v = (double)A.w;
                    self_dev += d2u64(dmul(dmul(v, v), a.mult));
                }
            }
            uint32_t j = i + d0;
            if (j >= n) j -= n;
            for (int k = 0; k < (int)L; k += 2) {
                const float4 B0 = P[j];
                if (++j == n) j = 0;
                const float4 B1 = P[j];
                if (++j == n) j = 0;
                const float2 dx = f2sub(make_float2(A.x, A.x), make_float2(B0.x, B1.x)),
                             dy = f2sub(make_float2(A.y, A.y), make_float2(B0.y, B1.y)),
                             dz = f2sub(make_float2(A.z, A.z), make_float2(B0.z, B1.z));
                const float2 s = f2add(f2add(f2fma(dx, dx, nz), f2fma(dy, dy, nz)), f2fma(dz, dz, nz));
                const float2 r = make_float2(__fsqrt_rn(s.x), __fsqrt_rn(s.y));
                float2 qq;
                if (a.divide)
                    qq = make_float2(__fdiv_rn(r.x, a.dqdx), __fdiv_rn(r.y, a.dqdx));
                else
                    qq = f2div(r, a.by_dq);
                const bool on[2] = {k < steps && !(r.x > a.maxq), k + 1 < steps && !(r.y > a.maxq)};
                const float q[2] = {qq.x, qq.y}, bw[2] = {B0.w, B1.w};
                if (INTERP == 0 && host) {
                    uint32_t bin[2], u[2], old[2];
                    float v[2];
                    bool rare[2];
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        // (uint)floor(q + 0.5) in double, as floor(fl(q + 0.49999997f)) for q < 2^23
                        floor_small(fadd(q[e], 0.49999997f), bin[e]);
                        v[e] = fmul(2.0f, fmul(A.w, bw[e]));
                        const bool fast = floor_small(v[e], u[e]) == v[e] && u[e] < (1u << 23) && bin[e] < a.size;
                        rare[e] = on[e] && !fast;
                        u[e] = on[e] && fast ? u[e] : 0u;
                    }
                    if (!__any_sync(0xffffffffu, rare[0] || rare[1])) {
#pragma unroll
                        for (int e = 0; e < 2; e++) old[e] = shared_add32(whole + (u[e] ? 4u * bin[e] : 0u), u[e]);
                        if (old[0] + u[0] < old[0]) shared_add32(whole + 4u * (a.size + bin[0]), 1u);
                        if (old[1] + u[1] < old[1]) shared_add32(whole + 4u * (a.size + bin[1]), 1u);
                    } else {
#pragma unroll
                        for (int e = 0; e < 2; e++)
                            if (on[e]) host_route_add(h.whole, a.size, a.counters, bin[e], v[e]);
                    }
                } else if (host) {
                    uint32_t at[2], bin[2], u[4];
                    float v[4];
                    bool rare[2], c[4];
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        // q = |q| / dq <= MaxQ / dq < 2^23
                        const float fq = floor_small(q[e], bin[e]);
                        const float sep = fsub(q[e], fq), pv = fmul(A.w, bw[e]);
                        v[2 * e] = fmul(2.0f, fmul(pv, fsub(1.0f, sep)));
                        v[2 * e + 1] = fmul(2.0f, fmul(pv, sep));
                        const bool in = on[e] && bin[e] < fix_bins;
                        at[e] = in ? fixed + 4u * bin[e] : fixed;  // off: adds 0
                        bool ok[2];
#pragma unroll
                        for (int m = 0; m < 2; m++) {
                            const float x = v[2 * e + m], s = fadd(x, a.fix_top);
                            const uint32_t w = __float_as_uint(s) - __float_as_uint(a.fix_top);
                            // below the top, exact, and no whole number
                            ok[m] = in && w < (1u << 23) && fsub(s, a.fix_top) == x && (w & a.fix_mask) != 0;
                            u[2 * e + m] = ok[m] ? w : 0u;
                        }
                        rare[e] = on[e] && !(ok[0] && ok[1]);
                    }
                    if (__any_sync(0xffffffffu, (u[0] | u[1] | u[2] | u[3]) != 0u)) {
#pragma unroll
                        for (int m = 0; m < 4; m++) c[m] = shared_add32(at[m >> 1] + 4u * (m & 1), u[m]) + u[m] < u[m];
                        if (c[0] | c[1] | c[2] | c[3]) {
#pragma unroll
                            for (int m = 0; m < 4; m++)
                                if (c[m]) shared_add32(at[m >> 1] + 4u * (m & 1) + 4u * a.size, 1u);
                        }
                    }
                    if (rare[0] || rare[1]) {
#pragma unroll
                        for (int m = 0; m < 4; m++)
                            if (u[m] == 0 && on[m >> 1]) host_route_add(h.whole, a.size, a.counters, bin[m >> 1] + (m & 1), v[m]);
                    }
                } else {
                    constexpr int N = INTERP ? 2 : 1;  // bins of a pair
                    uint32_t at[2], bin[2], u[2 * N];
                    double x[2 * N];
                    bool rare[2], c[2 * N], any = false;
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const double val = dmul((double)A.w, (double)bw[e]);
                        if (INTERP == 0) {
                            floor_small(fadd(q[e], 0.49999997f), bin[e]);  // as above
                            x[e] = dmul(val, a.mult);
                        } else {
                            const float fq = floor_small(q[e], bin[e]);
                            const double sep = (double)fsub(q[e], fq);
                            x[N * e] = dmul(dmul(val, dsub(1.0, sep)), a.mult);
                            x[N * e + N - 1] = dmul(dmul(val, sep), a.mult);
                        }
                        const bool in = on[e] && bin[e] < dev_bins;
                        at[e] = in ? dev + 4u * bin[e] : dev;  // off: adds 0
                        bool ok = in;
#pragma unroll
                        for (int m = N * e; m < N * e + N; m++) {  // twice floor(x), x in [0, 2^31)
                            const bool small = (uint32_t)__double2hiint(x[m]) < 0x41E00000u;
                            u[m] = in && small ? 2u * (uint32_t)__double2loint(__dadd_rz(x[m], 4503599627370496.0)) : 0u;
                            ok = ok && small;
                        }
                        rare[e] = on[e] && !ok;
                    }
#pragma unroll
                    for (int m = 0; m < 2 * N; m++) {
                        c[m] = shared_add32(at[m / N] + 4u * (m % N), u[m]) + u[m] < u[m];
                        any = any || c[m];
                    }
                    if (any) {
#pragma unroll
                        for (int m = 0; m < 2 * N; m++)
                            if (c[m]) shared_add32(at[m / N] + 4u * (m % N) + 4u * a.vecsize, 1u);
                    }
                    if (rare[0] || rare[1]) {
#pragma unroll 1
                        for (int m = 0; m < 2 * N; m++) {
                            const bool second = m >= N, last = m % N != 0;
                            const double y = second ? (last ? x[2 * N - 1] : x[N]) : (last ? x[N - 1] : x[0]);
                            const uint32_t b = second ? bin[1] : bin[0];
                            const bool small = b < dev_bins && (uint32_t)__double2hiint(y) < 0x41E00000u;
                            if ((second ? rare[1] : rare[0]) && !small) device_route_add(a, h, b + last, y);
                        }
                    }
                }
            }
        });
    uint32_t *int_lo = reinterpret_cast<uint32_t *>(h.whole), *int_hi = int_lo + a.size;
    const double *frac = reinterpret_cast<double *>(h.whole + a.size);
    for (int o = 16; o; o >>= 1) {
        self_int += __shfl_xor_sync(0xffffffffu, self_int, o);
        self_dev += __shfl_xor_sync(0xffffffffu, self_dev, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (self_int) shared_add_u64_split(int_lo, int_hi, 0, self_int);
        if (self_dev) shared_add_u64_split(h.dev_lo, h.dev_hi, 0, self_dev);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < a.vecsize; i += nthr) {
        const unsigned long long v = split_word(h.dev_lo, h.dev_hi, i);
        if (v) atomicAdd(&a.dev_out[i], v);
    }
    for (uint32_t i = threadIdx.x; i < a.size; i += nthr) {
        const unsigned long long v = split_word(int_lo, int_hi, i);
        if (v) atomicAdd(&a.int_out[i], v);
        double f = frac[i];
        if (a.fixed) f = dadd(f, dmul(__ull2double_rn(split_word(h.fix_lo, h.fix_hi, i)), (double)a.fix_top * 0x1p-23));
        if (f != 0.0) atomicAdd(&a.frac_out[i], f);
    }
}

// AC_UW[j] = dev[j] / Mult (j < VecSize) + int[j] + frac[j]
__global__ void ac1d_uw_finish_kernel(const unsigned long long *__restrict__ dev,
                                      const unsigned long long *__restrict__ in, const double *__restrict__ fr,
                                      uint32_t vecsize, uint32_t size, double mult, double *__restrict__ ac)
{
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= size) return;
    double v = j < vecsize ? __ddiv_rn((double)dev[j], mult) : 0.0;
    v = dadd(v, (double)in[j]);
    ac[j] = dadd(v, fr[j]);
}

typedef void (*PairKernel)(SparseArgs);

constexpr size_t pair_box_bytes(int r) { return sizeof(uint32_t) * (r + 1) * (2 * r + 1) * (2 * r + 1); }
constexpr size_t AC1D_HIST_BYTES = 216u << 10;  // of an AC1D CTA's histograms at most

static PairKernel pick_kernel(int dmap, int i1, int i2)
{
    if (!dmap) return i2 ? sparse_pairs_kernel<0, 0, 1> : sparse_pairs_kernel<0, 0, 0>;
    if (i1 == 0) return i2 ? sparse_pairs_kernel<1, 0, 1> : sparse_pairs_kernel<1, 0, 0>;
    return i2 ? sparse_pairs_kernel<1, 1, 1> : sparse_pairs_kernel<1, 1, 0>;
}

iac_status pair_kernel_limits()
{
    const PairKernel pair[] = {sparse_pairs_kernel<0, 0, 0>, sparse_pairs_kernel<0, 0, 1>, sparse_pairs_kernel<1, 0, 0>,
                               sparse_pairs_kernel<1, 0, 1>, sparse_pairs_kernel<1, 1, 0>, sparse_pairs_kernel<1, 1, 1>};
    for (PairKernel k : pair)
        IAC_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pair_box_bytes(BOX_R_MAX)));
    for (auto k : {ac1d_sparse_kernel<0>, ac1d_sparse_kernel<1>})
        IAC_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AC1D_HIST_BYTES));
    return IAC_OK;
}

// Explicit settings win; otherwise the autotuner row of the nearest mesh edge;
// otherwise built-in defaults.
static iac_sparse_tuning effective_tuning(iac_ctx *ctx, uint32_t size_ab)
{
    iac_sparse_tuning t;
    {
        std::lock_guard<std::mutex> lk(ctx->mu);
        t = ctx->tuning;
        if (!ctx->tuning_table.empty() && size_ab >= 2) {
            const uint32_t edge = size_ab - 2;
            const iac_ctx::TuningRow *best = nullptr;
            for (const auto &r : ctx->tuning_table)
                if (!best || (r.edge > edge ? r.edge - edge : edge - r.edge) <
                                 (best->edge > edge ? best->edge - edge : edge - best->edge))
                    best = &r;
            if (t.tile_pairs == 0) t.tile_pairs = best->tile_pairs;
            if (t.block_threads == 0) t.block_threads = best->block_threads;
            if (t.ctas_per_sm == 0) t.ctas_per_sm = best->ctas_per_sm;
            if (t.cache_hints == 0) t.cache_hints = best->cache_hints;
        }
    }
    if (t.tile_pairs == 0) t.tile_pairs = 4096;
    if (t.block_threads == 0) t.block_threads = 256;
    if (t.ctas_per_sm == 0) t.ctas_per_sm = 4;
    return t;
}

// Largest float s with sqrtf(s) <= m: since IEEE sqrt is monotonic,
// sqrtf(x) > m exactly when x > s (host sqrtf is correctly rounded like the
// device's __fsqrt_rn).
static float sqrt_threshold(float m)
{
    if (!(m >= 0.0f) || std::isinf(m)) return m;
    float s = m * m;
    while (std::sqrt(s) > m) s = std::nextafter(s, 0.0f);
    for (;;) {
        const float n = std::nextafter(s, INFINITY);
        if (std::isinf(n) || std::sqrt(n) > m) break;
        s = n;
    }
    return s;
}

static iac_status check_params(const iac_sparse_params *p)
{
    IAC_REQUIRE(p != nullptr, "sparse params are NULL");
    const iac_mesh_shape &s = p->shape;
    IAC_REQUIRE(s.size_ab >= 5 && (s.size_ab % 2) == 1 && s.size_c == s.size_ab,
                "sparse pair mesh must be cubic with an odd edge (got %u x %u)", s.size_ab, s.size_c);
    IAC_REQUIRE(s.size_ab <= 1621, "mesh edge %u too large (at most 1621)", s.size_ab);
    IAC_REQUIRE(s.voxel_per_dq > 0, "Voxel_per_dq is 0");
    IAC_REQUIRE((double)s.max_q * s.voxel_per_dq <= 4194304.0,
                "MaxQ * Voxel_per_dq must be at most 2^22 voxels (got %g)", (double)s.max_q * s.voxel_per_dq);
    IAC_REQUIRE(p->interp_first == 0 || p->interp_first == 1, "interp_first must be 0 or 1");
    IAC_REQUIRE(p->interp_second == 0 || p->interp_second == 1, "interp_second must be 0 or 1");
    IAC_REQUIRE(p->multiplicator > 0, "multiplicator must be positive");
    return IAC_OK;
}

// Threads of a CTA: block_threads x ctas_per_sm of the tuning setting, up to
// max_threads, which take all of an SM's registers.  The warps of a CTA share one box,
// and a larger box keeps more adds out of L2.  Settings of 2 048 and 4 096 threads an
// SM, 200 frames: 88 and 158 us as two and four CTAs, which wait for one another, 33
// as one.
static int pair_cta_threads(const iac_sparse_tuning &tun, int max_threads)
{
    return std::max(32, std::min(max_threads, (int)(tun.block_threads * tun.ctas_per_sm) / 32 * 32));
}

// Plan of one batch: planner header, table of frame starts
// (nframes + 1), per-frame flags (nframes bytes).
struct QueueMem {
    unsigned long long *cost_off;
    PlanHeader *head;
    unsigned char *flags;
};

// Planner with its count check, and pair kernel of one batch into the half mesh
// d_half.  Batches of up to PAIR_DIRECT frames are planned by the pair kernel's
// own CTAs in shared memory: a live event is one launch instead of three.
static iac_status launch_pair_batch(iac_ctx *ctx, const float *d_photons, const uint64_t *d_off,
                                    const float *d_rot9, uint32_t nframes, const iac_sparse_params *p,
                                    const QueueMem &q, uint64_t *d_half, cudaStream_t s)
{
    const iac_sparse_tuning tun = effective_tuning(ctx, p->shape.size_ab);
    const int i1 = p->double_map ? p->interp_first : 0;
    const int C = ((int)p->shape.size_ab - 1) / 2;
    const int threads = pair_cta_threads(tun, pair_threads(p->double_map, i1, p->interp_second));
    // one CTA an SM.  A first-level linear pair is 8 or 64 pairs' work: two CTAs an SM, one
    // after the other, and the smaller box that two had, even out the ends and leave the
    // walk its L1 (3 000 frames nearest on the second level 1342 us; one CTA 1395, with
    // R = 22 1464; 200 frames 142, 156 and 156)
    const bool heavy = p->double_map && i1;
    const int grid = ctx->sm_count * (heavy ? 2 : 1);
    const bool direct = nframes <= PAIR_DIRECT;
    SparseArgs a{};
    a.walk.photons = reinterpret_cast<const float4 *>(d_photons);
    a.walk.offsets = d_off;
    a.walk.head = direct ? nullptr : q.head;
    a.walk.cost_off = q.cost_off;
    a.walk.nframes = nframes;
    a.walk.steps_max = std::min(PAIR_STEPS_MAX, std::max(1u, tun.tile_pairs / 32));
    a.rot = d_rot9;
    a.half = reinterpret_cast<unsigned long long *>(d_half);
    a.counters = ctx->d_counters;
    a.S = (int)p->shape.size_ab;
    a.C = C;
    a.half_ss = (a.S + 1) / 2;
    a.plane = (uint32_t)a.S * (uint32_t)a.S;
    a.maxq2 = sqrt_threshold(p->shape.max_q);
    a.vpdq = (float)p->shape.voxel_per_dq;
    a.neg_zero = -0.0f;
    a.mult = p->multiplicator;
    a.mult_u = p->multiplicator >= 1.0 && p->multiplicator <= 1024.0 &&
                       p->multiplicator == std::floor(p->multiplicator)
                   ? (uint32_t)p->multiplicator
                   : 0u;
    a.fast_ok = std::isfinite(a.maxq2);
    a.check_here = direct ? 1 : 0;
    a.flags = q.flags;
    a.cache_hints = tun.cache_hints == 1 ? 1 : 0;
    a.box_max = std::min(heavy ? BOX_R_HEAVY : BOX_R_MAX, C);
    // |x| <= |row| (MaxQ Voxel_per_dq + the first level's rounding) < C + 1/2, with a margin for FP32
    const double reach = ((double)p->shape.max_q * p->shape.voxel_per_dq + 0.8661) * 1.00001;
    const double limit = ((double)C + 0.49) / reach;
    a.row_limit2 = std::isfinite(limit) ? (float)(limit * limit * 0.99999) : -1.0f;
    if (p->interp_second) a.row_limit2 = 1e12f;  // the linear path looks at every pair
    if (!direct) {
        const unsigned check = std::min<unsigned>((nframes + PLAN_THREADS / 32 - 1) / (PLAN_THREADS / 32),
                                                  2u * (unsigned)ctx->sm_count);
        const unsigned ctas = PLAN_CTAS + (check + PLAN_CTAS - 1) / PLAN_CTAS * PLAN_CTAS;
        sparse_plan_kernel<<<ctas, PLAN_THREADS, 0, s>>>(d_off, nframes, a.walk.steps_max,
                                                         (uint32_t)(grid * threads / 32), q.cost_off, q.head,
                                                         a.walk.photons, d_rot9, a.row_limit2, q.flags);
        IAC_LAUNCHED(ctx);
        IAC_CUDA(cudaGetLastError());
    }
    const size_t box_bytes = pair_box_bytes(a.box_max);
    const PairKernel k = pick_kernel(p->double_map, p->interp_first, p->interp_second);
    k<<<grid, threads, box_bytes, s>>>(a);
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    return IAC_OK;
}

// Planner and AC1D kernel of one batch (shared memory: both routes' histograms).
static iac_status launch_ac1d_batch(iac_ctx *ctx, const float *d_photons, const uint64_t *d_off,
                                    uint32_t nframes, int interp, double mult, const AC1DArgs &b, void *stream)
{
    DeviceGuard g(ctx->device);
    const iac_sparse_tuning tun = effective_tuning(ctx, 0);
    void *scratch = nullptr;
    const size_t table_bytes = ((sizeof(unsigned long long) * ((size_t)nframes + 1) + 127) / 128) * 128;
    iac_status st = stream_scratch(ctx, stream, SLOT_TILES, table_bytes + 128 + nframes, &scratch);
    if (st != IAC_OK) return st;
    cudaStream_t s = as_stream(stream);
    AC1DArgs a = b;
    // the fixed-point histogram where two CTAs an SM (one, for large shapes) still fit
    const size_t plain = sizeof(unsigned long long) * ((size_t)b.vecsize + 2 * (size_t)b.size),
                 more = sizeof(unsigned long long) * b.size;
    a.fixed = interp == 1 && b.size > 1 && plain + more <= AC1D_HIST_BYTES;
    const size_t smem = plain + (a.fixed ? more : 0);
    // |q| / dq from 2^e on is a multiple of 2^(e - 23): with 2^(e + 1) for the top, the
    // counts' values are too; the first 2^e bins, 1/32 of them, see few of the pairs
    int e = 2;
    while (e < 6 && (64u << (e - 1)) <= b.size) e++;
    a.fix_top = (float)(2u << e);
    a.fix_mask = (1u << (22 - e)) - 1;
    const int per_sm = (int)std::max<size_t>(1, std::min<size_t>(AC1D_PER_SM, (208u << 10) / std::max<size_t>(smem, 1)));
    // shapes that leave one CTA an SM: twice the threads, unless the batch is short (3435
    // bins, 1008 frames 92.7 -> 81.2 us; 4000 bins, 300 frames 27.8 -> 35.3)
    const int grid = ctx->sm_count * per_sm, threads = per_sm == 1 && nframes > 512 ? 2 * AC1D_THREADS : AC1D_THREADS;
    const bool direct = nframes <= AC1D_DIRECT;
    unsigned long long *cost_off = (unsigned long long *)scratch;
    PlanHeader *head = (PlanHeader *)((char *)scratch + table_bytes);
    a.walk.photons = reinterpret_cast<const float4 *>(d_photons);
    a.walk.offsets = d_off;
    a.walk.head = direct ? nullptr : head;
    a.walk.cost_off = cost_off;
    a.walk.nframes = nframes;
    a.walk.steps_max = std::min(PAIR_STEPS_MAX, std::max(1u, tun.tile_pairs / 32));
    a.counters = ctx->d_counters;
    a.by_dq = make_divisor(b.dqdx);
    a.divide = !(b.dqdx > 1e-30f && b.dqdx < 1e30f);
    a.neg_zero = -0.0f;
    a.mult = mult;
    if (!direct) {  // without the count check
        sparse_plan_kernel<<<PLAN_CTAS, PLAN_THREADS, 0, s>>>(d_off, nframes, a.walk.steps_max,
                                                              (uint32_t)(grid * threads / 32), cost_off, head,
                                                              a.walk.photons, nullptr, 0.0f, nullptr);
        IAC_LAUNCHED(ctx);
        IAC_CUDA(cudaGetLastError());
    }
    auto k = interp == 0 ? ac1d_sparse_kernel<0> : ac1d_sparse_kernel<1>;
    k<<<grid, threads, smem, s>>>(a);
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    return IAC_OK;
}

}  // namespace iac

using namespace iac;

extern "C" {

iac_status iac_sparse_set_tuning(iac_ctx *ctx, const iac_sparse_tuning *t)
{
    IAC_REQUIRE(ctx && t, "iac_sparse_set_tuning: NULL argument");
    IAC_REQUIRE(t->block_threads == 0 || (t->block_threads % 32 == 0 && t->block_threads <= 256 &&
                                          t->block_threads >= 64),
                "block_threads must be a multiple of 32 in [64, 256]");
    IAC_REQUIRE(t->tile_pairs == 0 || t->tile_pairs >= 64, "tile_pairs must be >= 64");
    IAC_REQUIRE(t->ctas_per_sm <= 32, "ctas_per_sm must be <= 32");
    IAC_REQUIRE(t->cache_hints <= 2, "cache_hints must be 0 (table), 1 (on) or 2 (off)");
    std::lock_guard<std::mutex> lk(ctx->mu);
    ctx->tuning = *t;
    return IAC_OK;
}

iac_status iac_sparse_get_tuning(iac_ctx *ctx, uint32_t size_ab, iac_sparse_tuning *t)
{
    IAC_REQUIRE(ctx && t, "iac_sparse_get_tuning: NULL argument");
    *t = effective_tuning(ctx, size_ab);
    return IAC_OK;
}

iac_status iac_sparse_ac_batch(iac_ctx *ctx, const float *d_photons, const uint64_t *d_off,
                               const float *d_rot9, uint32_t nframes, const iac_sparse_params *p,
                               uint64_t *d_half, void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx != nullptr, "iac_sparse_ac_batch: ctx is NULL");
    iac_status st = check_params(p);
    if (st != IAC_OK) return st;
    if (nframes == 0) return IAC_OK;
    IAC_REQUIRE(d_photons && d_off && d_rot9 && d_half, "iac_sparse_ac_batch: NULL pointer");
    IAC_REQUIRE((reinterpret_cast<uintptr_t>(d_photons) & 15) == 0,
                "photon array must be 16-byte aligned (float4 per photon)");
    DeviceGuard g(ctx->device);
    void *scratch = nullptr;
    const size_t table_bytes = ((sizeof(unsigned long long) * ((size_t)nframes + 1) + 127) / 128) * 128;
    st = stream_scratch(ctx, stream, SLOT_TILES, table_bytes + 128 + nframes, &scratch);
    if (st != IAC_OK) return st;
    const QueueMem q{(unsigned long long *)scratch, (PlanHeader *)((char *)scratch + table_bytes),
                     (unsigned char *)scratch + table_bytes + 128};
    return launch_pair_batch(ctx, d_photons, d_off, d_rot9, nframes, p, q, d_half, as_stream(stream));
}

iac_status iac_ac1d_sparse_batch(iac_ctx *ctx, const float *d_photons, const uint64_t *d_off,
                                 uint32_t nframes, float max_q, float dqdx, int interp,
                                 double mult, uint64_t *d_hist, void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx != nullptr, "iac_ac1d_sparse_batch: ctx is NULL");
    IAC_REQUIRE(interp == 0 || interp == 1, "interpolation must be 0 or 1");
    IAC_REQUIRE(dqdx > 0 && max_q > 0, "iac_ac1d_sparse_batch: MaxQ and dq must be positive");
    IAC_REQUIRE(mult > 0, "multiplicator must be positive");
    const uint32_t vecsize = iac_ac1d_vecsize(max_q, dqdx);
    IAC_REQUIRE(vecsize >= 1 && vecsize <= 24576, "VecSize %u out of range [1, 24576]", vecsize);
    if (nframes == 0) return IAC_OK;
    IAC_REQUIRE(d_photons && d_off && d_hist, "iac_ac1d_sparse_batch: NULL pointer");
    IAC_REQUIRE((reinterpret_cast<uintptr_t>(d_photons) & 15) == 0,
                "photon array must be 16-byte aligned (float4 per photon)");
    AC1DArgs b{};
    b.maxq = max_q;
    b.dqdx = dqdx;
    b.vecsize = vecsize;
    b.size = 0;
    b.det_pixels = 1.0f;
    b.route = 1;
    b.dev_out = (unsigned long long *)d_hist;
    return launch_ac1d_batch(ctx, d_photons, d_off, nframes, interp, mult, b, stream);
}

uint64_t iac_ac1d_uw_words(const iac_ac1d_shape *sh)
{
    if (!sh || !(sh->dq_per_step > 0) || !(sh->max_q > 0)) return 0;
    return (uint64_t)iac_ac1d_vecsize(sh->max_q, sh->dq_per_step) + 2ull * sh->size;
}

iac_status iac_ac1d_uw_batch(iac_ctx *ctx, const float *d_photons, const uint64_t *d_off, uint32_t nframes,
                             uint64_t detector_pixels, const iac_ac1d_shape *sh, int interp, int route,
                             uint64_t *d_acc, void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx != nullptr && sh != nullptr, "iac_ac1d_uw_batch: NULL argument");
    IAC_REQUIRE(interp == 0 || interp == 1, "interpolation must be 0 or 1");
    IAC_REQUIRE(route >= -1 && route <= 1, "route must be -1 (per frame), 0 (host) or 1 (device)");
    IAC_REQUIRE(sh->dq_per_step > 0 && sh->max_q > 0, "iac_ac1d_uw_batch: MaxQ and dq must be positive");
    IAC_REQUIRE(detector_pixels > 0 && detector_pixels < (1ull << 32),
                "iac_ac1d_uw_batch: detector pixel count %llu out of range", (unsigned long long)detector_pixels);
    const uint32_t vecsize = iac_ac1d_vecsize(sh->max_q, sh->dq_per_step);
    IAC_REQUIRE(sh->size >= 3 && vecsize >= 1, "AC1D size %u too small", sh->size);
    IAC_REQUIRE((uint64_t)vecsize + 2ull * sh->size <= 24576,
                "AC1D size %u too large: VecSize + 2 Size must be at most 24576 (shared-memory histograms)",
                sh->size);
    if (nframes == 0) return IAC_OK;
    IAC_REQUIRE(d_photons && d_off && d_acc, "iac_ac1d_uw_batch: NULL pointer");
    IAC_REQUIRE((reinterpret_cast<uintptr_t>(d_photons) & 15) == 0,
                "photon array must be 16-byte aligned (float4 per photon)");
    IAC_REQUIRE((reinterpret_cast<uintptr_t>(d_acc) & 7) == 0, "accumulator must be 8-byte aligned");
    AC1DArgs b{};
    b.maxq = sh->max_q;
    b.dqdx = sh->dq_per_step;
    b.vecsize = vecsize;
    b.size = sh->size;
    b.det_pixels = (float)detector_pixels;
    b.route = route;
    b.dev_out = (unsigned long long *)d_acc;
    b.int_out = b.dev_out + vecsize;
    b.frac_out = reinterpret_cast<double *>(b.int_out + sh->size);
    return launch_ac1d_batch(ctx, d_photons, d_off, nframes, interp, 100.0, b, stream);
}

iac_status iac_ac1d_uw_finish(iac_ctx *ctx, const uint64_t *d_acc, const iac_ac1d_shape *sh, double *d_ac_uw,
                              void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx && sh && d_acc && d_ac_uw, "iac_ac1d_uw_finish: NULL argument");
    IAC_REQUIRE(sh->dq_per_step > 0 && sh->max_q > 0 && sh->size >= 3, "iac_ac1d_uw_finish: bad shape");
    const uint32_t vecsize = iac_ac1d_vecsize(sh->max_q, sh->dq_per_step);
    DeviceGuard g(ctx->device);
    const unsigned long long *dev = (const unsigned long long *)d_acc;
    ac1d_uw_finish_kernel<<<(sh->size + 255) / 256, 256, 0, as_stream(stream)>>>(
        dev, dev + vecsize, reinterpret_cast<const double *>(dev + vecsize + sh->size), vecsize, sh->size, 100.0,
        d_ac_uw);
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    return IAC_OK;
}

uint32_t iac_ac1d_vecsize(float max_q, float dqdx)
{
    return (uint32_t)((int)std::ceil(max_q / dqdx) - 1);
}

iac_status iac_sparse_fold(iac_ctx *ctx, const uint64_t *d_half, uint32_t S, uint64_t *d_full,
                           void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx && d_half && d_full, "iac_sparse_fold: NULL argument");
    IAC_REQUIRE(S >= 3 && (S % 2) == 1 && S <= 2047, "iac_sparse_fold: bad mesh edge %u", S);
    DeviceGuard g(ctx->device);
    sparse_fold_kernel<<<ctx->sm_count * 4, 256, 0, as_stream(stream)>>>(
        reinterpret_cast<const unsigned long long *>(d_half), S,
        reinterpret_cast<unsigned long long *>(d_full));
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    return IAC_OK;
}

}  // extern "C"

namespace iac {

// Streams and events of the host-buffer entry points, created on first use.
static iac_status host_streams(iac_ctx *ctx)
{
    std::lock_guard<std::mutex> lk(ctx->mu);
    if (!ctx->host_stream) IAC_CUDA(cudaStreamCreateWithFlags(&ctx->host_stream, cudaStreamNonBlocking));
    if (!ctx->copy_stream) IAC_CUDA(cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking));
    if (!ctx->copy_events[0])
        for (auto &e : ctx->copy_events) IAC_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    if (!ctx->staging_free[0])
        for (auto &e : ctx->staging_free) IAC_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return IAC_OK;
}

// Host photon lists -> device staging (scratch of `key`) -> pair kernel into
// d_half on stream s.  Two staging sets alternate between calls, so a call's
// copies overlap the previous call's binning; each set is reused only after
// the binning that read it (staging_free).  When the previous call's binning
// is still running (a run of consecutive calls) the whole batch is copied
// behind it and binned in one launch.  Otherwise the frames are cut into
// chunks by photon count, chunk k+1 copied on the copy stream while chunk k
// is binned; binning is slower than the copy, so only the first chunk's copy
// is exposed: it is made a quarter of the others (1/29 of the photons for 8
// chunks).  Every chunk has its own rebased offsets so it is an independent
// batch.
static iac_status stage_and_bin(iac_ctx *ctx, const float *h_photons, const uint64_t *h_off, const float *h_rot9,
                                uint32_t nframes, const iac_sparse_params *p, uint64_t *d_half, cudaStream_t s,
                                void *key)
{
    iac_status st;
    cudaStream_t cs = ctx->copy_stream;
    const int set = ctx->staging_set;
    ctx->staging_set ^= 1;
    const bool behind = cudaEventQuery(ctx->staging_free[set ^ 1]) == cudaErrorNotReady;
    const uint64_t o0 = h_off[0];
    const uint64_t nph = h_off[nframes] - o0;
    const uint32_t nchunks =
        behind ? 1u : std::max<uint32_t>(1, std::min<uint32_t>(IAC_COPY_CHUNKS, nframes / 64));
    std::vector<uint32_t> cut(nchunks + 1, 0);
    cut[nchunks] = nframes;
    const uint64_t parts = 4 * (uint64_t)nchunks - 3;  // chunk 0: 1 part, the others 4
    for (uint32_t k = 1; k < nchunks; k++) {
        const uint64_t target = o0 + nph * (4 * (uint64_t)k - 3) / parts;
        cut[k] = (uint32_t)(std::lower_bound(h_off, h_off + nframes + 1, target) - h_off);
        cut[k] = std::max(cut[k], cut[k - 1]);
    }
    void *d_ph, *d_off, *d_rot;
    const int sp = set ? SLOT_PHOTONS2 : SLOT_PHOTONS, so = set ? SLOT_OFFSETS2 : SLOT_OFFSETS,
              sr = set ? SLOT_ROT2 : SLOT_ROT;
    if ((st = stream_scratch(ctx, key, sp, 16 * nph + 16, &d_ph)) != IAC_OK) return st;
    if ((st = stream_scratch(ctx, key, so, 8 * ((size_t)nframes + IAC_COPY_CHUNKS + 1), &d_off)) != IAC_OK)
        return st;
    if ((st = stream_scratch(ctx, key, sr, 36 * (size_t)nframes, &d_rot)) != IAC_OK) return st;
    std::vector<uint64_t> off((size_t)nframes + nchunks);
    size_t w = 0;
    std::vector<size_t> off_pos(nchunks);
    for (uint32_t k = 0; k < nchunks; k++) {
        off_pos[k] = w;
        for (uint32_t f = cut[k]; f <= cut[k + 1]; f++) off[w++] = h_off[f] - h_off[cut[k]];
    }
    {   // size the plan's scratch for the largest chunk now: growing it
        // between chunk launches would synchronise the device
        void *t = nullptr;
        const size_t tb = ((sizeof(unsigned long long) * ((size_t)nframes + 1) + 127) / 128) * 128;
        if ((st = stream_scratch(ctx, key, SLOT_TILES, tb + 128 + nframes, &t)) != IAC_OK) return st;
    }
    // the binning that last read this staging set is done before it is overwritten
    IAC_CUDA(cudaStreamWaitEvent(cs, ctx->staging_free[set], 0));
    IAC_CUDA(cudaMemcpyAsync(d_off, off.data(), 8 * w, cudaMemcpyHostToDevice, cs));
    for (uint32_t k = 0; k < nchunks; k++) {
        const uint32_t f0 = cut[k], f1 = cut[k + 1];
        const uint64_t p0 = h_off[f0] - o0, p1 = h_off[f1] - o0;
        if (p1 > p0)
            IAC_CUDA(cudaMemcpyAsync((char *)d_ph + 16 * p0, h_photons + 4 * (o0 + p0), 16 * (p1 - p0),
                                     cudaMemcpyHostToDevice, cs));
        if (f1 > f0)
            IAC_CUDA(cudaMemcpyAsync((char *)d_rot + 36 * (size_t)f0, h_rot9 + 9 * (size_t)f0,
                                     36 * (size_t)(f1 - f0), cudaMemcpyHostToDevice, cs));
        IAC_CUDA(cudaEventRecord(ctx->copy_events[k], cs));
        IAC_CUDA(cudaStreamWaitEvent(s, ctx->copy_events[k], 0));
        if (f1 > f0) {
            st = iac_sparse_ac_batch(ctx, (const float *)((char *)d_ph + 16 * p0),
                                     (const uint64_t *)d_off + off_pos[k], (const float *)d_rot + 9 * (size_t)f0,
                                     f1 - f0, p, d_half, (void *)s);
            if (st != IAC_OK) return st;
        }
    }
    IAC_CUDA(cudaEventRecord(ctx->staging_free[set], s));
    return IAC_OK;
}

}  // namespace iac

extern "C" {

iac_status iac_sparse_ac_frames_host(iac_ctx *ctx, const float *h_photons,
                                     const uint64_t *h_off, const float *h_rot9, uint32_t nframes,
                                     const iac_sparse_params *p, uint64_t *h_full)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx != nullptr, "iac_sparse_ac_frames_host: ctx is NULL");
    iac_status st = check_params(p);
    if (st != IAC_OK) return st;
    IAC_REQUIRE(h_off && h_full, "iac_sparse_ac_frames_host: NULL pointer");
    if (nframes == 0) return IAC_OK;
    IAC_REQUIRE(h_photons && h_rot9, "iac_sparse_ac_frames_host: NULL pointer");
    DeviceGuard g(ctx->device);
    std::lock_guard<std::mutex> hl(ctx->host_mu);
    if ((st = host_streams(ctx)) != IAC_OK) return st;
    cudaStream_t s = ctx->host_stream, cs = ctx->copy_stream;
    void *key = (void *)s;
    const uint32_t S = p->shape.size_ab;
    const size_t half_b = sizeof(uint64_t) * iac_half_mesh_words(S);
    const size_t full_b = sizeof(uint64_t) * iac_full_mesh_words(S);
    void *d_half, *d_full;
    if ((st = stream_scratch(ctx, key, SLOT_HALF, half_b, &d_half)) != IAC_OK) return st;
    if ((st = stream_scratch(ctx, key, SLOT_FULL, full_b, &d_full)) != IAC_OK) return st;
    IAC_CUDA(cudaMemsetAsync(d_half, 0, half_b, s));
    if ((st = stage_and_bin(ctx, h_photons, h_off, h_rot9, nframes, p, (uint64_t *)d_half, s, key)) != IAC_OK)
        return st;
    // the mesh the caller holds, uploaded behind the photon stream
    const uint32_t ev = IAC_COPY_CHUNKS;
    IAC_CUDA(cudaMemcpyAsync(d_full, h_full, full_b, cudaMemcpyHostToDevice, cs));
    IAC_CUDA(cudaEventRecord(ctx->copy_events[ev], cs));
    IAC_CUDA(cudaStreamWaitEvent(s, ctx->copy_events[ev], 0));
    st = iac_sparse_fold(ctx, (const uint64_t *)d_half, S, (uint64_t *)d_full, key);
    if (st != IAC_OK) return st;
    IAC_CUDA(cudaMemcpyAsync(h_full, d_full, full_b, cudaMemcpyDeviceToHost, s));
    IAC_CUDA(cudaStreamSynchronize(s));
    return IAC_OK;
}

iac_status iac_sparse_ac_frames_host_to_device(iac_ctx *ctx, const float *h_photons, const uint64_t *h_off,
                                               const float *h_rot9, uint32_t nframes, const iac_sparse_params *p,
                                               uint64_t *d_half, void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx != nullptr, "iac_sparse_ac_frames_host_to_device: ctx is NULL");
    iac_status st = check_params(p);
    if (st != IAC_OK) return st;
    IAC_REQUIRE(h_off && d_half, "iac_sparse_ac_frames_host_to_device: NULL pointer");
    if (nframes == 0) return IAC_OK;
    IAC_REQUIRE(h_photons && h_rot9, "iac_sparse_ac_frames_host_to_device: NULL pointer");
    DeviceGuard g(ctx->device);
    std::lock_guard<std::mutex> hl(ctx->host_mu);
    if ((st = host_streams(ctx)) != IAC_OK) return st;
    cudaStream_t s = as_stream(stream);
    if ((st = stage_and_bin(ctx, h_photons, h_off, h_rot9, nframes, p, d_half, s, stream)) != IAC_OK) return st;
    // the host buffers have been read once the copies are done; binning goes on
    IAC_CUDA(cudaStreamSynchronize(ctx->copy_stream));
    return IAC_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free variant of iac_sparse_ac_batch.
//
// Some callers may not allocate device memory once they are running: a
// detector acquisition loop that cannot absorb the device-wide
// synchronisation and unbounded latency a cudaMalloc/cudaFree can cause, or a
// host framework that hands out all device memory from its own pool and
// forbids allocations behind its back.  iac_sparse_ac_batch grows a per-stream
// scratch buffer on first use; this entry point instead keeps the same
// plan (table of frame starts, chunk counter, per-frame flags) in a fixed array of
// device memory that is part of the loaded library, so it never allocates.
//
// The array's name in host code only stands in for the symbol; the kernels
// need its device address, which cudaGetSymbolAddress gives.  The context
// looks it up once, when it is created (iac_ctx_create, with its device
// current: the step that may load the library's device code and place the
// array on that device), and keeps it; the entry point itself only reads it.
// A context does not outlive a reset of its device (cudaDeviceReset ends every
// context's device state), so the kept address is never stale while the
// context is usable.  The array is shared by every call on the device and
// keeps the previous call's contents: the planner kernel rewrites the whole
// table and resets the counter before the pair kernel reads them,
// so nothing has to be cleared from the host, but two calls running on the
// GPU at the same time (e.g. on two streams) would overwrite each other's
// plan.
// ---------------------------------------------------------------------------
namespace iac {

constexpr uint32_t STATIC_MAX_FRAMES = 200000;
constexpr size_t STATIC_TABLE_BYTES =
    ((sizeof(unsigned long long) * ((size_t)STATIC_MAX_FRAMES + 1) + 255) / 256) * 256;
constexpr size_t STATIC_QUEUE_BYTES = 256;
constexpr size_t STATIC_SCRATCH_BYTES = STATIC_TABLE_BYTES + STATIC_QUEUE_BYTES + STATIC_MAX_FRAMES;

static __device__ __align__(256) unsigned char g_sparse_static_scratch[STATIC_SCRATCH_BYTES];

iac_status static_scratch_setup(iac_ctx *ctx)
{
    DeviceGuard g(ctx->device);
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_sparse_static_scratch);
    if (e != cudaSuccess || !p) {
        set_error("cudaGetSymbolAddress of the fixed scratch failed on device %d: %s", ctx->device,
                  cudaGetErrorString(e));
        return IAC_ERR_CUDA;
    }
    ctx->static_scratch = p;
    return IAC_OK;
}

}  // namespace iac

extern "C" iac_status iac_sparse_ac_batch_static(iac_ctx *ctx, const float *d_photons,
                                                 const uint64_t *d_off, const float *d_rot9,
                                                 uint32_t nframes, const iac_sparse_params *p,
                                                 uint64_t *d_half, void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx != nullptr, "iac_sparse_ac_batch_static: ctx is NULL");
    iac_status st = check_params(p);
    if (st != IAC_OK) return st;
    if (nframes == 0) return IAC_OK;
    IAC_REQUIRE(d_photons && d_off && d_rot9 && d_half, "iac_sparse_ac_batch_static: NULL pointer");
    IAC_REQUIRE((reinterpret_cast<uintptr_t>(d_photons) & 15) == 0,
                "photon array must be 16-byte aligned (float4 per photon)");
    IAC_REQUIRE(nframes <= STATIC_MAX_FRAMES,
                "iac_sparse_ac_batch_static: %u frames requested; its fixed scratch holds the work "
                "queue of at most %u frames per call (split the batch or use iac_sparse_ac_batch)",
                nframes, STATIC_MAX_FRAMES);
    IAC_REQUIRE(ctx->static_scratch != nullptr, "iac_sparse_ac_batch_static: the context has no fixed scratch");
    DeviceGuard g(ctx->device);
    char *base = (char *)ctx->static_scratch;
    const QueueMem q{(unsigned long long *)base, (PlanHeader *)(base + STATIC_TABLE_BYTES),
                     (unsigned char *)base + STATIC_TABLE_BYTES + STATIC_QUEUE_BYTES};
    return launch_pair_batch(ctx, d_photons, d_off, d_rot9, nframes, p, q, d_half, as_stream(stream));
}
