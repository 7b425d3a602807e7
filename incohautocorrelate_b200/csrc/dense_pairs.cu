// dense_pairs.cu -- (b) dense mean-intensity C(q) on the small mesh and
// (c) the AC1D |q| histogram of the mean intensity.
//
// Replaces AutoCorr_CQ_small (IAC/kernel.cl:27-184, host
// Detector::AutoCorrelate_CofQ_SmallMesh, IAC/Detector.cpp:1184-1315) and
// AutoCorr_CQ_AV (IAC/kernel.cl:656-764, host AC1D::Calculate_CQ,
// IAC/AC1D.cpp:61-195).
//
// Both reference kernels visit every ordered pixel pair (ind, i), self pairs
// included.  The pair (i, ind) is the point reflection of (ind, i): q changes
// sign exactly, the value I_ind*I_i is the same float, and round()/floor()
// based binning is reflected exactly (nearest: round(-x) = -round(x); linear:
// the corner weights 1 - (x - floor x) of -x are the reflected weights of x,
// bit for bit).  So each unordered pair is evaluated once and its mesh
// contribution is added at the voxel and at its reflection through the mesh
// centre; for |q| the two orders are identical and the bin gets twice the
// value.  Self pairs (q = 0) are added once at the centre.
//
// Work decomposition.  Pixels are cut into tiles of 256: 16 x 16 patches of
// the detector when its row length is given, else 256 consecutive pixels.
// A persistent CTA pops tile pairs (P <= Q) from a queue: thread t owns pixel
// t of tile P and walks the TILE pixels of Q, staged in shared memory as float4
// (k, I).  Tile pairs whose k bounding boxes are farther apart than MaxQ are
// skipped whole.  Contributions are accumulated per thread while consecutive
// pixels of Q fall into the same voxel (row-adjacent pixels move q by a
// fraction of a voxel), then added to a shared-memory window covering the
// tile pair's q range, which is flushed to the global mesh (voxel and
// reflection) once per tile pair.  Tile pairs whose window would not fit fall
// back to global atomics.  The AC1D histogram lives in shared memory for the
// whole launch and is flushed once per CTA.
//
// All FP32 operations are the reference's, in its order, without FMA
// contraction; values are (uint64)(double(I_a*I_b) * Mult) per pair as the
// reference's casts do, so the integer meshes are bit-identical.
#include <algorithm>
#include <cmath>

#include "iac_internal.cuh"

namespace iac {

constexpr int DTILE = 256;        // pixels per tile == threads per CTA
// Shared-memory window: split 64-bit counters.  A tile pair whose q range is larger
// adds every pair, and its mirror, in L2 instead, which costs far more than the
// window's memory: as many words as six (linear: four) CTAs an SM leave room for.
// 2048, 4096 and 5440 words: linear 240 x 280, 253-edge mesh 128, 11.1 and 11.1 ms,
// 160 x 180 at 253 27.9 -> 15.7 from 4096 to 5440, 120 x 150 at 199 14.1, 11.5 and 2.7;
// nearest 120 x 150, 199-edge mesh 1.80 -> 0.55 ms from 2048 to 4096, but 300 x 350 at
// 253 6.34 -> 6.57 from 4096 to 5440, where only four CTAs fit.
template <int INTERP>
constexpr int WINDOW_WORDS = INTERP ? 5440 : 4096;

struct DenseArgs {
    const float *__restrict__ I;
    const float *__restrict__ K;     // 3 floats per pixel
    const float4 *__restrict__ box;  // per tile: min (x,y,z), max |I|; max (x,y,z), min I
    unsigned long long *__restrict__ out;
    unsigned long long *queue;
    DeviceCounters *counters;
    uint64_t npix;
    uint32_t ntiles;
    unsigned long long npairs;  // tile pairs
    uint32_t part, nparts;      // this launch takes the tile pairs p with p % nparts == part
    uint32_t nx, ny, ptx;       // 2D patch tiling: row length, rows, patches per row (nx = 0: linear)
    uint32_t mult_int;          // Multiplicator as an integer below 2^29, else 0
    int key_ok;                 // |round(q * Voxel_per_dq)| < 512 for every pair within MaxQ
    float maxq, maxq2;
    float vpdq;
    double mult;
    float mult_f;    // Multiplicator as a float when that is exact (and an integer), else 0
    float neg_zero;  // -0.0f: fma(x, y, -0) is x * y rounded once, and never merges with an add
    // C(q) small mesh
    int ab, sc, cab, cc;  // sizes and centres
    int ka, kb, kc;       // q axis on mesh fs / ms / ss
    // AC1D
    uint32_t hsize;
    float dq;
    Divisor by_dq;
    int in_range;  // no bin of a pair within MaxQ reaches hsize, and dq is a normal float
};

// tile-pair index -> (P, Q): first the ntiles diagonal pairs, then the
// circulant walk over distinct pairs (d = l / T + 1, P = l % T, Q = P + d mod T)
__device__ __forceinline__ void decode_tile_pair(unsigned long long p, uint32_t T, uint32_t &P,
                                                 uint32_t &Q)
{
    if (p < T) {
        P = Q = (uint32_t)p;
        return;
    }
    const unsigned long long l = p - T;
    const uint32_t d = (uint32_t)(l / T) + 1;
    P = (uint32_t)(l % T);
    Q = P + d;
    if (Q >= T) Q -= T;
}

// Pixel of slot j (0..255) of tile t.  With the row length known the tiles
// are 16 x 16 pixel patches, whose pair differences cover a few voxels, so the
// shared-memory window of a tile pair stays small; otherwise 256 consecutive
// pixels.  Returns npix for a slot outside the detector.
__device__ __forceinline__ uint64_t tile_pixel(const DenseArgs &a, uint32_t t, uint32_t j)
{
    if (a.nx) {
        const uint32_t py = t / a.ptx, px = t - py * a.ptx;
        const uint32_t y = py * 16 + (j >> 4), x = px * 16 + (j & 15);
        return (y < a.ny && x < a.nx) ? (uint64_t)y * a.nx + x : a.npix;
    }
    const uint64_t i = (uint64_t)t * DTILE + j;
    return i < a.npix ? i : a.npix;
}

// (uint64)((double)p * M) for finite p >= 0 and an integer M < 2^29: the double
// product of a 24-bit mantissa and M is exact, so the cast is the floor of the
// exact product, formed here in integers.
__device__ __forceinline__ unsigned long long scaled_floor(float p, uint32_t M)
{
    const uint32_t b = __float_as_uint(p);
    const int e = (int)((b >> 23) & 0xff);
    const uint64_t m = (b & 0x7fffffu) | (e ? 0x800000u : 0u);
    const int sh = (e ? e : 1) - 150;  // p = m * 2^sh
    const uint64_t prod = m * (uint64_t)M;
    if (sh >= 0) return prod << sh;
    return sh <= -64 ? 0ull : (prod >> (-sh));
}

__global__ void tile_box_kernel(const DenseArgs a, float4 *__restrict__ box)
{
    const uint32_t t = blockIdx.x;
    const uint64_t i = tile_pixel(a, t, threadIdx.x);
    const float *__restrict__ K = a.K;
    const float *__restrict__ I = a.I;
    float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    // largest |I| of the tile (infinite for a NaN or a k-vector that is not finite: the
    // tile then takes no fast path) and smallest I
    float imax = 0.0f, imin = 0.0f;
    if (i < a.npix && I[i] != 0.0f) {  // zero-intensity pixels never contribute
        bool finite = true;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            mn[d] = mx[d] = K[3 * i + d];
            finite = finite && fabsf(mn[d]) < INFINITY;
        }
        imax = fabsf(I[i]);
        imin = I[i];
        if (imax != imax || !finite) imax = INFINITY;
    }
#pragma unroll
    for (int d = 0; d < 3; d++)
        for (int o = 16; o; o >>= 1) {
            mn[d] = fminf(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
            mx[d] = fmaxf(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
        }
    for (int o = 16; o; o >>= 1) {
        imax = fmaxf(imax, __shfl_xor_sync(0xffffffffu, imax, o));
        imin = fminf(imin, __shfl_xor_sync(0xffffffffu, imin, o));
    }
    __shared__ float s[8][DTILE / 32];
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        for (int d = 0; d < 3; d++) {
            s[d][w] = mn[d];
            s[3 + d][w] = mx[d];
        }
        s[6][w] = imax;
        s[7][w] = imin;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float r[8];
        for (int d = 0; d < 8; d++) {
            r[d] = s[d][0];
            for (int j = 1; j < DTILE / 32; j++) r[d] = d < 3 || d == 7 ? fminf(r[d], s[d][j]) : fmaxf(r[d], s[d][j]);
        }
        box[2 * t] = make_float4(r[0], r[1], r[2], r[6]);
        box[2 * t + 1] = make_float4(r[3], r[4], r[5], r[7]);
    }
}

// lower bound of |k_a - k_b| over two boxes, inflated by a relative margin
__device__ __forceinline__ bool boxes_beyond(const float4 a0, const float4 a1, const float4 b0,
                                             const float4 b1, float maxq)
{
    const float gx = fmaxf(0.f, fmaxf(a0.x - b1.x, b0.x - a1.x));
    const float gy = fmaxf(0.f, fmaxf(a0.y - b1.y, b0.y - a1.y));
    const float gz = fmaxf(0.f, fmaxf(a0.z - b1.z, b0.z - a1.z));
    if (!(a0.x <= a1.x) || !(b0.x <= b1.x)) return true;  // an empty tile
    return sqrtf(gx * gx + gy * gy + gz * gz) > maxq * 1.0001f + 1e-6f;
}

__device__ __forceinline__ float pick(float x, float y, float z, int axis)
{
    return axis == 0 ? x : (axis == 1 ? y : z);
}

// --------------------------------------------------------------------------
// C(q) small mesh
// --------------------------------------------------------------------------
struct Window {
    int lo[3];  // first voxel (fs, ms, ss) of the window
    int dim[3];
    bool on;
};

__device__ __forceinline__ void global_put_pair(const DenseArgs &a, int fs, int ms, int ss,
                                                unsigned long long v)
{
    if (v == 0) return;
    if ((unsigned)fs >= (unsigned)a.ab || (unsigned)ms >= (unsigned)a.ab ||
        (unsigned)ss >= (unsigned)a.sc) {
        atomicAdd(&a.counters->out_of_mesh, 1ull);
    } else {
        atomicAdd(&a.out[(uint64_t)fs + (uint64_t)ms * a.ab + (uint64_t)ss * a.ab * a.ab], v);
    }
    const int rf = 2 * a.cab - fs, rm = 2 * a.cab - ms, rs = 2 * a.cc - ss;
    if ((unsigned)rf >= (unsigned)a.ab || (unsigned)rm >= (unsigned)a.ab ||
        (unsigned)rs >= (unsigned)a.sc) {
        atomicAdd(&a.counters->out_of_mesh, 1ull);
    } else {
        atomicAdd(&a.out[(uint64_t)rf + (uint64_t)rm * a.ab + (uint64_t)rs * a.ab * a.ab], v);
    }
}

template <int INTERP>
__device__ __forceinline__ void put(const DenseArgs &a, const Window &w, uint32_t *win,
                                    int fs, int ms, int ss, unsigned long long v)
{
    if (v == 0) return;
    const int x = fs - w.lo[0], y = ms - w.lo[1], z = ss - w.lo[2];
    if (w.on && (unsigned)x < (unsigned)w.dim[0] && (unsigned)y < (unsigned)w.dim[1] &&
        (unsigned)z < (unsigned)w.dim[2])
        shared_add_u64_split(win, win + WINDOW_WORDS<INTERP>, x + w.dim[0] * (y + w.dim[1] * z), v);
    else
        global_put_pair(a, fs, ms, ss, v);
}

// round half away from zero as an int: (int)trunc(x + copysign(0.5 - 2^-25, x)).
// The FP32 sum is correctly rounded and never reaches the next integer unless
// x is at or past the half, so this equals round(x) for every |x| < 2^23
// (checked exhaustively against roundf over all such floats).
__device__ __forceinline__ int round_half_away(float x)
{
    return __float2int_rz(fadd(x, copysignf(0.49999997f, x)));
}

// component of (x, y, z) on axis K (0..2), or the runtime axis k when K < 0
template <int K>
__device__ __forceinline__ float axis(float x, float y, float z, int k)
{
    if (K == 0) return x;
    if (K == 1) return y;
    if (K == 2) return z;
    return pick(x, y, z, k);
}

// the pairs (own pixel, staged pixels j0..TILE-1): the exact reference
// arithmetic, per-thread run-length accumulation of consecutive pairs that
// land in the same voxel.  KA/KB/KC: axis of q on mesh fs/ms/ss (-1: runtime).
// CHECK: apply the per-pair MaxQ test (skipped when the two tiles' bounding
// boxes are entirely within MaxQ, where every pair passes it).
template <int INTERP, int KA, int KB, int KC, bool CHECK>
__device__ __forceinline__ void cq_pairs(const DenseArgs &a, const Window &w, uint32_t *win,
                                         const float4 *sq, int j0, float k0, float k1, float k2, float Ia)
{
    int cur_f = 0, cur_m = 0, cur_s = 0;
    unsigned long long acc[INTERP ? 8 : 1];
#pragma unroll
    for (int c = 0; c < (INTERP ? 8 : 1); c++) acc[c] = 0;
    bool have = false;
    for (int j = j0; j < DTILE; j++) {
        const float4 b = sq[j];
        const float pv = fmul(Ia, b.w);  // (double)(I_a*I_b) < 1e-37f  <=>  pv < 1e-37f
        if (pv < 1e-37f) continue;
        float qx = fsub(k0, b.x), qy = fsub(k1, b.y), qz = fsub(k2, b.z);
        if (CHECK && fadd(fadd(fmul(qx, qx), fmul(qy, qy)), fmul(qz, qz)) > a.maxq2) continue;
        qx = fmul(qx, a.vpdq);
        qy = fmul(qy, a.vpdq);
        qz = fmul(qz, a.vpdq);
        const float qa = axis<KA>(qx, qy, qz, a.ka), qb = axis<KB>(qx, qy, qz, a.kb),
                    qc = axis<KC>(qx, qy, qz, a.kc);
        int f, m, s;
        if (INTERP == 0) {
            // (int)(round(q) + centre) of the reference, in integers
            f = round_half_away(qa) + a.cab;
            m = round_half_away(qb) + a.cab;
            s = round_half_away(qc) + a.cc;
        } else {
            f = __float2int_rd(qa) + a.cab;
            m = __float2int_rd(qb) + a.cab;
            s = __float2int_rd(qc) + a.cc;
        }
        if (!have || f != cur_f || m != cur_m || s != cur_s) {
            if (have) {
                if (INTERP == 0) {
                    put<INTERP>(a, w, win, cur_f, cur_m, cur_s, acc[0]);
                } else {
#pragma unroll
                    for (int c = 0; c < 8; c++)
                        put<INTERP>(a, w, win, cur_f + (c >> 2), cur_m + ((c >> 1) & 1), cur_s + (c & 1), acc[c]);
                }
            }
            have = true;
            cur_f = f;
            cur_m = m;
            cur_s = s;
#pragma unroll
            for (int c = 0; c < (INTERP ? 8 : 1); c++) acc[c] = 0;
        }
        if (INTERP == 0) {
            acc[0] += a.mult_int ? scaled_floor(pv, a.mult_int) : d2u64(dmul((double)pv, a.mult));
        } else {
            const double vm = dmul((double)pv, a.mult);
            // IAC/kernel.cl:139-179: Sep = 1 - (q - floor q) in float
            const double sf = (double)fsub(1.0f, fsub(qa, floorf(qa)));
            const double sm = (double)fsub(1.0f, fsub(qb, floorf(qb)));
            const double sz = (double)fsub(1.0f, fsub(qc, floorf(qc)));
            const double xf[2] = {sf, dsub(1.0, sf)}, yf[2] = {sm, dsub(1.0, sm)}, zf[2] = {sz, dsub(1.0, sz)};
#pragma unroll
            for (int c = 0; c < 8; c++)
                acc[c] += d2u64(dmul(vm, dmul(dmul(xf[c >> 2], yf[(c >> 1) & 1]), zf[c & 1])));
        }
    }
    if (have) {
        if (INTERP == 0) {
            put<INTERP>(a, w, win, cur_f, cur_m, cur_s, acc[0]);
        } else {
#pragma unroll
            for (int c = 0; c < 8; c++)
                put<INTERP>(a, w, win, cur_f + (c >> 2), cur_m + ((c >> 1) & 1), cur_s + (c & 1), acc[c]);
        }
    }
}

// scaled_floor for a normal p > 0 (every product that passes the 1e-37 test)
__device__ __forceinline__ unsigned long long scaled_floor_normal(float p, uint32_t M)
{
    const uint32_t b = __float_as_uint(p);
    const unsigned long long prod = (unsigned long long)((b & 0x7fffffu) | 0x800000u) * M;
    const int sh = (int)(b >> 23) - 150;  // p = mantissa * 2^sh
    return sh >= 0 ? (prod << min(sh, 63)) : (prod >> min(-sh, 63));
}

// nearest-voxel pairs with a compile-time axis mapping: the voxel is compared
// as one packed key f + 1024 m + 2^20 s (components within +-511, which
// key_ok guarantees for every pair inside MaxQ), the value path is chosen at
// compile time (MINT: integer Multiplicator)
template <int KA, int KB, int KC, bool CHECK, bool MINT>
__device__ __forceinline__ void cq_pairs_nn(const DenseArgs &a, const Window &w, uint32_t *win,
                                            const float4 *sq, int j0, float k0, float k1, float k2, float Ia)
{
    constexpr int NONE = -2147483647 - 1;
    int cur = NONE, cf = 0, cm = 0, cs = 0;
    unsigned long long acc = 0;
    const float vpdq = a.vpdq;
#pragma unroll 2
    for (int j = j0; j < DTILE; j++) {
        const float4 b = sq[j];
        const float pv = fmul(Ia, b.w);
        if (pv < 1e-37f) continue;
        float qx = fsub(k0, b.x), qy = fsub(k1, b.y), qz = fsub(k2, b.z);
        if (CHECK && fadd(fadd(fmul(qx, qx), fmul(qy, qy)), fmul(qz, qz)) > a.maxq2) continue;
        qx = fmul(qx, vpdq);
        qy = fmul(qy, vpdq);
        qz = fmul(qz, vpdq);
        const int f = round_half_away(axis<KA>(qx, qy, qz, 0));
        const int m = round_half_away(axis<KB>(qx, qy, qz, 0));
        const int s = round_half_away(axis<KC>(qx, qy, qz, 0));
        const int key = f + m * 1024 + s * 1048576;
        if (key != cur) {
            if (cur != NONE) put<0>(a, w, win, cf + a.cab, cm + a.cab, cs + a.cc, acc);
            cur = key;
            cf = f;
            cm = m;
            cs = s;
            acc = 0;
        }
        acc += MINT ? scaled_floor_normal(pv, a.mult_int) : d2u64(dmul((double)pv, a.mult));
    }
    if (cur != NONE) put<0>(a, w, win, cf + a.cab, cm + a.cab, cs + a.cc, acc);
}


// cq_pairs_nn when the window is on: every pair inside MaxQ lands in the
// window (it spans the two tiles' q range with a voxel of margin), so the run
// key is the voxel's window index itself and a finished run is one split 64-bit
// shared-memory add.  Pairs that fail the intensity or MaxQ test are masked
// rather than skipped, so a warp never diverges on them; the only branch is
// the guard for an index outside the window (non-finite k-vectors), which
// takes the global path of put().
template <int KA, int KB, int KC, bool CHECK, bool MINT>
__device__ __forceinline__ void cq_pairs_win(const DenseArgs &a, const Window &w, uint32_t *win,
                                             const float4 *sq, int j0, float k0, float k1, float k2, float Ia)
{
    const int D0 = w.dim[0], D01 = w.dim[0] * w.dim[1];
    const int words = D01 * w.dim[2];
    const int base = (a.cab - w.lo[0]) + D0 * (a.cab - w.lo[1]) + D01 * (a.cc - w.lo[2]);
    const float vpdq = a.vpdq;
    int cur = 0;
    bool on = false;  // a run is pending at window index cur
    unsigned long long acc = 0;
#pragma unroll 2
    for (int j = j0; j < DTILE; j++) {
        const float4 b = sq[j];
        const float pv = fmul(Ia, b.w);
        float qx = fsub(k0, b.x), qy = fsub(k1, b.y), qz = fsub(k2, b.z);
        bool ok = !(pv < 1e-37f);
        if (CHECK) ok = ok && !(fadd(fadd(fmul(qx, qx), fmul(qy, qy)), fmul(qz, qz)) > a.maxq2);
        qx = fmul(qx, vpdq);
        qy = fmul(qy, vpdq);
        qz = fmul(qz, vpdq);
        const int f = round_half_away(axis<KA>(qx, qy, qz, 0));
        const int m = round_half_away(axis<KB>(qx, qy, qz, 0));
        const int sz = round_half_away(axis<KC>(qx, qy, qz, 0));
        const int key = base + f + D0 * m + D01 * sz;
        const unsigned long long v = MINT ? scaled_floor_normal(pv, a.mult_int) : d2u64(dmul((double)pv, a.mult));
        const bool brk = ok && (!on || key != cur);  // a new run starts at this pair
        if (brk && on) shared_add_u64_split(win, win + WINDOW_WORDS<0>, (uint32_t)cur, acc);
        const bool inwin = (unsigned)key < (unsigned)words;
        if (brk && !inwin) global_put_pair(a, f + a.cab, m + a.cab, sz + a.cc, v);
        acc = brk ? (inwin ? v : 0ull) : (ok ? acc + v : acc);
        cur = brk ? key : cur;
        on = brk ? inwin : on;
    }
    if (on) shared_add_u64_split(win, win + WINDOW_WORDS<0>, (uint32_t)cur, acc);
}

// ---- two consecutive staged pixels per step, FP32 work as f32x2 pairs ----
// round half away from zero of both lanes, as ints (see round_half_away)
__device__ __forceinline__ int2 f2round_half_away(float2 x)
{
    const float2 t = f2add(x, make_float2(copysignf(0.49999997f, x.x), copysignf(0.49999997f, x.y)));
    return make_int2(__float2int_rz(t.x), __float2int_rz(t.y));
}

// floor(p * M) for 0 <= p < 2^23 and an integer M < 2^29: p's 24-bit
// significand times M is below 2^53, so the double product is exact and its
// truncation is the floor.  One multiply on the (otherwise idle) FP64 pipe and
// two conversions take fewer issue slots than the integer form (significand
// product shifted by the exponent), which measured 1.025 s against 0.864 s at
// 1024^2 with the run flush below.
__device__ __forceinline__ unsigned long long scaled_floor_small(float p, uint32_t M)
{
    return __double2ull_rz(__dmul_rn((double)p, (double)M));
}

// one pair of the packed window path: a pair that fails the intensity or
// MaxQ test adds 0 at the pending voxel (it neither starts nor ends a run)
__device__ __forceinline__ void win_step(const DenseArgs &a, uint32_t *win, int words, bool ok, int key, float pv,
                                         int f, int m, int sz, int &cur, unsigned long long &acc)
{
    if (ok && (unsigned)key >= (unsigned)words) {  // non-finite k-vectors only
        global_put_pair(a, f + a.cab, m + a.cab, sz + a.cc, scaled_floor_small(pv, a.mult_int));
        ok = false;
    }
    const int k = ok ? key : cur;
    const unsigned long long v = scaled_floor_small(ok ? pv : 0.0f, a.mult_int);
    const bool brk = k != cur;
    if (brk) shared_add_u64_split(win, win + WINDOW_WORDS<0>, (uint32_t)cur, acc);  // acc may be 0: adds nothing
    acc = (brk ? 0ull : acc) + v;
    cur = k;
}

// cq_pairs_win for an integer Multiplicator and tile pairs whose products stay
// below 2^23: the staged tile holds consecutive pixels j, j+1 as
// (x_j, x_j+1, y_j, y_j+1), (z_j, z_j+1, I_j, I_j+1), and each step evaluates
// both pairs with f32x2 arithmetic (the same roundings as the scalar path),
// then bins them in order.  j0 may be odd (diagonal tiles): the first step
// then masks its lower lane.
template <int KA, int KB, int KC, bool CHECK>
__device__ __forceinline__ void cq_pairs_win2(const DenseArgs &a, const Window &w, uint32_t *win,
                                              const float4 *sp, int j0, float k0, float k1, float k2, float Ia)
{
    const int D0 = w.dim[0], D01 = w.dim[0] * w.dim[1];
    const int words = D01 * w.dim[2];
    const int base = (a.cab - w.lo[0]) + D0 * (a.cab - w.lo[1]) + D01 * (a.cc - w.lo[2]);
    const float2 vp2 = make_float2(a.vpdq, a.vpdq), K0 = make_float2(k0, k0), K1 = make_float2(k1, k1),
                 K2 = make_float2(k2, k2), IA = make_float2(Ia, Ia), nz = make_float2(a.neg_zero, a.neg_zero);
    int cur = 0;  // pending run: window index cur, value acc (0 before the first pair)
    unsigned long long acc = 0;
    auto step = [&](int jp, bool lo_on) {
        const float4 A = sp[2 * jp], B = sp[2 * jp + 1];
        const float2 pv = f2mul(IA, make_float2(B.z, B.w));
        float2 qx = f2sub(K0, make_float2(A.x, A.y)), qy = f2sub(K1, make_float2(A.z, A.w)),
               qz = f2sub(K2, make_float2(B.x, B.y));
        bool ok0 = lo_on && !(pv.x < 1e-37f), ok1 = !(pv.y < 1e-37f);
        if (CHECK) {  // scalar: ptxas may fuse a packed multiply and add into one FFMA2
            ok0 = ok0 && !(fadd(fadd(fmul(qx.x, qx.x), fmul(qy.x, qy.x)), fmul(qz.x, qz.x)) > a.maxq2);
            ok1 = ok1 && !(fadd(fadd(fmul(qx.y, qx.y), fmul(qy.y, qy.y)), fmul(qz.y, qz.y)) > a.maxq2);
        }
        qx = f2fma(qx, vp2, nz);  // an add follows
        qy = f2fma(qy, vp2, nz);
        qz = f2fma(qz, vp2, nz);
        const int2 f = f2round_half_away(KA == 0 ? qx : KA == 1 ? qy : qz);
        const int2 m = f2round_half_away(KB == 0 ? qx : KB == 1 ? qy : qz);
        const int2 sz = f2round_half_away(KC == 0 ? qx : KC == 1 ? qy : qz);
        win_step(a, win, words, ok0, base + f.x + D0 * m.x + D01 * sz.x, pv.x, f.x, m.x, sz.x, cur, acc);
        win_step(a, win, words, ok1, base + f.y + D0 * m.y + D01 * sz.y, pv.y, f.y, m.y, sz.y, cur, acc);
    };
    int jp = j0 >> 1;
    if (j0 & 1) step(jp++, false);
#pragma unroll 2
    for (; jp < DTILE / 2; jp++) step(jp, true);
    if (acc) shared_add_u64_split(win, win + WINDOW_WORDS<0>, (uint32_t)cur, acc);
}

// ---------------------------------------------------------------------------
// Tiles whose products times the Multiplicator stay below SMALL_VALUE (2^23), which
// the usual maps do (the Multiplicator puts the mean product between 1e5 and 1e6):
// the values need no 64-bit arithmetic.  A negative product counts as 0.  For an integer Multiplicator M below 2^24, p M + 2^23 rounded
// toward zero is 2^23 + floor(p M), one f32x2 fma for two pairs.  A run of 256
// pairs sums to less than 2^31 and goes to the window in two halves, its low 16
// bits into one word and the rest into another: a tile pair adds at most 65 536
// runs, so neither word overflows and no add has to return anything.  Pixels of
// intensity 0 (masked, or absent from a ragged tile) are not staged; an odd rest is
// filled up at a corner of the tile's box, so that every pair lands in the window.
// 1024 x 512 map with 5 % masked, 199-edge mesh, nearest: 214.9 -> 141.8 ms (147.4 with
// the masked pixels staged); linear at 244 x 250, 127-edge mesh: 17.6 -> 7.5 ms (8.4).
// Larger products keep the 64-bit paths above.
// ---------------------------------------------------------------------------
constexpr float SMALL_VALUE = 8388608.0f;

__device__ __forceinline__ bool small_values(const DenseArgs &a, const float4 p0, const float4 q0)
{
    // a Multiplicator past 1e30 could lift products that the 1e-37 cut drops to whole numbers
    return a.mult > 0.0 && a.mult < 1e30 && __fmul_ru(__fmul_ru(p0.w, q0.w), __double2float_ru(a.mult)) < SMALL_VALUE;
}
// a product of the two tiles may be negative: it adds nothing
__device__ __forceinline__ bool negative(const float4 p1, const float4 q1) { return p1.w < 0.0f || q1.w < 0.0f; }

// staged pixel j of the paths that take two at a time: (x, x', y, y'), (z, z', I, I')
__device__ __forceinline__ void put_interleaved(float4 *sq, int j, const float4 v)
{
    float *s = reinterpret_cast<float *>(sq) + (j >> 1) * 8 + (j & 1);
    s[0] = v.x;
    s[2] = v.y;
    s[4] = v.z;
    s[6] = v.w;
}

// The tile's pixels of nonzero intensity, staged in their order: their number, and in
// `rank` the place of this thread's (pixel threadIdx.x).
// A map of mostly masked pixels then costs what its others do (95 % of 200 x 220
// masked: nearest 902 -> 151 us, linear 2859 -> 312; AC1D 969 -> 99 and 1340 -> 117).
// `staged` has a word per warp.
__device__ __forceinline__ int rank_staged(bool on, uint32_t *staged, int &rank)
{
    const uint32_t ball = __ballot_sync(0xffffffffu, on);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) staged[w] = ball;
    __syncthreads();
    int n = 0;
    rank = 0;
#pragma unroll
    for (int k = 0; k < DTILE / 32; k++) {
        if (k == w) rank = n + __popc(ball & ((1u << lane) - 1));
        n += __popc(staged[k]);
    }
    return n;
}
// the staged pixels up to and with pixel `own` of the tile
__device__ __forceinline__ int staged_through(const uint32_t *staged, int own)
{
    int n = __popc(staged[own >> 5] & (0xffffffffu >> (31 - (own & 31))));
    for (int k = 0; k < own >> 5; k++) n += __popc(staged[k]);
    return n;
}

// add `acc` (< 2^31) in two halves at window word `at` if `on`
__device__ __forceinline__ void window_add_halves(uint32_t win, int at, uint32_t acc, bool on)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %0, 0;\n\t@p red.shared.add.u32 [%1], %2;\n\t"
        "@p red.shared.add.u32 [%1+%4], %3;\n\t}" ::"r"((int)on),
        "r"(win + 4u * (uint32_t)at), "r"(acc & 0xffffu), "r"(acc >> 16), "n"(4 * WINDOW_WORDS<0>)
        : "memory");
}

// nearest voxel, two staged pixels per step; win: shared-memory address of the window
template <int KA, int KB, int KC, bool CHECK, bool SIGNED>
__device__ __forceinline__ void cq_pairs_small(const DenseArgs &a, const Window &w, uint32_t win, const float4 *sp, int j0,
                                               int n, float k0, float k1, float k2, float Ia)
{
    const int D0 = w.dim[0], D01 = w.dim[0] * w.dim[1];
    const int base = (a.cab - w.lo[0]) + D0 * (a.cab - w.lo[1]) + D01 * (a.cc - w.lo[2]);
    auto dup = [](float x) { return make_float2(x, x); };
    int cur = 0;  // pending run: window word, sum (0 before the first pair)
    uint32_t acc = 0;
    auto put = [&](int key, uint32_t v) {
        const bool brk = key != cur;
        window_add_halves(win, cur, acc, brk);
        acc = (brk ? 0u : acc) + v;
        cur = key;
    };
    auto step = [&](int jp, bool lo_on) {
        const float4 A = sp[2 * jp], B = sp[2 * jp + 1];
        float2 pv = f2mul(dup(Ia), make_float2(B.z, B.w));
        if (SIGNED) pv = make_float2(fmaxf(pv.x, 0.0f), fmaxf(pv.y, 0.0f));
        float2 qx = f2sub(dup(k0), make_float2(A.x, A.y)), qy = f2sub(dup(k1), make_float2(A.z, A.w)),
               qz = f2sub(dup(k2), make_float2(B.x, B.y));
        const float2 vb = f2fma_rz(pv, dup(a.mult_f), dup(8388608.0f));
        uint32_t v0 = __float_as_uint(vb.x) - 0x4B000000u, v1 = __float_as_uint(vb.y) - 0x4B000000u;
        bool ok0 = lo_on, ok1 = true;
        if (CHECK) {
            const float2 nz = dup(a.neg_zero);
            const float2 s = f2add(f2add(f2fma(qx, qx, nz), f2fma(qy, qy, nz)), f2fma(qz, qz, nz));
            ok0 = ok0 && !(s.x > a.maxq2);  // a MaxQ that is no number bounds nothing
            ok1 = !(s.y > a.maxq2);
        }
        const float2 vp = dup(a.vpdq), zero = dup(a.neg_zero);  // products that an add follows
        qx = f2fma(qx, vp, zero);
        qy = f2fma(qy, vp, zero);
        qz = f2fma(qz, vp, zero);
        const int2 f = f2round_half_away(KA == 0 ? qx : KA == 1 ? qy : qz);
        const int2 m = f2round_half_away(KB == 0 ? qx : KB == 1 ? qy : qz);
        const int2 sz = f2round_half_away(KC == 0 ? qx : KC == 1 ? qy : qz);
        // a pair that is off adds 0 to the pending run
        const int key0 = base + f.x + D0 * m.x + D01 * sz.x, key1 = base + f.y + D0 * m.y + D01 * sz.y;
        if (CHECK || !lo_on)
            put(ok0 ? key0 : cur, ok0 ? v0 : 0u);
        else
            put(key0, v0);
        if (CHECK)
            put(ok1 ? key1 : cur, ok1 ? v1 : 0u);
        else
            put(key1, v1);
    };
    int jp = j0 >> 1;
    if (j0 & 1) step(jp++, false);
#pragma unroll 2
    for (; 2 * jp < n; jp++) step(jp, true);
    window_add_halves(win, cur, acc, true);
}

// 8-corner linear, for the same tiles and any Multiplicator: the floor of a
// corner's double product is the low word of that product plus 2^52 rounded toward
// zero, and the eight sums of a run are 32-bit words, which go to the window's
// split counters with their carries.
template <int KA, int KB, int KC, bool CHECK>
__device__ __forceinline__ void cq_pairs_small_linear(const DenseArgs &a, const Window &w, uint32_t win, const float4 *sq,
                                                      int j0, int n, float k0, float k1, float k2, float Ia)
{
    const int D0 = w.dim[0], D01 = w.dim[0] * w.dim[1];
    const int base = (a.cab - w.lo[0]) + D0 * (a.cab - w.lo[1]) + D01 * (a.cc - w.lo[2]);
    int cur = 0;
    uint32_t acc[8];  // [4 fs + 2 ms + ss]
#pragma unroll
    for (int c = 0; c < 8; c++) acc[c] = 0;
    auto at = [&](int c) { return win + 4u * (uint32_t)(cur + (c >> 2) + ((c >> 1) & 1) * D0 + (c & 1) * D01); };
    auto flush = [&]() {
        uint32_t old[8];
#pragma unroll
        for (int c = 0; c < 8; c++)
            asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old[c]) : "r"(at(c)), "r"(acc[c]) : "memory");
#pragma unroll
        for (int c = 0; c < 8; c++) {
            if (old[c] + acc[c] < old[c])  // rare: the carry out of the low word
                asm volatile("red.shared.add.u32 [%0+%1], 1;" ::"r"(at(c)), "n"(4 * WINDOW_WORDS<1>) : "memory");
            acc[c] = 0;
        }
    };
    // floor of |x| < 2^22 as an integer; frac: x - floor x, as the reference forms it
    auto floor_frac = [](float x, float &frac) {
        const float t = __fadd_rd(x, ROUND_MAGIC);
        frac = fsub(x, fsub(t, ROUND_MAGIC));
        return __float_as_int(t) - 0x4B400000;
    };
#pragma unroll 1
    for (int j = j0; j < n; j++) {
        const float4 b = sq[j];
        float pv = fmul(Ia, b.w);
        float qx = fsub(k0, b.x), qy = fsub(k1, b.y), qz = fsub(k2, b.z);
        const bool ok = !CHECK || !(fadd(fadd(fmul(qx, qx), fmul(qy, qy)), fmul(qz, qz)) > a.maxq2);
        qx = fmul(qx, a.vpdq);
        qy = fmul(qy, a.vpdq);
        qz = fmul(qz, a.vpdq);
        float ff, fm, fz;
        const int f = floor_frac(axis<KA>(qx, qy, qz, 0), ff), m = floor_frac(axis<KB>(qx, qy, qz, 0), fm),
                  s = floor_frac(axis<KC>(qx, qy, qz, 0), fz);
        const int key = ok ? base + f + D0 * m + D01 * s : cur;
        if (key != cur) {
            flush();
            cur = key;
        }
        const double vm = dmul((double)(ok ? fmaxf(pv, 0.0f) : 0.0f), a.mult);
        // IAC/kernel.cl:139-179: Sep = 1 - (q - floor q) in float
        const double sf = (double)fsub(1.0f, ff), sm = (double)fsub(1.0f, fm), sz = (double)fsub(1.0f, fz);
        const double xf[2] = {sf, dsub(1.0, sf)}, yf[2] = {sm, dsub(1.0, sm)}, zf[2] = {sz, dsub(1.0, sz)};
#pragma unroll
        for (int c = 0; c < 8; c += 2) {
            const double xy = dmul(xf[c >> 2], yf[(c >> 1) & 1]);
#pragma unroll
            for (int z = 0; z < 2; z++)
                acc[c + z] += (uint32_t)__double2loint(__dadd_rz(dmul(vm, dmul(xy, zf[z])), 4503599627370496.0));
        }
    }
    flush();
}

// upper bound of |k_a - k_b| over two boxes is below MaxQ with a margin that
// covers the FP32 rounding of the per-pair test (every pair passes it)
__device__ __forceinline__ bool boxes_within(const float4 a0, const float4 a1, const float4 b0, const float4 b1,
                                             float maxq)
{
    const float dx = fmaxf(a1.x - b0.x, b1.x - a0.x);
    const float dy = fmaxf(a1.y - b0.y, b1.y - a0.y);
    const float dz = fmaxf(a1.z - b0.z, b1.z - a0.z);
    return dx * dx + dy * dy + dz * dz < maxq * maxq * 0.9999f;
}

// index within the 16 x 16 patch of thread t's own pixel: lane l of warp w takes
// x = 4 (l % 4) + w % 4, y = 2 (l / 4) + w / 4 (a bijection of 0..255)
__device__ __forceinline__ int own_pixel(int t)
{
    const int w = t >> 5, l = t & 31;
    return (2 * (l >> 2) + (w >> 2)) * 16 + 4 * (l & 3) + (w & 3);
}

template <int INTERP, int KA, int KB, int KC>
__global__ void __launch_bounds__(DTILE, INTERP ? 4 : 6) cq_small_kernel(const DenseArgs a)
{
    __shared__ float4 sq[DTILE];
    __shared__ uint32_t win[2 * WINDOW_WORDS<INTERP>];  // split 64-bit counters: low words, then high words
    __shared__ unsigned long long s_pair;
    __shared__ unsigned long long s_self[DTILE / 32];
    __shared__ uint32_t s_staged[DTILE / 32];
    const uint32_t T = a.ntiles;
    for (;;) {
        if (threadIdx.x == 0) s_pair = atomicAdd(a.queue, 1ull);
        __syncthreads();
        const unsigned long long p = s_pair * a.nparts + a.part;
        if (p >= a.npairs) break;
        uint32_t P, Q;
        decode_tile_pair(p, T, P, Q);
        const float4 p0 = a.box[2 * P], p1 = a.box[2 * P + 1], q0 = a.box[2 * Q], q1 = a.box[2 * Q + 1];
        if (boxes_beyond(p0, p1, q0, q1, a.maxq)) {
            __syncthreads();
            continue;
        }
        const bool check = !boxes_within(p0, p1, q0, q1, a.maxq);
        // window over the q range of the pair (P - Q), one voxel of margin
        Window w;
        {
            const float lo3[3] = {p0.x - q1.x, p0.y - q1.y, p0.z - q1.z};
            const float hi3[3] = {p1.x - q0.x, p1.y - q0.y, p1.z - q0.z};
            const int ax[3] = {a.ka, a.kb, a.kc};
            const int cen[3] = {a.cab, a.cab, a.cc};
            int words = 1;
            bool ok = true;
            for (int d = 0; d < 3; d++) {
                const float l = (ax[d] == 0 ? lo3[0] : ax[d] == 1 ? lo3[1] : lo3[2]) * a.vpdq;
                const float h = (ax[d] == 0 ? hi3[0] : ax[d] == 1 ? hi3[1] : hi3[2]) * a.vpdq;
                // coordinates below 2^22, where their roundings are exact and nothing here
                // overflows; false for a range that is not finite
                ok = ok && l > -4194304.0f && h < 4194304.0f && h - l <= (float)WINDOW_WORDS<INTERP>;
                w.lo[d] = ok ? (int)floorf(l) - 1 + cen[d] : 0;
                w.dim[d] = ok ? (int)ceilf(h) + 2 + cen[d] - w.lo[d] + (INTERP ? 1 : 0) : 0;
                ok = ok && w.dim[d] >= 1 && w.dim[d] <= WINDOW_WORDS<INTERP>;
                if (ok) words *= w.dim[d];  // at most WINDOW_WORDS^2 here
                ok = ok && words <= WINDOW_WORDS<INTERP>;
            }
            w.on = ok;
            if (w.on)
                for (int i = threadIdx.x; i < words; i += DTILE) win[i] = win[WINDOW_WORDS<INTERP> + i] = 0u;
        }
        const bool small = KA >= 0 && w.on && (INTERP || a.mult_f != 0.0f) && small_values(a, p0, q0);
        // integer Multiplicator and every product of the two tiles below 2^23
        // (the tiles' largest |I|): the packed window path
        const bool packed =
            INTERP == 0 && (small || (KA >= 0 && w.on && a.mult_int != 0u && fmul(p0.w, q0.w) < 8388608.0f));
        // stage tile Q: (k, I) per pixel, or interleaved per pixel pair for the packed path
        int staged = DTILE;
        {
            const uint64_t j = tile_pixel(a, Q, threadIdx.x);
            float4 v = j < a.npix ? make_float4(a.K[3 * j], a.K[3 * j + 1], a.K[3 * j + 2], a.I[j])
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
            int at = threadIdx.x;
            if (small) {
                staged = rank_staged(v.w != 0.0f, s_staged, at);
                if (!INTERP && (staged & 1) && threadIdx.x == 0) put_interleaved(sq, staged, make_float4(q0.x, q0.y, q0.z, 0.f));
            }
            if (small && v.w == 0.0f) {
            } else if (packed) {
                put_interleaved(sq, at, v);
            } else {
                sq[at] = v;
            }
        }
        __syncthreads();
        // own pixel: spread over the patch (x 4 apart, y 2 apart within a warp) so
        // that a warp's lanes rarely share a voxel and their window adds for one
        // staged pixel rarely meet at one address; the staged tile keeps its
        // order (runs of consecutive pixels land in one voxel)
        const int own = own_pixel(threadIdx.x);
        const uint64_t ia = tile_pixel(a, P, own);
        unsigned long long self = 0;
        if (ia < a.npix) {
            const float k0 = a.K[3 * ia], k1 = a.K[3 * ia + 1], k2 = a.K[3 * ia + 2];
            const float Ia = a.I[ia];
            if (P == Q) {
                const float sv = fmul(Ia, Ia);
                if (!(sv < 1e-37f))
                    self = a.mult_int ? scaled_floor(sv, a.mult_int) : d2u64(dmul((double)sv, a.mult));
            }
            const int j0 = P != Q ? 0 : small ? staged_through(s_staged, own) : own + 1;
            if (small) {
                const uint32_t wa = (uint32_t)__cvta_generic_to_shared(win);
                if (Ia == 0.0f) {
                } else if (INTERP && check)
                    cq_pairs_small_linear<KA, KB, KC, true>(a, w, wa, sq, j0, staged, k0, k1, k2, Ia);
                else if (INTERP)
                    cq_pairs_small_linear<KA, KB, KC, false>(a, w, wa, sq, j0, staged, k0, k1, k2, Ia);
                else if (negative(p1, q1))
                    cq_pairs_small<KA, KB, KC, true, true>(a, w, wa, sq, j0, staged, k0, k1, k2, Ia);
                else if (check)
                    cq_pairs_small<KA, KB, KC, true, false>(a, w, wa, sq, j0, staged, k0, k1, k2, Ia);
                else
                    cq_pairs_small<KA, KB, KC, false, false>(a, w, wa, sq, j0, staged, k0, k1, k2, Ia);
            } else if (packed) {
                if (check)
                    cq_pairs_win2<KA, KB, KC, true>(a, w, win, sq, j0, k0, k1, k2, Ia);
                else
                    cq_pairs_win2<KA, KB, KC, false>(a, w, win, sq, j0, k0, k1, k2, Ia);
            } else if (INTERP == 0 && KA >= 0 && w.on) {
                if (a.mult_int) {
                    if (check)
                        cq_pairs_win<KA, KB, KC, true, true>(a, w, win, sq, j0, k0, k1, k2, Ia);
                    else
                        cq_pairs_win<KA, KB, KC, false, true>(a, w, win, sq, j0, k0, k1, k2, Ia);
                } else {
                    if (check)
                        cq_pairs_win<KA, KB, KC, true, false>(a, w, win, sq, j0, k0, k1, k2, Ia);
                    else
                        cq_pairs_win<KA, KB, KC, false, false>(a, w, win, sq, j0, k0, k1, k2, Ia);
                }
            } else if (INTERP == 0 && KA >= 0 && a.key_ok) {
                if (a.mult_int) {
                    if (check)
                        cq_pairs_nn<KA, KB, KC, true, true>(a, w, win, sq, j0, k0, k1, k2, Ia);
                    else
                        cq_pairs_nn<KA, KB, KC, false, true>(a, w, win, sq, j0, k0, k1, k2, Ia);
                } else {
                    if (check)
                        cq_pairs_nn<KA, KB, KC, true, false>(a, w, win, sq, j0, k0, k1, k2, Ia);
                    else
                        cq_pairs_nn<KA, KB, KC, false, false>(a, w, win, sq, j0, k0, k1, k2, Ia);
                }
            } else if (check) {
                cq_pairs<INTERP, KA, KB, KC, true>(a, w, win, sq, j0, k0, k1, k2, Ia);
            } else {
                cq_pairs<INTERP, KA, KB, KC, false>(a, w, win, sq, j0, k0, k1, k2, Ia);
            }
        }
        // self pairs of a diagonal tile: once, at the centre
        for (int o = 16; o; o >>= 1) self += __shfl_xor_sync(0xffffffffu, self, o);
        if ((threadIdx.x & 31) == 0) s_self[threadIdx.x >> 5] = self;
        __syncthreads();
        if (threadIdx.x == 0 && P == Q) {
            unsigned long long t = 0;
            for (int i = 0; i < DTILE / 32; i++) t += s_self[i];
            if (t) atomicAdd(&a.out[(uint64_t)a.cab + (uint64_t)a.cab * a.ab + (uint64_t)a.cc * a.ab * a.ab], t);
        }
        if (w.on) {
            const int words = w.dim[0] * w.dim[1] * w.dim[2];
            for (int i = threadIdx.x; i < words; i += DTILE) {
                const unsigned long long v =
                    small && !INTERP ? win[i] + ((unsigned long long)win[WINDOW_WORDS<INTERP> + i] << 16)
                                     : split_word(win, win + WINDOW_WORDS<INTERP>, i);
                if (!v) continue;
                const int x = i % w.dim[0], y = (i / w.dim[0]) % w.dim[1], z = i / (w.dim[0] * w.dim[1]);
                global_put_pair(a, x + w.lo[0], y + w.lo[1], z + w.lo[2], v);
            }
        }
        __syncthreads();
    }
}

// --------------------------------------------------------------------------
// AC1D C(q): |q| histogram in shared memory for the whole launch
// --------------------------------------------------------------------------
// b % n without the division when b < n (bins past the histogram are rare)
__device__ __forceinline__ uint32_t wrap_bin(uint32_t b, uint32_t n)
{
    if (b >= n) b %= n;
    return b;
}

// Pairs (own pixel, staged pixels j0 ..) of finite tiles whose bins all lie in the
// histogram: two staged pixels per step, |q| / dq by the two-word reciprocal, the
// bin's address from the bits of |q| / dq + 2^23.  SMALL: tiles with small values (see
// cq_pairs_small) and no negative ones, below 2^24 into the split counters; else any,
// 64 bits each (200 x 220, intensities past the limit, nearest 2.23 -> 1.68 ms, linear
// 2.83 -> 2.17; some negative 2.45 -> 1.94 and 2.70 -> 1.96).  CHECK: as cq_pairs.
// 512^2 map with 5 % masked, linear, 88.4 -> 51.8 ms (issue 88 %, conversion unit 42 %);
// nearest 78.1 -> 35.8 ms.
template <int INTERP, bool CHECK, bool SMALL>
__device__ __forceinline__ void ac1d_pairs(const DenseArgs &a, uint32_t hist, const float4 *sp, int j0, int n,
                                           float k0, float k1, float k2, float Ia)
{
    auto dup = [](float x) { return make_float2(x, x); };
    const float2 nz = dup(a.neg_zero);
    const uint32_t bin0 = hist - 4u * (uint32_t)TWO23_BITS;  // address of bin 0, minus the bits of 2^23
    auto add = [&](uint32_t at, uint32_t v) {
        uint32_t old;
        asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(at), "r"(v) : "memory");
        return old + v < old;
    };
    auto carry = [&](uint32_t at) {
        asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(at + 4u * a.hsize) : "memory");
    };
    auto add64 = [&](uint32_t at, unsigned long long v) {
        const uint32_t up = (uint32_t)(v >> 32) + (add(at, (uint32_t)v) ? 1u : 0u);
        if (up) asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(at + 4u * a.hsize), "r"(up) : "memory");
    };
    auto step = [&](int jp, bool lo_on) {
        const float4 A = sp[2 * jp], B = sp[2 * jp + 1];
        const float2 pv = f2mul(dup(Ia), make_float2(B.z, B.w));
        const float2 dx = f2sub(dup(k0), make_float2(A.x, A.y)), dy = f2sub(dup(k1), make_float2(A.z, A.w)),
                     dz = f2sub(dup(k2), make_float2(B.x, B.y));
        const float2 s = f2add(f2add(f2fma(dx, dx, nz), f2fma(dy, dy, nz)), f2fma(dz, dz, nz));
        const float2 q = f2div(make_float2(__fsqrt_rn(s.x), __fsqrt_rn(s.y)), a.by_dq);
        const bool ok[2] = {lo_on && (!CHECK || s.x <= a.maxq2), !CHECK || s.y <= a.maxq2};
        const float qs[2] = {q.x, q.y}, ps[2] = {pv.x, pv.y};
        if (!SMALL) {
#pragma unroll
            for (int e = 0; e < 2; e++) {
                if (!ok[e] || ps[e] < 1e-37f) continue;
                if (INTERP == 0) {
                    const uint32_t b = __float_as_uint(__fadd_rz(fadd(qs[e], 0.49999997f), 8388608.0f));
                    add64(bin0 + 4u * b, 2ull * (a.mult_int ? scaled_floor(ps[e], a.mult_int)
                                                            : (unsigned long long)(long long)dmul((double)ps[e], a.mult)));
                } else {
                    const float t = __fadd_rz(qs[e], 8388608.0f);
                    const double val = (double)ps[e], sep = (double)fsub(qs[e], fsub(t, 8388608.0f));
                    const uint32_t at = bin0 + 4u * __float_as_uint(t);
                    add64(at, 2ull * (unsigned long long)(long long)dmul(dmul(val, dsub(1.0, sep)), a.mult));
                    add64(at + 4u, 2ull * (unsigned long long)(long long)dmul(dmul(val, sep), a.mult));
                }
            }
        } else if (INTERP == 0) {
            // floor(fl(q + 0.49999997f)), see ac1d_cq_kernel
            uint32_t at[2], v[2];
            bool c[2];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const uint32_t b = __float_as_uint(__fadd_rz(fadd(qs[e], 0.49999997f), 8388608.0f));
                v[e] = 2u * (__float_as_uint(__fmaf_rz(ps[e], a.mult_f, 8388608.0f)) - (uint32_t)TWO23_BITS);
                at[e] = bin0 + 4u * b;
                if (CHECK || !lo_on) {
                    v[e] = ok[e] ? v[e] : 0u;
                    at[e] = ok[e] ? at[e] : hist;
                }
            }
#pragma unroll
            for (int e = 0; e < 2; e++) c[e] = add(at[e], v[e]);
            if (c[0]) carry(at[0]);
            if (c[1]) carry(at[1]);
        } else {
            uint32_t at[2], v1[2], v2[2];
            bool c[4];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const float t = __fadd_rz(qs[e], 8388608.0f);
                const double val = (double)ps[e], sep = (double)fsub(qs[e], fsub(t, 8388608.0f));
                v1[e] = 2u * (uint32_t)__double2loint(
                                 __dadd_rz(dmul(dmul(val, dsub(1.0, sep)), a.mult), 4503599627370496.0));
                v2[e] = 2u * (uint32_t)__double2loint(__dadd_rz(dmul(dmul(val, sep), a.mult), 4503599627370496.0));
                at[e] = bin0 + 4u * __float_as_uint(t);
                if (CHECK || !lo_on) {
                    v1[e] = ok[e] ? v1[e] : 0u;
                    v2[e] = ok[e] ? v2[e] : 0u;
                    at[e] = ok[e] ? at[e] : hist;
                }
            }
#pragma unroll
            for (int e = 0; e < 2; e++) {
                c[2 * e] = add(at[e], v1[e]);
                c[2 * e + 1] = add(at[e] + 4u, v2[e]);
            }
            if (c[0] | c[1] | c[2] | c[3]) {
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (c[e]) carry(at[e >> 1] + 4u * (e & 1));
            }
        }
    };
    int jp = j0 >> 1;
    if (j0 & 1) step(jp++, false);
#pragma unroll 2
    for (; 2 * jp < n; jp++) step(jp, true);
}

// Six CTAs an SM: 40 registers; without the bound nearest is 3 % slower, and with eight
// CTAs (32 registers) 5 %.
template <int INTERP>
__global__ void __launch_bounds__(DTILE, 6) ac1d_cq_kernel(const DenseArgs a)
{
    // the launch's histogram as split 64-bit counters: low words, then high words
    extern __shared__ uint32_t hist32[];
    uint32_t *const hlo = hist32, *const hhi = hist32 + a.hsize;
    __shared__ float4 sq[DTILE];
    __shared__ unsigned long long s_pair;
    __shared__ uint32_t s_staged[DTILE / 32];
    for (uint32_t i = threadIdx.x; i < 2 * a.hsize; i += DTILE) hist32[i] = 0;
    const uint32_t T = a.ntiles;
    for (;;) {
        if (threadIdx.x == 0) s_pair = atomicAdd(a.queue, 1ull);
        __syncthreads();
        const unsigned long long p = s_pair * a.nparts + a.part;
        if (p >= a.npairs) break;
        uint32_t P, Q;
        decode_tile_pair(p, T, P, Q);
        const float4 p0 = a.box[2 * P], p1 = a.box[2 * P + 1], q0 = a.box[2 * Q], q1 = a.box[2 * Q + 1];
        if (boxes_beyond(p0, p1, q0, q1, a.maxq)) {
            __syncthreads();
            continue;
        }
        // no bin past the histogram, everything finite
        const bool ranged = a.in_range && p0.w < INFINITY && q0.w < INFINITY;
        const bool small = ranged && (INTERP || a.mult_f != 0.0f) && !negative(p1, q1) && small_values(a, p0, q0);
        const bool check = !boxes_within(p0, p1, q0, q1, a.maxq);
        int staged = DTILE;
        {
            const uint64_t j = tile_pixel(a, Q, threadIdx.x);
            float4 v = j < a.npix ? make_float4(a.K[3 * j], a.K[3 * j + 1], a.K[3 * j + 2], a.I[j])
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
            if (ranged) {
                int at;
                staged = rank_staged(v.w != 0.0f, s_staged, at);
                if ((staged & 1) && threadIdx.x == 0)  // adds 0 within the tile's reach
                    put_interleaved(sq, staged, make_float4(q0.x, q0.y, q0.z, 0.f));
                if (v.w != 0.0f) put_interleaved(sq, at, v);
            } else {
                sq[threadIdx.x] = v;
            }
        }
        __syncthreads();
        // own pixel 8 apart from the neighbouring lanes' (a bijection of the tile):
        // the lanes of a warp then add into different bins for one staged pixel
        const int own = (int)((threadIdx.x & 31) * 8 + (threadIdx.x >> 5));
        const uint64_t ia = tile_pixel(a, P, own);
        if (ia < a.npix) {
            const float k0 = a.K[3 * ia], k1 = a.K[3 * ia + 1], k2 = a.K[3 * ia + 2];
            const float Ia = a.I[ia];
            if (P == Q) {  // self pair: q = 0 -> bin 0, once
                const float sv = fmul(Ia, Ia);
                if (!(sv < 1e-37f))
                    shared_add_u64_split(hlo, hhi, 0,
                                         a.mult_int ? scaled_floor(sv, a.mult_int)
                                                    : (unsigned long long)(long long)dmul((double)sv, a.mult));
            }
            const int j0 = P != Q ? 0 : ranged ? staged_through(s_staged, own) : own + 1;
            if (ranged && Ia != 0.0f) {
                const uint32_t ha = (uint32_t)__cvta_generic_to_shared(hist32);
                if (small && check)
                    ac1d_pairs<INTERP, true, true>(a, ha, sq, j0, staged, k0, k1, k2, Ia);
                else if (small)
                    ac1d_pairs<INTERP, false, true>(a, ha, sq, j0, staged, k0, k1, k2, Ia);
                else
                    ac1d_pairs<INTERP, true, false>(a, ha, sq, j0, staged, k0, k1, k2, Ia);
            }
            for (int j = ranged ? DTILE : j0; j < DTILE; j++) {
                const float4 b = sq[j];
                const float pv = fmul(Ia, b.w);
                if (pv < 1e-37f) continue;
                const double val = (double)pv;
                const float dx = fsub(k0, b.x), dy = fsub(k1, b.y), dz = fsub(k2, b.z);
                float q = __fsqrt_rn(fadd(fadd(fmul(dx, dx), fmul(dy, dy)), fmul(dz, dz)));
                if (q > a.maxq) continue;
                q = __fdiv_rn(q, a.dq);
                if (INTERP == 0) {
                    // sc = (uint)floor(q + 0.5) with q + 0.5 in double: floor(fl(q +
                    // 0.49999997f)) equals it for every float 0 <= q < 2^23 (the
                    // identity of round_half_away); fl(q + 0.5f) does not at
                    // q = 0.5 - 2^-25, whose sum rounds up to 1
                    const uint32_t sc = wrap_bin((uint32_t)floorf(fadd(q, 0.49999997f)), a.hsize);
                    const unsigned long long v =
                        a.mult_int ? scaled_floor(pv, a.mult_int) : (unsigned long long)(long long)dmul(val, a.mult);
                    shared_add_u64_split(hlo, hhi, sc, 2ull * v);
                } else {
                    uint32_t iq;  // q = |q| / dq <= MaxQ / dq < 2^23
                    const float fq = floor_small(q, iq);
                    const uint32_t sc1 = wrap_bin(iq, a.hsize), sc2 = wrap_bin(iq + 1, a.hsize);
                    const double sep = (double)fsub(q, fq);
                    const unsigned long long v1 =
                        (unsigned long long)(long long)dmul(dmul(val, dsub(1.0, sep)), a.mult);
                    const unsigned long long v2 = (unsigned long long)(long long)dmul(dmul(val, sep), a.mult);
                    shared_add_u64_split(hlo, hhi, sc1, 2ull * v1);
                    shared_add_u64_split(hlo, hhi, sc2, 2ull * v2);
                }
            }
        }
        __syncthreads();
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < a.hsize; i += DTILE) {
        const unsigned long long v = split_word(hlo, hhi, i);
        if (v) atomicAdd(&a.out[i], v);
    }
}

// --------------------------------------------------------------------------
// Row lists: the reference's own work decomposition.  Work item `ind` of
// AutoCorr_CQ_small / AutoCorr_CQ_AV visits every pixel i and bins the
// ordered pair (ind, i) (IAC/kernel.cl:78-182, :696-762); the mesh is the sum
// of these independent items.  The kernels below evaluate the items of a list
// of rows, each pair in the reference's arithmetic and order, so that a
// full-size detector can be checked against the oracle on a subset of rows and
// the unordered-pair kernels above against the sum over every row.  A CTA
// stages 256 consecutive pixels and each thread walks them for its row.
// --------------------------------------------------------------------------
__device__ __forceinline__ void global_put(const DenseArgs &a, int fs, int ms, int ss, unsigned long long v)
{
    if (v == 0) return;
    if ((unsigned)fs >= (unsigned)a.ab || (unsigned)ms >= (unsigned)a.ab || (unsigned)ss >= (unsigned)a.sc)
        atomicAdd(&a.counters->out_of_mesh, 1ull);
    else
        atomicAdd(&a.out[(uint64_t)fs + (uint64_t)ms * a.ab + (uint64_t)ss * a.ab * a.ab], v);
}

// the staged column tile of a row-list kernel: 256 consecutive pixels as (k, I)
__device__ __forceinline__ void stage_columns(const DenseArgs &a, uint64_t col_tile, float4 *sq)
{
    const uint64_t j = col_tile * DTILE + threadIdx.x;
    sq[threadIdx.x] = j < a.npix ? make_float4(a.K[3 * j], a.K[3 * j + 1], a.K[3 * j + 2], a.I[j])
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
}

// C(q) small mesh, rows x all pixels: grid (column tiles, row tiles)
template <int INTERP>
__global__ void __launch_bounds__(DTILE) cq_rows_kernel(const DenseArgs a, const uint32_t *__restrict__ rows,
                                                        uint32_t nrows)
{
    __shared__ float4 sq[DTILE];
    stage_columns(a, blockIdx.x, sq);
    __syncthreads();
    const uint32_t r = blockIdx.y * DTILE + threadIdx.x;
    if (r >= nrows) return;
    const uint32_t ind = rows[r];
    if (ind >= a.npix) {
        if (blockIdx.x == 0) atomicAdd(&a.counters->out_of_mesh, 1ull);
        return;
    }
    const float k0 = a.K[3 * (uint64_t)ind], k1 = a.K[3 * (uint64_t)ind + 1], k2 = a.K[3 * (uint64_t)ind + 2];
    const float Ia = a.I[ind];
    int cf = 0, cm = 0, cs = 0;
    bool have = false;
    unsigned long long acc[INTERP ? 8 : 1];
#pragma unroll
    for (int c = 0; c < (INTERP ? 8 : 1); c++) acc[c] = 0;
    for (int j = 0; j < DTILE; j++) {
        const float4 b = sq[j];
        const float pv = fmul(Ia, b.w);  // Val = (double)(I_ind * I_i)
        if (pv < 1e-37f) continue;
        float qx = fsub(k0, b.x), qy = fsub(k1, b.y), qz = fsub(k2, b.z);
        if (fadd(fadd(fmul(qx, qx), fmul(qy, qy)), fmul(qz, qz)) > a.maxq2) continue;
        qx = fmul(qx, a.vpdq);
        qy = fmul(qy, a.vpdq);
        qz = fmul(qz, a.vpdq);
        const float qa = pick(qx, qy, qz, a.ka), qb = pick(qx, qy, qz, a.kb), qc = pick(qx, qy, qz, a.kc);
        int f, m, sv;
        if (INTERP == 0) {
            f = round_half_away(qa) + a.cab;
            m = round_half_away(qb) + a.cab;
            sv = round_half_away(qc) + a.cc;
        } else {
            f = __float2int_rd(qa) + a.cab;
            m = __float2int_rd(qb) + a.cab;
            sv = __float2int_rd(qc) + a.cc;
        }
        if (!have || f != cf || m != cm || sv != cs) {
            if (have) {
#pragma unroll
                for (int c = 0; c < (INTERP ? 8 : 1); c++)
                    global_put(a, cf + (c >> 2), cm + ((c >> 1) & 1), cs + (c & 1), acc[c]);
            }
            have = true;
            cf = f;
            cm = m;
            cs = sv;
#pragma unroll
            for (int c = 0; c < (INTERP ? 8 : 1); c++) acc[c] = 0;
        }
        if (INTERP == 0) {
            acc[0] += a.mult_int ? scaled_floor(pv, a.mult_int) : d2u64(dmul((double)pv, a.mult));
        } else {
            const double vm = dmul((double)pv, a.mult);
            const double sf = (double)fsub(1.0f, fsub(qa, floorf(qa)));
            const double sm = (double)fsub(1.0f, fsub(qb, floorf(qb)));
            const double sz = (double)fsub(1.0f, fsub(qc, floorf(qc)));
            const double xf[2] = {sf, dsub(1.0, sf)}, yf[2] = {sm, dsub(1.0, sm)}, zf[2] = {sz, dsub(1.0, sz)};
#pragma unroll
            for (int c = 0; c < 8; c++) acc[c] += d2u64(dmul(vm, dmul(dmul(xf[c >> 2], yf[(c >> 1) & 1]), zf[c & 1])));
        }
    }
    if (have) {
#pragma unroll
        for (int c = 0; c < (INTERP ? 8 : 1); c++)
            global_put(a, cf + (c >> 2), cm + ((c >> 1) & 1), cs + (c & 1), acc[c]);
    }
}

// AC1D |q| histogram, rows x all pixels: persistent CTAs over (row tile,
// column tile) items, the histogram in shared memory for the whole launch
template <int INTERP>
__global__ void __launch_bounds__(DTILE) ac1d_rows_kernel(const DenseArgs a, const uint32_t *__restrict__ rows,
                                                          uint32_t nrows)
{
    extern __shared__ unsigned long long hist[];
    __shared__ float4 sq[DTILE];
    __shared__ unsigned long long s_item;
    for (uint32_t i = threadIdx.x; i < a.hsize; i += DTILE) hist[i] = 0;
    const uint64_t ncol = (a.npix + DTILE - 1) / DTILE;
    const unsigned long long nitems = (unsigned long long)ncol * ((nrows + DTILE - 1) / DTILE);
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(a.queue, 1ull);
        __syncthreads();
        const unsigned long long it = s_item;
        if (it >= nitems) break;
        const uint64_t rt = it / ncol, ct = it - rt * ncol;
        stage_columns(a, ct, sq);
        __syncthreads();
        const uint64_t r = rt * DTILE + threadIdx.x;
        const uint32_t ind = r < nrows ? rows[r] : 0xffffffffu;
        if (r < nrows && ind >= a.npix && ct == 0) atomicAdd(&a.counters->out_of_mesh, 1ull);
        if (ind < a.npix) {
            const float k0 = a.K[3 * (uint64_t)ind], k1 = a.K[3 * (uint64_t)ind + 1], k2 = a.K[3 * (uint64_t)ind + 2];
            const float Ia = a.I[ind];
            for (int j = 0; j < DTILE; j++) {
                const float4 b = sq[j];
                const float pv = fmul(Ia, b.w);
                if (pv < 1e-37f) continue;
                const double val = (double)pv;
                const float dx = fsub(k0, b.x), dy = fsub(k1, b.y), dz = fsub(k2, b.z);
                float q = __fsqrt_rn(fadd(fadd(fmul(dx, dx), fmul(dy, dy)), fmul(dz, dz)));
                if (q > a.maxq) continue;
                q = __fdiv_rn(q, a.dq);
                if (INTERP == 0) {
                    const uint32_t sc = wrap_bin((uint32_t)floor(dadd((double)q, 0.5)), a.hsize);
                    atomicAdd(&hist[sc], a.mult_int ? scaled_floor(pv, a.mult_int)
                                                    : (unsigned long long)(long long)dmul(val, a.mult));
                } else {
                    const float fq = floorf(q);
                    const double sep = (double)fsub(q, fq);
                    atomicAdd(&hist[wrap_bin((uint32_t)fq, a.hsize)],
                              (unsigned long long)(long long)dmul(dmul(val, dsub(1.0, sep)), a.mult));
                    atomicAdd(&hist[wrap_bin((uint32_t)fq + 1, a.hsize)],
                              (unsigned long long)(long long)dmul(dmul(val, sep), a.mult));
                }
            }
        }
        __syncthreads();
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < a.hsize; i += DTILE)
        if (hist[i]) atomicAdd(&a.out[i], hist[i]);
}

constexpr uint32_t AC1D_MAX_SIZE = 24576;  // bins of a shared-memory histogram of 64-bit words

iac_status dense_kernel_limits()
{
    constexpr int hist = (int)(sizeof(unsigned long long) * AC1D_MAX_SIZE);
    for (auto k : {ac1d_cq_kernel<0>, ac1d_cq_kernel<1>})
        IAC_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, hist));
    for (auto k : {ac1d_rows_kernel<0>, ac1d_rows_kernel<1>})
        IAC_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, hist));
    return IAC_OK;
}

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

// tile boxes + queue counter in stream scratch; returns args with common fields
static iac_status prepare(iac_ctx *ctx, void *stream, const float *d_I, const float *d_K,
                          uint64_t npix, uint32_t fast_size, double mult, DenseArgs &a)
{
    a.I = d_I;
    a.K = d_K;
    a.npix = npix;
    a.mult = mult;
    a.mult_int = (mult >= 1.0 && mult < 536870912.0 && mult == std::floor(mult)) ? (uint32_t)mult : 0u;
    if (fast_size >= 16 && npix % fast_size == 0) {
        a.nx = fast_size;
        a.ny = (uint32_t)(npix / fast_size);
        a.ptx = (a.nx + 15) / 16;
        a.ntiles = a.ptx * ((a.ny + 15) / 16);
    } else {
        a.nx = a.ny = a.ptx = 0;
        a.ntiles = (uint32_t)((npix + DTILE - 1) / DTILE);
    }
    a.mult_f = a.mult_int && (double)(float)mult == mult ? (float)mult : 0.0f;
    a.neg_zero = -0.0f;
    a.npairs = (unsigned long long)a.ntiles * (a.ntiles + 1) / 2;
    a.part = 0;
    a.nparts = 1;
    a.counters = ctx->d_counters;
    void *scr = nullptr;
    const size_t box_bytes = sizeof(float4) * 2 * (size_t)a.ntiles;
    iac_status st = stream_scratch(ctx, stream, SLOT_AUX0, box_bytes + 256, &scr);
    if (st != IAC_OK) return st;
    a.box = (const float4 *)scr;
    a.queue = (unsigned long long *)((char *)scr + ((box_bytes + 127) / 128) * 128);
    cudaStream_t s = as_stream(stream);
    IAC_CUDA(cudaMemsetAsync(a.queue, 0, sizeof(unsigned long long), s));
    tile_box_kernel<<<a.ntiles, DTILE, 0, s>>>(a, (float4 *)scr);
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    return IAC_OK;
}

}  // namespace iac

using namespace iac;

extern "C" {

iac_status iac_cq_small(iac_ctx *ctx, const float *d_I, const float *d_kmap, uint64_t npix,
                        uint32_t fast_size, const iac_mesh_shape *sh, int interp, double mult,
                        uint64_t *d_mesh, void *stream)
{
    return iac_cq_small_part(ctx, d_I, d_kmap, npix, fast_size, sh, interp, mult, 0, 1, d_mesh, stream);
}

iac_status iac_cq_small_part(iac_ctx *ctx, const float *d_I, const float *d_kmap, uint64_t npix,
                             uint32_t fast_size, const iac_mesh_shape *sh, int interp, double mult,
                             uint32_t part, uint32_t nparts, uint64_t *d_mesh, void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx && d_I && d_kmap && sh && d_mesh, "iac_cq_small: NULL argument");
    IAC_REQUIRE(nparts >= 1 && part < nparts, "iac_cq_small_part: part %u of %u", part, nparts);
    IAC_REQUIRE(interp == 0 || interp == 1, "interpolation must be 0 or 1");
    IAC_REQUIRE(npix > 0 && npix < (1ull << 32), "iac_cq_small: pixel count %llu out of range",
                (unsigned long long)npix);
    IAC_REQUIRE(sh->size_ab >= 5 && sh->size_ab % 2 == 1 && sh->size_c >= 1 && sh->size_c % 2 == 1,
                "small mesh sizes must be odd");
    IAC_REQUIRE(sh->k_a < 3 && sh->k_b < 3 && sh->k_c < 3, "bad axis alignment");
    IAC_REQUIRE(mult > 0, "multiplicator must be positive");
    DeviceGuard g(ctx->device);
    DenseArgs a{};
    iac_status st = prepare(ctx, stream, d_I, d_kmap, npix, fast_size, mult, a);
    if (st != IAC_OK) return st;
    a.part = part;
    a.nparts = nparts;
    a.out = (unsigned long long *)d_mesh;
    a.maxq = sh->max_q;
    a.maxq2 = sqrt_threshold(sh->max_q);
    a.vpdq = (float)sh->voxel_per_dq;
    a.ab = (int)sh->size_ab;
    a.sc = (int)sh->size_c;
    a.cab = (a.ab - 1) / 2;
    a.cc = (a.sc - 1) / 2;
    a.ka = (int)sh->k_a;
    a.kb = (int)sh->k_b;
    a.kc = (int)sh->k_c;
    // every pair within MaxQ has |q * Voxel_per_dq| <= MaxQ * Voxel_per_dq (up to
    // rounding): below 500 the packed voxel key cannot alias
    a.key_ok = (double)sh->max_q * (double)sh->voxel_per_dq < 500.0;
    const int grid = ctx->sm_count * 8;
    // the axis mapping is a permutation for every real detector: one
    // instantiation per permutation, a runtime-mapped one otherwise
    const int perm = (a.ka == 0 && a.kb == 1 && a.kc == 2)   ? 0
                     : (a.ka == 0 && a.kb == 2 && a.kc == 1) ? 1
                     : (a.ka == 1 && a.kb == 0 && a.kc == 2) ? 2
                     : (a.ka == 1 && a.kb == 2 && a.kc == 0) ? 3
                     : (a.ka == 2 && a.kb == 0 && a.kc == 1) ? 4
                     : (a.ka == 2 && a.kb == 1 && a.kc == 0) ? 5
                                                             : 6;
    cudaStream_t s = as_stream(stream);
#define IAC_CQ_LAUNCH(I)                                                          \
    switch (perm) {                                                               \
    case 0: cq_small_kernel<I, 0, 1, 2><<<grid, DTILE, 0, s>>>(a); break;         \
    case 1: cq_small_kernel<I, 0, 2, 1><<<grid, DTILE, 0, s>>>(a); break;         \
    case 2: cq_small_kernel<I, 1, 0, 2><<<grid, DTILE, 0, s>>>(a); break;         \
    case 3: cq_small_kernel<I, 1, 2, 0><<<grid, DTILE, 0, s>>>(a); break;         \
    case 4: cq_small_kernel<I, 2, 0, 1><<<grid, DTILE, 0, s>>>(a); break;         \
    case 5: cq_small_kernel<I, 2, 1, 0><<<grid, DTILE, 0, s>>>(a); break;         \
    default: cq_small_kernel<I, -1, -1, -1><<<grid, DTILE, 0, s>>>(a); break;     \
    }
    if (interp == 0) {
        IAC_CQ_LAUNCH(0)
    } else {
        IAC_CQ_LAUNCH(1)
    }
#undef IAC_CQ_LAUNCH
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    return IAC_OK;
}

iac_status iac_ac1d_cq(iac_ctx *ctx, const float *d_I, const float *d_kmap, uint64_t npix,
                       const iac_ac1d_shape *sh, int interp, double mult, uint64_t *d_hist,
                       void *stream)
{
    return iac_ac1d_cq_part(ctx, d_I, d_kmap, npix, sh, interp, mult, 0, 1, d_hist, stream);
}

iac_status iac_ac1d_cq_part(iac_ctx *ctx, const float *d_I, const float *d_kmap, uint64_t npix,
                            const iac_ac1d_shape *sh, int interp, double mult, uint32_t part, uint32_t nparts,
                            uint64_t *d_hist, void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx && d_I && d_kmap && sh && d_hist, "iac_ac1d_cq: NULL argument");
    IAC_REQUIRE(nparts >= 1 && part < nparts, "iac_ac1d_cq_part: part %u of %u", part, nparts);
    IAC_REQUIRE(interp == 0 || interp == 1, "interpolation must be 0 or 1");
    IAC_REQUIRE(npix > 0 && npix < (1ull << 32), "iac_ac1d_cq: pixel count out of range");
    IAC_REQUIRE(sh->size >= 3 && sh->size <= AC1D_MAX_SIZE, "AC1D size %u out of range [3, %u]", sh->size,
                AC1D_MAX_SIZE);
    IAC_REQUIRE(sh->dq_per_step > 0 && (double)sh->max_q / sh->dq_per_step < 4194304.0,
                "iac_ac1d_cq: MaxQ / dq must be below 2^22 (dq %g, MaxQ %g)", (double)sh->dq_per_step,
                (double)sh->max_q);
    IAC_REQUIRE(mult > 0, "multiplicator must be positive");
    DeviceGuard g(ctx->device);
    DenseArgs a{};
    // linear tiles: the pixels of a 16 x 16 patch pair share few |q| bins, and
    // a warp's shared-memory histogram atomics would collide on them
    iac_status st = prepare(ctx, stream, d_I, d_kmap, npix, 0, mult, a);
    if (st != IAC_OK) return st;
    a.part = part;
    a.nparts = nparts;
    a.out = (unsigned long long *)d_hist;
    a.maxq = sh->max_q;
    a.maxq2 = sqrt_threshold(sh->max_q);
    a.hsize = sh->size;
    a.dq = sh->dq_per_step;
    a.by_dq = make_divisor(sh->dq_per_step);
    a.in_range = sh->dq_per_step > 1e-30f && sh->dq_per_step < 1e30f &&
                 (double)sh->max_q / sh->dq_per_step * 1.000001 < (double)sh->size - 1.0;
    const size_t smem = sizeof(unsigned long long) * sh->size;
    auto k = interp == 0 ? ac1d_cq_kernel<0> : ac1d_cq_kernel<1>;
    k<<<ctx->sm_count * 8, DTILE, smem, as_stream(stream)>>>(a);
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    return IAC_OK;
}

}  // extern "C"

extern "C" {

iac_status iac_cq_small_rows(iac_ctx *ctx, const float *d_I, const float *d_kmap, uint64_t npix,
                             const uint32_t *d_rows, uint32_t nrows, const iac_mesh_shape *sh, int interp,
                             double mult, uint64_t *d_mesh, void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx && d_I && d_kmap && sh && d_mesh && d_rows, "iac_cq_small_rows: NULL argument");
    IAC_REQUIRE(interp == 0 || interp == 1, "interpolation must be 0 or 1");
    IAC_REQUIRE(npix > 0 && npix < (1ull << 32), "iac_cq_small_rows: pixel count %llu out of range",
                (unsigned long long)npix);
    IAC_REQUIRE(nrows >= 1 && nrows <= 65535u * DTILE, "iac_cq_small_rows: %u rows out of range [1, %u]", nrows,
                65535u * DTILE);
    IAC_REQUIRE(sh->size_ab >= 5 && sh->size_ab % 2 == 1 && sh->size_c >= 1 && sh->size_c % 2 == 1,
                "small mesh sizes must be odd");
    IAC_REQUIRE(sh->k_a < 3 && sh->k_b < 3 && sh->k_c < 3, "bad axis alignment");
    IAC_REQUIRE(mult > 0, "multiplicator must be positive");
    DeviceGuard g(ctx->device);
    DenseArgs a{};
    a.I = d_I;
    a.K = d_kmap;
    a.npix = npix;
    a.mult = mult;
    a.mult_int = (mult >= 1.0 && mult < 536870912.0 && mult == std::floor(mult)) ? (uint32_t)mult : 0u;
    a.counters = ctx->d_counters;
    a.out = (unsigned long long *)d_mesh;
    a.maxq = sh->max_q;
    a.maxq2 = sqrt_threshold(sh->max_q);
    a.vpdq = (float)sh->voxel_per_dq;
    a.ab = (int)sh->size_ab;
    a.sc = (int)sh->size_c;
    a.cab = (a.ab - 1) / 2;
    a.cc = (a.sc - 1) / 2;
    a.ka = (int)sh->k_a;
    a.kb = (int)sh->k_b;
    a.kc = (int)sh->k_c;
    const dim3 grid((unsigned)((npix + DTILE - 1) / DTILE), (nrows + DTILE - 1) / DTILE);
    if (interp == 0)
        cq_rows_kernel<0><<<grid, DTILE, 0, as_stream(stream)>>>(a, d_rows, nrows);
    else
        cq_rows_kernel<1><<<grid, DTILE, 0, as_stream(stream)>>>(a, d_rows, nrows);
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    return IAC_OK;
}

iac_status iac_ac1d_cq_rows(iac_ctx *ctx, const float *d_I, const float *d_kmap, uint64_t npix,
                            const uint32_t *d_rows, uint32_t nrows, const iac_ac1d_shape *sh, int interp,
                            double mult, uint64_t *d_hist, void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx && d_I && d_kmap && sh && d_hist && d_rows, "iac_ac1d_cq_rows: NULL argument");
    IAC_REQUIRE(interp == 0 || interp == 1, "interpolation must be 0 or 1");
    IAC_REQUIRE(npix > 0 && npix < (1ull << 32), "iac_ac1d_cq_rows: pixel count out of range");
    IAC_REQUIRE(nrows >= 1, "iac_ac1d_cq_rows: no rows");
    IAC_REQUIRE(sh->size >= 3 && sh->size <= AC1D_MAX_SIZE, "AC1D size %u out of range [3, %u]", sh->size,
                AC1D_MAX_SIZE);
    IAC_REQUIRE(mult > 0, "multiplicator must be positive");
    DeviceGuard g(ctx->device);
    DenseArgs a{};
    a.I = d_I;
    a.K = d_kmap;
    a.npix = npix;
    a.mult = mult;
    a.mult_int = (mult >= 1.0 && mult < 536870912.0 && mult == std::floor(mult)) ? (uint32_t)mult : 0u;
    a.counters = ctx->d_counters;
    a.out = (unsigned long long *)d_hist;
    a.maxq = sh->max_q;
    a.hsize = sh->size;
    a.dq = sh->dq_per_step;
    void *scr = nullptr;
    iac_status st = stream_scratch(ctx, stream, SLOT_AUX0, 256, &scr);
    if (st != IAC_OK) return st;
    a.queue = (unsigned long long *)scr;
    cudaStream_t s = as_stream(stream);
    IAC_CUDA(cudaMemsetAsync(a.queue, 0, sizeof(unsigned long long), s));
    const size_t smem = sizeof(unsigned long long) * sh->size;
    auto k = interp == 0 ? ac1d_rows_kernel<0> : ac1d_rows_kernel<1>;
    k<<<ctx->sm_count * 4, DTILE, smem, s>>>(a, d_rows, nrows);
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    return IAC_OK;
}

}  // extern "C"
