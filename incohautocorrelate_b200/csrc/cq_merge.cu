// cq_merge.cu -- (b') rotate-and-weight merge of the small C(q) mesh into
// the big cubic mesh.
//
// Replaces Merge_CQ (IAC/kernel.cl:189-344) and the device part of
// Detector::Merge_smallCofQ (IAC/Detector.cpp:1321-1573).  For every small-mesh
// voxel with C >= 1e-37 and every frame f, the voxel's q (in voxels) is rotated
// by the frame's RotMatrix and (uint64)(C * w_f * Mult) is added at the
// nearest voxel (or split over 8 corners) of the cubic mesh.
//
// The non-zero voxels are first compacted in blocks of 2 x 4 x 4, so that a warp
// holds a small cube and, for one frame, scatters to a small rotated cube: its
// adds share the 32-byte sectors of a few rows.  L2 takes scattered 64-bit adds at
// about 2.2e11 a second, one request each; words of one sector travel together,
// here 3.2e11 a second (L2 77 % busy).  Linear: two lanes add the two adjacent
// words of one voxel's row in one instruction.  Each CTA stages a chunk of frames'
// rotations and weights in shared memory, two frames side by side for f32x2
// arithmetic, and walks them for its voxels; coordinates and values are rounded
// with adds, without the conversion unit.  199-edge mesh, 10 000 frames, nearest:
// 15.0 -> 10.3 ms; 1 000 frames linear: 11.3 -> 6.9 ms.
//
// Reference quirks kept: the slow index uses the A/B centre (:287, :306) and
// the NN value is (C * w) * Mult while the linear one is (C * Mult) * w * corner.
#include <algorithm>

#include "iac_internal.cuh"

namespace iac {

constexpr int MERGE_THREADS = 256;
constexpr int MERGE_FRAMES = 128;  // frames per shared-memory chunk
// A warp's voxels.  10 000 frames: 32 x 1 x 1 13.2 ms, 8 x 4 x 1 12.1, 8 x 2 x 2 11.8,
// 4 x 4 x 2 10.8, 4 x 2 x 4 10.5, 2 x 4 x 4 10.3.
constexpr uint32_t BLOCK_X = 2, BLOCK_Y = 4, BLOCK_Z = 4;

struct MergeArgs {
    const double *__restrict__ small;
    const float *__restrict__ rw;  // 10 floats per frame
    const uint32_t *__restrict__ list;  // compacted voxel indices
    const uint32_t *__restrict__ count;
    unsigned long long *__restrict__ big;
    DeviceCounters *counters;
    uint32_t nframes;
    int ab, sc, cab, cc;
    int ka, kb, kc;
    double mult;
    float neg_zero;
};

__global__ void merge_compact_kernel(const double *__restrict__ small, uint32_t ab, uint32_t sc,
                                     uint32_t *__restrict__ list, uint32_t *__restrict__ count)
{
    __shared__ uint32_t s_warp[MERGE_THREADS / 32];
    __shared__ uint32_t s_base;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // the warp's block of the mesh and the lane's voxel in it
    const uint32_t b = blockIdx.x * (MERGE_THREADS / 32) + w, nx = (ab + BLOCK_X - 1) / BLOCK_X,
                   ny = (ab + BLOCK_Y - 1) / BLOCK_Y;
    const uint32_t by = b / nx, bz = by / ny;
    const uint32_t x = (b - by * nx) * BLOCK_X + lane % BLOCK_X, y = (by - bz * ny) * BLOCK_Y + lane / BLOCK_X % BLOCK_Y,
                   z = bz * BLOCK_Z + lane / (BLOCK_X * BLOCK_Y);
    const uint32_t i = x + ab * (y + ab * z);
    const bool keep = x < ab && y < ab && z < sc && !(small[i] < 1e-37f);  // IAC/kernel.cl:260
    const unsigned ball = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) s_warp[w] = __popc(ball);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int k = 0; k < MERGE_THREADS / 32; k++) {
            const uint32_t c = s_warp[k];
            s_warp[k] = t;
            t += c;
        }
        s_base = t ? atomicAdd(count, t) : 0;
    }
    __syncthreads();
    if (keep) list[s_base + s_warp[w] + __popc(ball & ((1u << lane) - 1))] = i;
}

__device__ __forceinline__ void big_put(const MergeArgs &a, int fs, int ms, int ss,
                                        unsigned long long v)
{
    if (v == 0) return;
    if ((unsigned)fs >= (unsigned)a.ab || (unsigned)ms >= (unsigned)a.ab ||
        (unsigned)ss >= (unsigned)a.ab) {
        atomicAdd(&a.counters->out_of_mesh, 1ull);
        return;
    }
    atomicAdd(&a.big[(uint64_t)fs + (uint64_t)ms * a.ab + (uint64_t)ss * a.ab * a.ab], v);
}

// the cast of a value: below 2^52 by an add rounded toward zero
__device__ __forceinline__ unsigned long long merge_value(double x)
{
    if ((uint32_t)__double2hiint(x) < 0x43300000u) {
        const double y = __dadd_rz(x, 4503599627370496.0);
        return (unsigned long long)__double_as_longlong(y) & 0xfffffffffffffull;
    }
    return d2u64(x);
}

// a pair at q = (q0, q1, q2) by the reference's steps, wherever it lands
template <int INTERP>
__device__ __forceinline__ void merge_any(const MergeArgs &a, double vin, double w, float o0, float o1, float o2)
{
    const float cabf = (float)a.cab;
    if (INTERP == 0) {
        big_put(a, (int)fadd(round_away_f(o0), cabf), (int)fadd(round_away_f(o1), cabf),
                (int)fadd(round_away_f(o2), cabf), d2u64(dmul(dmul(vin, w), a.mult)));
        return;
    }
    const float f0x = floorf(o0), f1x = floorf(o1), f2x = floorf(o2);
    const double sf = (double)fsub(1.0f, fsub(o0, f0x)), sm = (double)fsub(1.0f, fsub(o1, f1x)),
                 sz = (double)fsub(1.0f, fsub(o2, f2x));
    const int fs = (int)fadd(f0x, cabf), ms = (int)fadd(f1x, cabf), ss = (int)fadd(f2x, cabf);
    const double base = dmul(dmul(vin, a.mult), w);
#pragma unroll 1
    for (int c = 0; c < 8; c++)
        big_put(a, fs + (c >> 2), ms + ((c >> 1) & 1), ss + (c & 1),
                d2u64(dmul(base, dmul(dmul(c >> 2 ? dsub(1.0, sf) : sf, (c >> 1) & 1 ? dsub(1.0, sm) : sm),
                                      c & 1 ? dsub(1.0, sz) : sz))));
}

__device__ __forceinline__ void big_add(unsigned long long *p, unsigned long long v)
{
    if (v) atomicAdd(p, v);
}

// One CTA per SM as the bound: ptxas then takes 48 registers and keeps both frames'
// chains in flight, 10.3 ms; with the 32 it takes without a bound 12.3.
template <int INTERP>
__global__ void __launch_bounds__(MERGE_THREADS, 1) merge_kernel(const MergeArgs a)
{
    // two frames f, f + 1 at a time: rows' elements as (r_f, r_f+1), weights as doubles
    __shared__ float4 s_r[MERGE_FRAMES / 2][5];  // two elements each, the last alone
    __shared__ double2 s_w[MERGE_FRAMES / 2];
    const uint32_t nvox = *a.count;
    const uint32_t f0 = blockIdx.y * MERGE_FRAMES;
    const uint32_t nf = min((uint32_t)MERGE_FRAMES, a.nframes - f0);
    for (uint32_t k = threadIdx.x; k < (nf + 1) / 2 * 20; k += MERGE_THREADS) {
        const uint32_t f = k / 10, e = k - 10 * f;
        const float r = f < nf ? a.rw[(size_t)f0 * 10 + k] : 0.0f;
        reinterpret_cast<float *>(s_r[f >> 1])[2 * e + (f & 1)] = r;
        if (e == 9) reinterpret_cast<double *>(&s_w[f >> 1])[f & 1] = (double)r;
    }
    __syncthreads();
    const uint32_t ab = (uint32_t)a.ab, AB2 = ab * ab;
    const float2 nz = make_float2(a.neg_zero, a.neg_zero);
    const bool odd = threadIdx.x & 1;
    for (uint32_t t = blockIdx.x * MERGE_THREADS + threadIdx.x; (t & ~31u) < nvox; t += gridDim.x * MERGE_THREADS) {
        const bool active = t < nvox;
        const uint32_t ind = a.list[active ? t : nvox - 1];
        const uint32_t ss_in = ind / AB2, ms_in = (ind - ss_in * AB2) / ab, fs_in = ind - ss_in * AB2 - ms_in * ab;
        float qi[3];
        qi[a.ka] = (float)((int)fs_in - a.cab);
        qi[a.kb] = (float)((int)ms_in - a.cab);
        qi[a.kc] = (float)((int)ss_in - a.cc);
        const double vin = a.small[ind];
        const float2 x = make_float2(qi[0], qi[0]), y = make_float2(qi[1], qi[1]), z = make_float2(qi[2], qi[2]);
        for (uint32_t p = 0; 2 * p < nf; p++) {
            float2 r[10];
#pragma unroll
            for (int k = 0; k < 5; k++) {
                const float4 v = s_r[p][k];
                r[2 * k] = make_float2(v.x, v.y);
                r[2 * k + 1] = make_float2(v.z, v.w);
            }
            const double2 ww = s_w[p];
            float2 o[3];
#pragma unroll
            for (int k = 0; k < 3; k++)  // rot_row's roundings
                o[k] = f2add(f2add(f2fma(x, r[3 * k], nz), f2fma(y, r[3 * k + 1], nz)), f2fma(z, r[3 * k + 2], nz));
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const float q[3] = {e ? o[0].y : o[0].x, e ? o[1].y : o[1].x, e ? o[2].y : o[2].x};
                const double w = e ? ww.y : ww.x;
                const bool on = active && 2 * p + e < nf;
                if (INTERP == 0) {
                    uint32_t i[3];
#pragma unroll
                    for (int k = 0; k < 3; k++) i[k] = (uint32_t)(round_away_rz_i(q[k]) + a.cab);
                    if (on) {
                        if (i[0] < ab && i[1] < ab && i[2] < ab)
                            big_add(a.big + (i[0] + ab * (i[1] + ab * (unsigned long long)i[2])),
                                    merge_value(dmul(dmul(vin, w), a.mult)));
                        else
                            merge_any<0>(a, vin, w, q[0], q[1], q[2]);
                    }
                } else {
                    uint32_t i[3];
                    double s[3], c[3];
#pragma unroll
                    for (int k = 0; k < 3; k++) {  // floor by an add rounded down, for |q| < 2^22
                        const float m = __fadd_rd(q[k], ROUND_MAGIC);
                        i[k] = (uint32_t)(__float_as_int(m) - __float_as_int(ROUND_MAGIC) + a.cab);
                        s[k] = (double)fsub(1.0f, fsub(q[k], fsub(m, ROUND_MAGIC)));
                        c[k] = dsub(1.0, s[k]);
                    }
                    const bool in = i[0] < ab - 1 && i[1] < ab - 1 && i[2] < ab - 1;
                    if (on && !in) merge_any<1>(a, vin, w, q[0], q[1], q[2]);
                    const bool add = on && in;
                    if (!add)
#pragma unroll
                        for (int k = 0; k < 3; k++) s[k] = c[k] = 0.0;  // NaN where q is not finite: 0 * NaN is no 0
                    const double base = add ? dmul(dmul(vin, a.mult), w) : 0.0;
                    const unsigned long long at = add ? i[0] + ab * (i[1] + ab * (unsigned long long)i[2]) : 0ull;
                    // even lanes add a voxel's lower word while odd lanes add the upper one of
                    // the same voxel: first the even lanes' voxels, then the odd lanes'
                    const unsigned long long there = __shfl_xor_sync(0xffffffffu, at, 1);
                    unsigned long long *const first = a.big + (odd ? there + 1 : at),
                                             *const second = a.big + (odd ? at + 1 : there);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const double fm = k >> 1 ? c[1] : s[1], fz = k & 1 ? c[2] : s[2];
                        const unsigned long long lo = merge_value(dmul(base, dmul(dmul(s[0], fm), fz))),
                                                 hi = merge_value(dmul(base, dmul(dmul(c[0], fm), fz)));
                        const unsigned long long got = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);
                        const size_t off = (k >> 1) * (size_t)ab + (k & 1) * (size_t)AB2;
                        big_add(first + off, odd ? got : lo);
                        big_add(second + off, odd ? hi : got);
                    }
                }
            }
        }
    }
}

}  // namespace iac

using namespace iac;

extern "C" iac_status iac_cq_merge(iac_ctx *ctx, const double *d_small_cq, const float *d_rw10,
                                   uint32_t nframes, const iac_mesh_shape *sh, int interp,
                                   double mult, uint64_t *d_big, void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx && d_small_cq && sh && d_big, "iac_cq_merge: NULL argument");
    IAC_REQUIRE(interp == 0 || interp == 1, "interpolation must be 0 or 1");
    IAC_REQUIRE(sh->size_ab >= 5 && sh->size_ab % 2 == 1 && sh->size_c % 2 == 1 &&
                    sh->size_c <= sh->size_ab && sh->size_ab <= 1625,
                "iac_cq_merge: bad small mesh %u x %u", sh->size_ab, sh->size_c);
    IAC_REQUIRE(sh->k_a < 3 && sh->k_b < 3 && sh->k_c < 3 &&
                    sh->k_a + sh->k_b + sh->k_c == 3 && sh->k_a != sh->k_b,
                "iac_cq_merge: axis alignment is not a permutation");
    IAC_REQUIRE(mult > 0, "multiplicator must be positive");
    if (nframes == 0) return IAC_OK;
    IAC_REQUIRE(d_rw10 != nullptr, "iac_cq_merge: NULL rotation/weight table");
    DeviceGuard g(ctx->device);
    const uint32_t n = sh->size_ab * sh->size_ab * sh->size_c;
    void *scr = nullptr;
    iac_status st = stream_scratch(ctx, stream, SLOT_AUX1, sizeof(uint32_t) * ((size_t)n + 64), &scr);
    if (st != IAC_OK) return st;
    uint32_t *count = (uint32_t *)scr;
    uint32_t *list = count + 32;
    cudaStream_t s = as_stream(stream);
    IAC_CUDA(cudaMemsetAsync(count, 0, sizeof(uint32_t), s));
    const uint64_t blocks = (uint64_t)((sh->size_ab + BLOCK_X - 1) / BLOCK_X) *
                            ((sh->size_ab + BLOCK_Y - 1) / BLOCK_Y) * ((sh->size_c + BLOCK_Z - 1) / BLOCK_Z);
    constexpr uint32_t per_cta = MERGE_THREADS / 32;
    merge_compact_kernel<<<(uint32_t)((blocks + per_cta - 1) / per_cta), MERGE_THREADS, 0, s>>>(
        d_small_cq, sh->size_ab, sh->size_c, list, count);
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    MergeArgs a;
    a.small = d_small_cq;
    a.rw = d_rw10;
    a.list = list;
    a.count = count;
    a.big = (unsigned long long *)d_big;
    a.counters = ctx->d_counters;
    a.nframes = nframes;
    a.ab = (int)sh->size_ab;
    a.sc = (int)sh->size_c;
    a.cab = (a.ab - 1) / 2;
    a.cc = (a.sc - 1) / 2;
    a.ka = (int)sh->k_a;
    a.kb = (int)sh->k_b;
    a.kc = (int)sh->k_c;
    a.mult = mult;
    a.neg_zero = -0.0f;
    const uint32_t chunks = (nframes + MERGE_FRAMES - 1) / MERGE_FRAMES;
    // enough voxel blocks per frame chunk to fill the GPU several times over
    const uint32_t vblocks = std::max<uint32_t>(1, std::min<uint32_t>(
        (n + MERGE_THREADS - 1) / MERGE_THREADS, (uint32_t)(ctx->sm_count * 8 + chunks - 1) / chunks));
    dim3 grid(vblocks, chunks);
    if (interp == 0)
        merge_kernel<0><<<grid, MERGE_THREADS, 0, s>>>(a);
    else
        merge_kernel<1><<<grid, MERGE_THREADS, 0, s>>>(a);
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    return IAC_OK;
}
